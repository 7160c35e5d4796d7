"""The autotuner keeps the two-level dedispersion in reach at every bit depth."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("nbits", [1, 4, 8])
def test_width_at_every_depth(gpu, nbits):
    """96 channels x 700 trials one sample apart, where two levels take about half
    of the channel-by-channel kernel's time: the tuned plan has a width, and the
    candidates are those of the batch before."""
    from pulsarsr_gb300 import batch, dedisperse, fbank, search, synth
    nch, ns, tsamp = 96, 300000, 72e-6
    h = fbank.HeaderInfo(nch, nbits, tsamp, 1447.5, -1.0, 0)
    freqs = 1447.5 - np.arange(nch)
    trials = dedisperse.dm_step(freqs, tsamp) * np.arange(700)
    cfg = search.Config(min_hz=15.0, max_hz=2000.0, threshold=8.0)
    n = ns - int(dedisperse.delays(freqs, tsamp, float(trials[-1])).max())
    b = batch.Batch([dict(header=h, nsamples=ns, trials=trials, discovery=n, config=cfg,
                          rfi_block=1389, rfi_threshold=8.0)])
    rng = np.random.default_rng(nbits)
    x = np.clip(np.rint(rng.normal(2 ** nbits / 2, 2 ** nbits / 5, (ns, nch))), 0,
                2 ** nbits - 1)
    b.load(0, synth.pack(x, nbits))
    b.run()
    b.sync()
    want = b.candidates(0)
    widths = b.tune()[2]
    assert widths[0] in (4, 8)
    b.run()
    b.sync()
    got = b.candidates(0)
    assert np.array_equal(got[0], want[0]) and got[1].tobytes() == want[1].tobytes()
