"""The two-level dedispersion (intra-subband delay patterns summed once per
chunk of trials) against the channel-by-channel kernel, which
tests/test_gpu_parity.py compares with the oracle: bit-identical series and
sums over every form of plan and sample that it takes."""
import numpy as np
import pytest

NOISE = {1: (0.5, 0.6), 2: (1.5, 0.8), 4: (7.5, 3.0), 8: (128.0, 60.0)}


def both(fb, trials, n, widths=(4, 8, -1)):
    from pulsarsr_gb300 import dedisperse
    out = {}
    try:
        for g in (0, *widths):
            dedisperse.set_subbands(g)
            out[g] = dedisperse.apply_trials(fb, trials, n, with_sums=True)
    finally:
        dedisperse.set_subbands(-1)
    for g in widths:
        assert out[g][0].tobytes() == out[0][0].tobytes(), g
        assert out[g][1].tobytes() == out[0][1].tobytes(), g


@pytest.mark.gpu
@pytest.mark.parametrize("nbits,nch", [(1, 9), (2, 64), (4, 97), (4, 8), (8, 5), (8, 256),
                                       (8, 261), (8, 1030)])
@pytest.mark.parametrize("order", ["up", "down", "repeat", "shuffled", "jumps", "one"])
def test_orders_and_channel_counts(gpu, nbits, nch, order):
    """Ascending, descending, repeated, shuffled and jumping plans, a single
    trial; channel counts around the subband widths, the 16-bit limit (257
    8-bit channels) and several flushes; lengths around the 1024-sample tile."""
    from pulsarsr_gb300 import dedisperse, synth
    mean, sigma = NOISE[nbits]
    fb = synth.device(nch, nbits, 9000, 64e-6, 1500.0, -300.0 / nch, seed=7 + nch,
                      noise_mean=mean, noise_sigma=sigma, gain_spread=0.1)
    freqs = fb.header.frequencies()
    step = dedisperse.dm_step(freqs, 64e-6)
    rng = np.random.default_rng(nch)
    t = {"up": step * np.arange(37), "down": step * np.arange(40, 0, -1) * 0.5,
         "repeat": np.repeat(step * np.arange(9), 3), "shuffled": step * rng.permutation(50),
         "jumps": step * np.concatenate([np.arange(20), 900 + np.arange(21), 300 + np.arange(7)]),
         "one": np.array([step * 77.3])}[order]
    md = int(dedisperse.delays(freqs, 64e-6, float(t.max())).max())
    for n in (1023, 1024, 1025, 9000 - md):
        both(fb, t, n)


@pytest.mark.gpu
def test_segments(gpu):
    """More pattern rows than one scratch segment holds: the series is made in
    several segments, the last one ragged."""
    from pulsarsr_gb300 import dedisperse, synth
    nch, ns = 1024, 400011
    fb = synth.device(nch, 8, ns, 64e-6, 1500.0, -300.0 / nch, seed=3, noise_mean=128.0,
                      noise_sigma=60.0)
    step = dedisperse.dm_step(fb.header.frequencies(), 64e-6)
    both(fb, 400 * step + step * np.arange(100), ns - 520, widths=(8,))
