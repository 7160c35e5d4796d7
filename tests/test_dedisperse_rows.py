"""Blocks of trials of f32 and 16-bit samples (staged rows, one warp per trial)
against sequential f32 sums in channel order and sequential f64 sums of the
series: bit for bit, at trial counts around 8 and 16, channel counts around a
stage, lengths around the 1024-sample tile, odd shifts, plans in any order and
with delays too far apart to stage; sums that are exact in any order and sums
that are not."""
import numpy as np
import pytest


def reference(x, delays, n):
    out = np.zeros((len(delays), n), np.float32)
    for i, d in enumerate(delays):
        for c in range(x.shape[0]):
            out[i] = out[i] + x[c, d[c]:d[c] + n]
    sums = np.array([np.add.accumulate(r.astype(np.float64))[-1] for r in out])
    return out, sums


def observation(nbits, nch, ns, values, seed):
    from pulsarsr_gb300 import fbank, synth
    rng = np.random.default_rng(seed)
    if nbits == 16:
        x = rng.integers(0, 65536, (ns, nch))
    else:
        x = {"integers": rng.integers(-9, 99, (ns, nch)), "noise": rng.normal(100, 10, (ns, nch)),
             "mixed": rng.normal(0, 1, (ns, nch)) * 10.0 ** rng.integers(-30, 9, (ns, nch)),
             "zeros": np.zeros((ns, nch))}[values]
    x = x.astype(np.float32)
    raw = synth.header_bytes(nch, nbits, 64e-6, 1500.0, -300.0 / nch) + synth.pack(x, nbits)
    return fbank.decode(raw), np.ascontiguousarray(x.T)


@pytest.mark.gpu
@pytest.mark.parametrize("nbits,values", [(16, "integers"), (32, "integers"), (32, "noise"),
                                          (32, "mixed"), (32, "zeros")])
@pytest.mark.parametrize("nch,ntrials", [(1, 8), (5, 7), (6, 8), (7, 15), (33, 16), (300, 17)])
@pytest.mark.parametrize("order", ["up", "shuffled", "jumps"])
def test_blocks_of_trials(gpu, nbits, values, nch, ntrials, order):
    from pulsarsr_gb300 import dedisperse
    ns = 9001
    fb, x = observation(nbits, nch, ns, values, nch * 100 + ntrials)
    freqs = fb.header.frequencies()
    step = dedisperse.dm_step(freqs, 64e-6) if nch > 1 else 1.0
    rng = np.random.default_rng(ntrials)
    k = np.arange(ntrials)
    t = step * {"up": 3.0 * k, "shuffled": 5.0 * rng.permutation(ntrials),
                "jumps": np.where(k % 3 == 1, 6000.0, 0.0) + k}[order]
    delays = [dedisperse.delays(freqs, 64e-6, float(v)) for v in t]
    top = int(max(d.max() for d in delays))
    for n in (1023, 1024, 1025, ns - top):
        got, sums = dedisperse.apply_trials(fb, t, n, with_sums=True)
        want, wsums = reference(x, delays, n)
        assert got.tobytes() == want.tobytes(), n
        assert np.asarray(sums, np.float64).tobytes() == wsums.tobytes(), n
