"""Channel means and variances at the edges of their parallel form (chunks of
512 terms, 32 chunks per scan step, binade guesses from plain sums) against
the oracle's sequential loops, bit for bit."""
import numpy as np
import pytest

SIZES = [2, 15, 16, 17, 511, 512, 513, 16383, 16384, 16385, 40961]


def columns(kind, ns, rng):
    if kind == "u8":
        return np.stack([np.full(ns, 255.0), rng.integers(0, 256, ns), rng.integers(200, 256, ns),
                         np.where(np.arange(ns) == ns - 1, 255, 0), np.zeros(ns),
                         rng.integers(0, 2, ns)], 1), 8
    if kind == "u16":
        # (a mean far above the spread: the plain sums guess the variance's binades badly)
        return np.stack([np.full(ns, 65535.0), 60000 + rng.integers(0, 2, ns),
                         rng.integers(0, 65536, ns), np.zeros(ns)], 1), 16
    return np.stack([rng.random(ns) * 1e-3, rng.normal(0, 1, ns), rng.random(ns) * 1e30,
                     rng.random(ns) * 1e-42, np.where(rng.random(ns) < 0.01, 1e20, 1e-3),
                     rng.integers(0, 9, ns) * 0.125, np.zeros(ns) - 0.0, np.full(ns, 3.4e38)],
                    1), 32


@pytest.mark.gpu
@pytest.mark.parametrize("ns", SIZES)
@pytest.mark.parametrize("kind", ["u8", "u16", "f32"])
def test_means_and_variances(gpu, oracle, kind, ns):
    from pulsarsr_gb300 import fbank, rfi, synth
    x, nbits = columns(kind, ns, np.random.default_rng(ns))
    raw = synth.header_bytes(x.shape[1], nbits, 64e-6, 1450.0, -1.0) + \
        synth.pack(x.astype(np.float32), nbits)
    m, v = rfi.channel_stats(fbank.decode(raw))
    _, d = oracle.decode(raw)
    om, ov = oracle.channel_stats(d)
    same = lambda a, b: (np.asarray(a).view(np.uint32) == np.asarray(b).view(np.uint32)) | \
        (np.isnan(a) & np.isnan(b))  # noqa: E731
    assert same(m, om).all(), (m, om)
    assert same(v, ov).all(), (v, ov)
