"""The fill values of masked blocks (channel medians by digits, over several
CTAs per channel) against the oracle: 16-bit and f32 samples around one and two
CTAs' shares (16,384 samples), even and odd counts, few values, equal values,
signed zeros, subnormals, extremes and medians at the ends of the key range."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("nbits", [16, 32])
@pytest.mark.parametrize("ns", [2, 3, 255, 16383, 16384, 16385, 40001])
def test_fill_values(gpu, oracle, nbits, ns):
    from pulsarsr_gb300 import fbank, rfi, synth
    rng = np.random.default_rng(ns + nbits)
    if nbits == 16:
        cols = [rng.integers(0, 65536, ns), rng.integers(100, 103, ns), np.full(ns, 65535),
                np.zeros(ns), rng.integers(0, 2, ns) * 65535, 2047 + rng.integers(0, 3, ns)]
    else:
        cols = [rng.normal(100, 10, ns), rng.normal(0, 1, ns), np.full(ns, -3.5),
                np.where(rng.random(ns) < 0.5, 0.0, -0.0), rng.random(ns) * 1e-41,
                rng.choice([-3e38, 3e38], ns), -rng.random(ns) * 1e20,
                rng.integers(0, 3, ns) * 0.5]
    x = np.stack(cols, 1).astype(np.float32)
    raw = synth.header_bytes(x.shape[1], nbits, 64e-6, 1500.0, -0.5) + synth.pack(x, nbits)
    fb = fbank.decode(raw)
    block = max(2, ns // 7)
    m = rfi.mask(fb, block, 0.5)  # a low threshold: channels and blocks are filled
    _, d = oracle.decode(raw)
    od, om = oracle.rfi_mask(d, block, 0.5)
    assert m.channels == [int(c) for c in om["channels"]]
    assert m.blocks == [int(b) for b in om["blocks"]]
    assert fb.data.tobytes() == np.ascontiguousarray(od).tobytes()
