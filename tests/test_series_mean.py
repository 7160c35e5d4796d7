"""The f64 sum behind the mean periodicity subtracts, where its order matters:
equal to the sequential sum bit for bit whatever mixture of exact segments,
fine quanta, cancellations and binade crossings a series holds."""
import numpy as np
import pytest


def series(kind, n, rng):
    x = rng.normal(0, 1, n)
    if kind == "tiny":  # a few samples whose low bits cannot be kept
        x[rng.integers(0, n, max(n // 500, 2))] *= 1e-9
    if kind == "cancel":  # the running sum returns to small values
        x = np.where(np.arange(n) % 600 < 300, 1e7, -1e7) + rng.normal(0, 1e-3, n)
    if kind == "growing":
        x = np.exp(rng.uniform(-60, 60, n)) * np.sign(x)
    if kind == "integers":
        x = np.rint(500 + 30 * x)
    if kind == "zeros":
        x = np.where(rng.random(n) < 0.01, x, -0.0)
    return x.astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["noise", "tiny", "cancel", "growing", "integers", "zeros"])
@pytest.mark.parametrize("n", [2, 255, 256, 257, 8191, 8193, 100003])
def test_series_sum_is_sequential(gpu, oracle, kind, n):
    from pulsarsr_gb300 import dedisperse, fbank, search, synth
    x = series(kind, n, np.random.default_rng(n))
    want = float(np.add.accumulate(x.astype(np.float64))[-1])
    # one f32 channel at DM 0 is the series itself
    pad = np.concatenate([x, np.zeros(8, np.float32)])
    fb = fbank.decode(synth.header_bytes(1, 32, 64e-6, 1450.0, -1.0) + pad.tobytes())
    out, sums = dedisperse.apply_trials(fb, np.zeros(3), n, with_sums=True)
    assert out[0].tobytes() == (x + np.float32(0)).tobytes()
    assert [float(v) for v in sums] == [want] * 3
    assert search.raw_power(x).tobytes() == oracle.raw_power(x).tobytes()
