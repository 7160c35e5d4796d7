"""The floor of a spectrum's scales, 1e-6 of its mean power (search/src/lib.rs:
53-54), where the powers' sum passes f32's range."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n,bins", [
    (4096, (20, 84, 148, 212)),          # one CTA per spectrum: warps 0, 2, 4, 6
    (16384, (300, 812, 1324, 1836)),     # one row group of the second pass, its four warps
    (524288, (20012, 20012 + 8192, 20012 + 16384, 20012 + 40960)),
])
def test_sum_past_f32(gpu, oracle, n, bins):
    """Tapered lines of power 0.8e38 (each line's sum is below f32's largest, all
    together are not) over noise well below the floor."""
    from pulsarsr_gb300 import search
    cfg = dict(min_hz=3.0, max_hz=7000.0, threshold=4.0, max_candidates=40)
    rng = np.random.default_rng(n)
    t = np.arange(n)
    x = np.sqrt(1e26 / n) * rng.normal(0, 1, n)
    for k in bins:
        x += 4.0 * np.sqrt(0.8e38) / n * np.hanning(n) * np.cos(np.pi * k * t / n + k)
    x = x.astype(np.float32)
    p = oracle.raw_power(x).astype(np.float64)
    assert np.isfinite(p).all() and p.sum() > 2 * float(np.finfo(np.float32).max)
    o = oracle.periodicity(x, 64e-6, 0.0, **cfg)
    assert len(o) > 0
    assert search.periodicity(x, 64e-6, 0.0, search.Config(**cfg)).tobytes() == o.tobytes()
