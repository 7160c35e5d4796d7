"""Scales, gates, harmonic filter, exact scores and selection where their rules
change, against the oracle: candidate lists bit for bit."""
import numpy as np
import pytest


def series(kind, n, rng):
    t = np.arange(n)
    if kind == "white":
        return np.rint(rng.normal(500, 40, n))
    if kind == "red":  # steep spectrum: window medians far from their neighbours'
        return np.rint(np.cumsum(rng.normal(0, 3, n)) + 1000)
    if kind == "comb":  # hundreds of harmonics: long candidate lists, many near-equal
        return np.rint(rng.normal(500, 20, n) + 300 * (np.mod(t, 211.37) < 3))
    if kind == "tones":  # exact bin centres and exact half bins: clamped and zero offsets
        N = 2 * (1 << (n - 1).bit_length())
        return 500 + 50 * np.sin(2 * np.pi * 400 * t / N) + 50 * np.sin(2 * np.pi * 800.5 * t / N)
    if kind == "step":  # zero half: flat spectrum next to strong lines
        return np.where(t < n // 2, 0.0, np.rint(rng.normal(500, 5, n)))
    return np.where(t == n // 3, 1e6, 0.0)  # one impulse: equal power in every bin


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["white", "red", "comb", "tones", "step", "impulse"])
@pytest.mark.parametrize("n", [513, 5000, 70001])
@pytest.mark.parametrize("threshold,harmonics", [(6.0, 16), (2.5, 32), (0.0, 16), (-3.0, 16)])
def test_candidates_match_oracle(gpu, oracle, kind, n, threshold, harmonics):
    """Thresholds down to ones that every bin reaches (lists past the sort's
    capacity, queues past their first size), with and without birdies."""
    from pulsarsr_gb300 import search
    x = series(kind, n, np.random.default_rng(n)).astype(np.float32)
    cfg = dict(min_hz=3.0, max_hz=7000.0, threshold=threshold, max_candidates=40,
               max_harmonics=harmonics)
    for birdies in ([], [(60.0, 5.0), (1000.0, 40.0)]):
        c = search.periodicity(x, 64e-6, 3.0, search.Config(**cfg, birdies=birdies))
        o = oracle.periodicity(x, 64e-6, 3.0, **cfg, birdies=birdies)
        assert c.tobytes() == o.tobytes(), birdies
