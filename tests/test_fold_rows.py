"""Refinements with as many trial periods as a fold launch takes (64), one more,
and several launches: the best profile and its statistics against the oracle."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [1, 62, 63, 64, 127, 128, 150])
def test_refine_row_batches(gpu, oracle, steps):
    from pulsarsr_gb300 import fold
    n, ts = 20000, 1e-3
    x = np.random.default_rng(steps).integers(0, 60, n).astype(np.float32)
    x[np.arange(n) % 37 < 3] += 9
    # the best period lies at either end of the span, so in the last launch too
    for f in (1 / 0.037 - 0.4 / n / ts, 1 / 0.037 + 0.4 / n / ts):
        r = fold.refine(x, ts, f, 0.45 / (n * ts), steps, 32)
        o = oracle.refine(x, ts, f, 0.45 / (n * ts), steps, 32)
        assert r["period_s"] == o["period_s"]
        assert np.array_equal(r["counts"], o["counts"])
        assert np.array_equal(r["bins"], o["bins"])
        # (statistics: f64 sums of bins in another order)
        assert np.isclose(r["reduced_chi_square"], o["reduced_chi_square"], rtol=1e-9)
