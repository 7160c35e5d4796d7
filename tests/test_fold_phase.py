"""Folding and measuring with the fixed-point phase: bins and counts equal the
oracle's f64 ones, sample times on bin edges, long and short periods, offsets
and bin counts around the copies' limits included; integer and other series."""
import numpy as np
import pytest

PERIODS = {  # of tsamp 2^-14 s
    "edges": 64 * 2.0 ** -14,         # every sample on a bin edge of 64 bins
    "edges3": 96 * 2.0 ** -14,        # two thirds of a bin per sample
    "short": 1.7 * 2.0 ** -14,        # many cycles: wide margins
    "tiny": 3e-9,                     # more cycles than the fixed point allows for
    "pulsar": 0.0046214,
    "slow": 3.3,
    "beyond": 1e5,                    # everything in the first bins
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(PERIODS))
@pytest.mark.parametrize("bins", [4, 64, 100, 129, 257, 1024])
@pytest.mark.parametrize("kind", ["small", "large", "floats", "negative"])
def test_profile_matches_oracle(gpu, oracle, name, bins, kind):
    from pulsarsr_gb300 import fold
    rng = np.random.default_rng(bins)
    n = 20011
    x = {"small": rng.integers(0, 2000, n), "large": rng.integers(0, 1 << 24, n),
         "floats": rng.normal(0, 1, n), "negative": rng.integers(-5, 5, n)}[kind]
    x = x.astype(np.float32)
    for offset in (0, 123457):
        g = fold.profile_at(x, 2.0 ** -14, PERIODS[name], bins, offset)
        o = oracle.profile_at(x, 2.0 ** -14, PERIODS[name], bins, offset)
        assert np.array_equal(g["counts"], o["counts"])
        if kind != "floats":
            assert np.asarray(g["bins"]).tobytes() == np.asarray(o["bins"]).tobytes()
        # other values: f64 sums in another order, then rounded to f32
        np.testing.assert_allclose(g["bins"], o["bins"], rtol=2e-7, atol=1e-12)
        np.testing.assert_allclose(g["reduced_chi_square"], o["reduced_chi_square"], rtol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["integers", "floats"])
@pytest.mark.parametrize("window", [(0, 1, 4), (60, 10, 64), (0, 64, 64), (1023, 3, 1024)])
def test_measure_matches_oracle(gpu, oracle, kind, window):
    from pulsarsr_gb300 import fold
    rng = np.random.default_rng(5)
    x = rng.integers(0, 3000, 30011) if kind == "integers" else rng.normal(0, 1, 30011)
    x = x.astype(np.float32)
    for period in (64 * 2.0 ** -14, 0.0046214):
        g = fold.measure(x, 777, 2.0 ** -14, period, *window)
        o = oracle.measure(x, 777, 2.0 ** -14, period, *window)
        assert g == o
