"""Twiddle tables on both sides of the size (2^17 points) from which they are made
by angle sums: raw power spectra bit for bit the oracle's."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [32768, 32769, 65536, 65537, 262145, 1048577])
def test_raw_power_across_table_forms(gpu, oracle, n):
    from pulsarsr_gb300 import search
    x = np.random.default_rng(n).integers(0, 255, n).astype(np.float32)
    got, want = search.raw_power(x), np.asarray(oracle.raw_power(x), np.float32)
    assert got.tobytes() == want.tobytes()
