"""The fixed-point phase of a fold: the exact ratio, and the f64 operations for
every sample where there is none, the same on every host."""
import ctypes as C
from fractions import Fraction

import pytest

ALWAYS_F64 = 1 << 31


def phase(tsamp, period, last=1000, bins=64):
    from pulsarsr_gb300._lib import check, lib
    out = (C.c_uint64 * 3)()
    check(lib().psr_test_fold_phase(C.c_double(tsamp), C.c_double(period), C.c_uint64(last),
                                    C.c_uint64(bins), out))
    return (out[0] << 64) + out[1], out[2]


@pytest.mark.parametrize("tsamp,period", [(2.0 ** -14, 0.0046214), (72e-6, 3.3), (1.0, 0.3),
                                          (64e-6, 1e5)])
def test_ratio(tsamp, period):
    f, margin = phase(tsamp, period)
    exact = Fraction(tsamp) / Fraction(period) % 1
    assert abs(Fraction(f, 2 ** 128) - exact) < Fraction(1, 2 ** 100)
    assert 64 <= margin < 128


@pytest.mark.parametrize("tsamp,period", [(-2.0 ** -14, 0.0046214), (-1.0, 1e-9),
                                          (float("nan"), 1.0), (float("inf"), 1.0),
                                          (1.0, 1e-310)])
def test_no_ratio(tsamp, period):
    assert phase(tsamp, period) == (0, ALWAYS_F64)
