"""Limits of the two-level dedispersion's plan: what its launches cannot hold goes
by segments, or channel by channel."""
import ctypes as C

import numpy as np
import pytest

TILE, GRID = 1024, 65535


def plan(delays, n, max_value, subbands, chunk=256, once=False):
    """(width, flush, samples per segment, segments, scratch bytes)."""
    from pulsarsr_gb300._lib import check, lib
    d = np.ascontiguousarray(delays, dtype=np.uint32)
    info = (C.c_uint64 * 5)()
    check(lib().psr_test_subband_plan(d.ctypes.data_as(C.c_void_p), C.c_uint64(d.shape[1]),
                                      C.c_uint64(d.shape[0]), C.c_uint64(chunk), C.c_uint64(n),
                                      C.c_double(max_value), C.c_int(subbands),
                                      C.c_int(int(once)), info))
    return tuple(info)


@pytest.mark.parametrize("subbands", [4, -1])
@pytest.mark.parametrize("tiles", [1, GRID - 1, GRID, GRID + 1, 2 * GRID, 5 * GRID + 3])
def test_tiles_of_a_segment(subbands, tiles):
    """Few pattern rows over a long series: the scratch alone would allow segments
    of more tiles than a grid has."""
    n = tiles * TILE - 5
    width, _, seg, nseg, _ = plan(np.zeros((20, 8)), n, 255.0, subbands)
    assert width in (4, 8) and seg % TILE == 0 and seg // TILE <= GRID
    assert (nseg - 1) * seg < n <= nseg * seg


@pytest.mark.parametrize("delay,want", [(2 ** 31 - 1, 4), (2 ** 31, 0), (2 ** 32 - 1, 0)])
def test_delays_of_31_bits(delay, want):
    assert plan(np.full((3, 6), delay), 5000, 255.0, 4)[0] == want


@pytest.mark.gpu
def test_more_tiles_than_a_grid(gpu):
    from pulsarsr_gb300 import dedisperse, synth
    n = GRID * TILE + 5001
    fb = synth.device(2, 8, n + 100, 64e-6, 1500.0, -50.0, seed=1, noise_mean=128.0,
                      noise_sigma=50.0)
    try:
        out = []
        for width in (0, 4):
            dedisperse.set_subbands(width)
            out.append(dedisperse.apply_trials(fb, [0.0, 0.05], n, with_sums=True))
    finally:
        dedisperse.set_subbands(-1)
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
