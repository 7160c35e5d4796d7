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


def delay_table(nch, trials, fch1=1500.0, bw=300.0, tsamp=64e-6):
    f = fch1 - np.arange(nch) * (bw / nch)
    x = 4148.808 * np.asarray(trials)[:, None] * (1 / f ** 2 - 1 / f[0] ** 2) / tsamp
    return np.floor(x + 0.5).astype(np.uint32)


@pytest.mark.parametrize("nbits,nch", [(1, 9), (2, 64), (4, 97), (4, 8), (8, 5), (8, 256),
                                       (8, 261), (8, 1030)])
def test_widths_are_taken(nbits, nch):
    """The plans of tests/test_dedisperse_two_level.py are there at the widths it asks
    for, with flushes past 65,535; its long case takes several segments."""
    step = 1.0 / (4148.808 * (1 / 1200.0 ** 2 - 1 / 1500.0 ** 2) / 64e-6)
    maxv = 2.0 ** nbits - 1
    for order in (np.arange(37), np.arange(40, 0, -1) * 0.5, np.repeat(np.arange(9), 3)):
        for width in (4, 8):
            w, flush, _, nseg, _ = plan(delay_table(nch, step * order), 9000, maxv, width,
                                        chunk=len(order), once=True)
            assert (w, flush, nseg) == (width, int(nch * maxv > 65535), 1)
    if nch == 1030:
        t = delay_table(1024, 400 * step + step * np.arange(100))
        w, _, _, nseg, _ = plan(t, 399491, 255.0, 8, chunk=100, once=True)
        assert w == 8 and nseg > 1


# a search that the plan's own choice takes in two levels, in five blocks of trials
AUTO = dict(nch=96, ntrials=300, chunk=64, n=100000)


def test_own_choice():
    step = 1.0 / (4148.808 * (1 / 1200.0 ** 2 - 1 / 1500.0 ** 2) / 64e-6)
    t = delay_table(AUTO["nch"], step * np.arange(AUTO["ntrials"]))
    assert plan(t, AUTO["n"], 255.0, -1, chunk=AUTO["chunk"])[0] in (4, 8)
    assert plan(t, 1000, 255.0, -1, once=True)[0] == 0  # (does not pay for one short pass)


@pytest.mark.gpu
def test_own_choice_over_blocks(gpu):
    """The chosen plan (whose middle block reuses the patterns it was chosen by)
    against channel by channel, over blocks with a short last one."""
    from pulsarsr_gb300 import batch, dedisperse, fbank, search, synth
    nch, n = AUTO["nch"], AUTO["n"]
    fb = synth.device(nch, 8, n + 500, 64e-6, 1500.0, -300.0 / nch, seed=2, noise_mean=100.0,
                      noise_sigma=20.0, pulsars=[synth.Pulsar(0.02, 2.0, 0.1, 1.0)])
    step = dedisperse.dm_step(fb.header.frequencies(), 64e-6)
    cfg = search.Config(min_hz=2.0, max_hz=3000.0, threshold=4.0)
    b = batch.Batch([dict(header=fbank.HeaderInfo(nch, 8, 64e-6, 1500.0, -300.0 / nch, 0),
                          nsamples=n + 500, trials=step * np.arange(AUTO["ntrials"]),
                          discovery=n, config=cfg, rfi_block=0)])
    b.load_fb(0, fb)
    got = {}
    try:
        for width in (0, -1):
            dedisperse.set_subbands(width)
            b.set_chunking(0, AUTO["chunk"], 0)
            b.run()
            b.sync()
            got[width] = b.candidates(0)
    finally:
        dedisperse.set_subbands(-1)
    assert got[0][0].sum() > 0 and np.array_equal(got[0][0], got[-1][0])
    assert got[0][1].tobytes() == got[-1][1].tobytes()
