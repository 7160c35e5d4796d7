"""The ends of the searched band against the oracle, bit for bit: a line on the
band's last bin, whose power the candidate one bin below takes as its score
(search/src/lib.rs:73-96), at every place that bin can have in the gate kernel's
groups of four bins, warps of 128 and blocks of 16,128."""
import numpy as np
import pytest

N_SAMPLES, TSAMP, THRESHOLD = 20000, 64e-6, 8.0
BIN_HZ = 1.0 / (65536 * TSAMP)
BLOCK = 252 * 64  # bins of a CTA


def sweep(bin_, seed):
    """Noise and a line at bin_ + 0.2 of rising strength, so that the power of
    bin_ passes the threshold before that of bin_ - 1."""
    rng = np.random.default_rng(seed)
    t = np.arange(N_SAMPLES)
    noise = rng.normal(500, 40, N_SAMPLES)
    line = np.cos(2 * np.pi * (bin_ + 0.2) * t / 65536 + rng.uniform(0, 2 * np.pi))
    for a in np.linspace(1.0, 3.0, 16):
        yield np.rint(8 * (noise + a * line)).astype(np.float32)


# lanes 0, 30 and 31 of a warp hold bins 3, 123 and 127 of its 128 last; the last
# groups of a block and the first of the next
ENDS = [7424 + k for k in (1, 2, 3, 4, 124, 125, 126, 127, 128)] + \
       [BLOCK + k for k in (-64, -4, -1, 0, 1, 2, 4)] + [2 * BLOCK]


@pytest.mark.gpu
@pytest.mark.parametrize("end", ENDS)
def test_line_on_the_last_bin(gpu, oracle, end):
    from pulsarsr_gb300 import search
    cfg = dict(min_hz=3.0, max_hz=(end + 0.5) * BIN_HZ, threshold=THRESHOLD, max_candidates=40)
    taken = 0  # candidates half a bin below the line's: the bin before it took its power
    for seed in range(3):
        for x in sweep(end, seed):
            c = search.periodicity(x, TSAMP, 0.0, search.Config(**cfg))
            o = oracle.periodicity(x, TSAMP, 0.0, **cfg)
            assert c.tobytes() == o.tobytes(), seed
            taken += int(np.any(np.abs(o["frequency_hz"] / BIN_HZ - (end - 0.5)) < 1e-6))
    assert taken > 0


@pytest.mark.gpu
@pytest.mark.parametrize("first", [512, 513, 514, 515, 635, 639, BLOCK - 1, BLOCK])
def test_line_on_the_first_bins(gpu, oracle, first):
    from pulsarsr_gb300 import search
    cfg = dict(min_hz=(first - 0.5) * BIN_HZ, max_hz=7000.0, threshold=THRESHOLD,
               max_candidates=40)
    for seed in range(2):
        for x in sweep(first + 1, seed):
            c = search.periodicity(x, TSAMP, 0.0, search.Config(**cfg))
            o = oracle.periodicity(x, TSAMP, 0.0, **cfg)
            assert c.tobytes() == o.tobytes(), seed
