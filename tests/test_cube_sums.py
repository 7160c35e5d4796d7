"""The channel sums behind the cube's variance keep what an f64 sum keeps: f32
samples whose sums and sums of squares are exact in f64 give the same objective
whatever order they come in."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("subints,length", [(1, 16384), (2, 8192)])
def test_order_of_periods(gpu, subints, length):
    """Periods of 256 samples at 16 bins, half of each in multiples of 2^7 up to 2^16
    and half in multiples of 2^-4 up to 2^5: every bin's sums are exact in f32 and
    the sum of squares in f64 (below 2^44, in units of 2^-8).  Whole periods change
    places inside each subint."""
    from pulsarsr_gb300 import fbank, fold, synth
    tsamp, period = 2.0 ** -12, 2.0 ** -4
    rng = np.random.default_rng(subints)
    npd = length // 256
    x = np.empty((subints, npd, 256))
    x[..., :128] = rng.integers(1, 512, (subints, npd, 128)) * 128.0
    x[..., 128:] = rng.integers(-512, 512, (subints, npd, 128)) / 16.0
    values = set()
    for _ in range(12):
        for s in range(subints):
            x[s] = x[s][rng.permutation(npd)]
        flat = np.append(x.ravel(), np.zeros(64)).astype(np.float32)[:, None]
        raw = synth.header_bytes(1, 32, tsamp, 1500.0, -1.0) + synth.pack(flat, 32)
        ref = (period, 0.0, 0.0)
        J, _ = fold.refine_cube_objective(fbank.decode(raw), x.size, ref, [ref], 16, subints)
        values.add(float(J[0]))
    assert len(values) == 1, values
