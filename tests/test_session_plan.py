"""What a session reports of its dedispersion plan."""
import numpy as np
import pytest

from test_subband_plan import plan


@pytest.mark.gpu
@pytest.mark.parametrize("subbands", [0, 4, 8, -1])
def test_reported_plan(gpu, subbands):
    from pulsarsr_gb300 import dedisperse, fbank, search, session
    nch, n, ns = 96, 60000, 61000
    h = fbank.HeaderInfo(nch, 4, 72e-6, 1447.5, -1.0, 0)
    freqs = 1447.5 - np.arange(nch)
    trials = dedisperse.dm_step(freqs, 72e-6) * np.arange(200)
    d = np.stack([dedisperse.delays(freqs, 72e-6, float(t)) for t in trials])
    try:
        dedisperse.set_subbands(subbands)
        s = session.SearchSession(h, ns, trials, n, search.Config(min_hz=2.0), 0, 8.0)
        assert s.dedispersion() == plan(d, n, 15.0, subbands)[::3]
    finally:
        dedisperse.set_subbands(-1)
