"""Searches of several chunks whose candidate lists or gate queues overflow: each
chunk's lists are grown and made again (from the power spectra where they still
stand); every trial's list is that of its own series searched alone."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("ntrials", [40, 290, 600])
@pytest.mark.parametrize("threshold", [0.2, -0.8])
def test_every_chunk_overflows(gpu, ntrials, threshold):
    from pulsarsr_gb300 import dedisperse, search, synth
    fb = synth.device(12, 8, 15000, 64e-6, 1500.0, -20.0, seed=9, noise_mean=100.0,
                      noise_sigma=20.0, pulsars=[synth.Pulsar(0.0113, 30.0, 0.05, 2.0)])
    t = 0.4 * np.arange(ntrials)
    n = 12000
    cfg = search.Config(min_hz=3.0, max_hz=7000.0, threshold=threshold, max_candidates=24)
    counts, cands = search.search_trials(fb, t, n, cfg)
    x = dedisperse.apply_trials(fb, t, n)
    at = 0
    for i in range(ntrials):
        alone = search.periodicity(x[i], 64e-6, float(t[i]), cfg)
        got = cands[at:at + int(counts[i])]
        at += int(counts[i])
        assert got.tobytes() == alone.tobytes(), i
