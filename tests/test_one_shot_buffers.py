"""Temporary buffers of the one-shot calls: results do not depend on what the
memory held before, on the sizes of the calls in between (below and above the
largest pooled block) or on calls that other threads make meanwhile."""
import threading

import numpy as np
import pytest


@pytest.mark.gpu
def test_repeated_and_threaded_calls_give_the_same_bytes(gpu):
    from pulsarsr_gb300 import dedisperse, fold, search, synth
    rng = np.random.default_rng(4)
    short = rng.integers(0, 255, 5001).astype(np.float32)
    mid = rng.normal(size=70001).astype(np.float32)
    long = rng.integers(0, 15, 16_000_001).astype(np.float32)  # 128 MiB of work: past the blocks
    cfg = search.Config(min_hz=2.0, max_hz=300.0, threshold=3.0)
    fb = synth.device(64, 8, 40000, 64e-6, 1500.0, -4.0, seed=2, noise_mean=128.0,
                      noise_sigma=50.0)
    dms = np.linspace(0.0, 40.0, 33)
    calls = [
        lambda: search.raw_power(short).tobytes(),
        lambda: search.raw_power(mid).tobytes(),
        lambda: repr(search.periodicity(mid, 1e-3, 0.0, cfg)),
        lambda: repr(fold.refine(short, 1e-3, 5.0, 0.05, 12, 32)),
        lambda: dedisperse.apply_trials(fb, dms, 30000).tobytes(),
    ]
    first = [c() for c in calls]
    big = search.raw_power(long).tobytes()
    assert [c() for c in reversed(calls)] == first[::-1]
    assert search.raw_power(long).tobytes() == big
    got, errors = {}, []

    def work(k):
        try:
            got[k] = [calls[(i + k) % len(calls)]() for i in range(3 * len(calls))]
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for k, out in got.items():
        assert out == [first[(i + k) % len(calls)] for i in range(len(out))]
