"""Device memory of the searches: what is only a faster way gives way where it does
not fit, and buffers that a plan no longer needs are returned."""
import ctypes as C

import numpy as np
import pytest

MIB = 1 << 20


def memory(limit=0):
    """(held, peak, cudaMalloc calls) of this thread's buffers since the last call; a
    limit in bytes from now on."""
    from pulsarsr_gb300._lib import check, lib
    v = [C.c_uint64() for _ in range(3)]
    check(lib().psr_test_device_memory(C.c_uint64(limit), *(C.byref(x) for x in v)))
    return tuple(int(x.value) for x in v)


@pytest.fixture
def observation(gpu):
    """64 8-bit channels x 60,000 samples and 48 trials a sample apart; all limits
    and widths back to their defaults afterwards."""
    from pulsarsr_gb300 import dedisperse, synth
    fb = synth.device(64, 8, 60000, 64e-6, 1500.0, -4.0, seed=3, noise_mean=100.0,
                      noise_sigma=20.0, pulsars=[synth.Pulsar(0.01, 20.0, 0.1, 3.0)])
    trials = dedisperse.dm_step(fb.header.frequencies(), 64e-6) * np.arange(48)
    yield fb, trials
    memory(0)
    dedisperse.set_subbands(-1)


def config():
    from pulsarsr_gb300 import search
    return search.Config(min_hz=2.0, max_hz=3000.0, threshold=7.0)


@pytest.mark.gpu
def test_plan_that_does_not_fit(observation):
    """The two-level plan's scratch past the memory left: channel by channel."""
    from pulsarsr_gb300 import dedisperse, search
    fb, trials = observation
    for call in (lambda: dedisperse.apply_trials(fb, trials, 50000),
                 lambda: search.search_trials(fb, trials, 50000, config())):
        dedisperse.set_subbands(0)
        held = memory()[0]
        want = call()
        need = memory()[1] - held
        dedisperse.set_subbands(4)
        with_plan = call()
        assert memory(held + need + MIB)[1] - held > need + MIB  # (the plan takes more)
        got = call()
        assert memory()[0] == held
        for w, p, g in zip(want, with_plan, got):
            assert np.asarray(w).tobytes() == np.asarray(p).tobytes()
            assert np.asarray(w).tobytes() == np.asarray(g).tobytes()


@pytest.mark.gpu
def test_plan_dropped(observation):
    """A batch prepared again without a plan gives the plan's buffers back."""
    from pulsarsr_gb300 import batch, dedisperse, fbank
    fb, trials = observation
    h = fbank.HeaderInfo(64, 8, 64e-6, 1500.0, -4.0, 0)
    obs = [dict(header=h, nsamples=60000, trials=trials, discovery=50000, config=config(),
                rfi_block=0)]
    held = {}
    for width in (0, 4):
        dedisperse.set_subbands(width)
        before = memory()[0]
        b = batch.Batch(obs)
        b.set_chunking(0, 48, 48)
        held[width] = memory()[0] - before
        if width == 4:
            assert held[4] > held[0] + MIB
            dedisperse.set_subbands(0)
            b.set_chunking(0, 48, 48)
            assert memory()[0] - before == held[0]
        del b


@pytest.mark.gpu
@pytest.mark.parametrize("budget", [48 * MIB, 96 * MIB])
def test_batch_budget(observation, budget):
    """A batch's scratch takes an eighth of the budget at most, whatever the number
    of observations, and lowers the trials per block for the rest."""
    from pulsarsr_gb300 import batch, dedisperse, fbank, search
    fb, trials = observation
    h = fbank.HeaderInfo(64, 8, 64e-6, 1500.0, -4.0, 0)
    obs = [dict(header=h, nsamples=60000, trials=trials, discovery=50000, config=config(),
                rfi_block=0)] * 3
    want = search.search_trials(fb, trials, 50000, config())
    held, tables = {}, MIB  # (a plan's tables and the rounding of its rows)
    for width in (0, 4):
        dedisperse.set_subbands(width)
        before = memory()[0]
        b = batch.Batch(obs, budget)
        held[width] = memory()[0] - before
        for i in range(3):
            b.load_fb(i, fb)
        b.run()
        b.sync()
        for i in range(3):
            counts, cands = b.candidates(i)
            assert np.array_equal(counts, want[0]) and cands.tobytes() == want[1].tobytes()
        del b
    assert held[4] - held[0] <= budget // 8 + 3 * tables


@pytest.mark.gpu
@pytest.mark.parametrize("nch,ntrials,length", [(2, 130, 300001), (1, 3, 17000001)])
def test_series_block(gpu, nch, ntrials, length):
    """Series with gaps between them are packed by blocks: no second copy of all
    of them, and one by one where there is no room for a block."""
    from pulsarsr_gb300 import dedisperse, synth
    ns = length + 200
    fb = synth.device(nch, 8, ns, 64e-6, 1500.0, -50.0, seed=5, noise_mean=100.0,
                      noise_sigma=20.0)
    trials = 0.1 * np.arange(ntrials)
    dedisperse.set_subbands(0)
    try:
        even = length + 63 - (length - 1) % 64
        want = dedisperse.apply_trials(fb, trials, even)[:, :length]
        series = ntrials * even * 4
        held = memory()[0]
        got = dedisperse.apply_trials(fb, trials, length)
        need = memory()[1] - held
        assert need < series + 64 * MIB + 4 * MIB
        assert np.array_equal(got, want)
        memory(held + series + 4 * MIB)
        assert np.array_equal(dedisperse.apply_trials(fb, trials, length), want)
    finally:
        memory(0)
        dedisperse.set_subbands(-1)


@pytest.mark.gpu
@pytest.mark.parametrize("harmonics", [16, 32])
def test_exact_lists_of_most_bins(observation, harmonics):
    """A threshold that half of the bins pass, with a birdie over the whole band (the
    gates do not look at birdies, the scores do): gate queues grow to every bin, the
    exact lists stay in their memory, taken by fewer trials at a time."""
    from pulsarsr_gb300 import search
    fb, trials = observation
    n, bins = 12000, 16385
    peak = {}
    for threshold in (60.0, 0.2):
        cfg = search.Config(min_hz=3.0, max_hz=7000.0, threshold=threshold,
                            max_harmonics=harmonics, birdies=[(3900.0, 3905.0)])
        held = memory()[0]
        counts, _ = search.search_trials(fb, trials, n, cfg)
        peak[threshold] = memory()[1] - held
        assert not counts.any()
    queues = 2 * len(trials) * (bins - bins // 4 - 1024) * 4
    assert queues <= peak[0.2] - peak[60.0] <= queues + MIB


@pytest.mark.gpu
def test_lists_of_many_chunks(gpu):
    """Raw lists that overflow in all of nine chunks grow for the first of them, not
    again for each; lists are those of the trials alone."""
    from pulsarsr_gb300 import dedisperse, search, synth
    fb = synth.device(4, 8, 101000, 64e-6, 1500.0, -20.0, seed=9, noise_mean=100.0,
                      noise_sigma=20.0)
    trials, n, peak = 0.01 * np.arange(2304), 100000, {}
    for threshold in (60.0, 2.5):
        cfg = search.Config(min_hz=3.0, max_hz=7000.0, threshold=threshold, max_candidates=24)
        held = memory()[0]
        counts, cands = search.search_trials(fb, trials, n, cfg)
        peak[threshold] = memory()[1] - held
    assert peak[2.5] - peak[60.0] <= 256 * (16 - 1) * 2048 * 24 + MIB
    at = np.concatenate([[0], np.cumsum(counts)]).astype(int)
    for i in (0, 255, 256, 1000, 2015, 2016, 2303):
        x = dedisperse.apply_trials(fb, trials[i:i + 1], n)[0]
        alone = search.periodicity(x, 64e-6, float(trials[i]), cfg)
        assert cands[at[i]:at[i + 1]].tobytes() == alone.tobytes(), i


@pytest.mark.gpu
def test_confirmation_of_a_session(observation):
    """A session's confirmation takes its temporary buffers from the pool, as a
    filterbank's does, and says the same."""
    from pulsarsr_gb300 import confirmation, fbank, search, session
    fb, trials = observation
    h = fbank.HeaderInfo(64, 8, 64e-6, 1500.0, -4.0, 0)
    s = session.SearchSession(h, 60000, trials, 50000, config(), 0, 8.0)
    s.load(np.rint(fb.data.T).astype(np.uint8).tobytes())
    s.run()
    s.sync()
    _, cands = s.candidates()
    memory()
    of_fb = confirmation.analyze(fb, trials, cands)
    calls = memory()[2]
    of_session = confirmation.analyze_session(s)
    assert memory()[2] <= calls
    assert len(of_fb.data) and of_fb.json() == of_session.json()


@pytest.mark.gpu
def test_freed_by_another_thread(gpu):
    """A handle made on one thread and closed on another, which goes on allocating."""
    import threading

    from pulsarsr_gb300 import synth

    def make():
        return synth.device(4, 8, 60000, 64e-6, 1500.0, -4.0, seed=3, noise_mean=100.0,
                            noise_sigma=20.0)

    fb, seen = make(), []

    def work():
        fb.close()
        seen.append(make().data.shape)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert seen == [(4, 60000)]
