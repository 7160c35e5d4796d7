"""Timed cases of the pulsar search path, each through a public entry point.

A case is a dict of plain values; `kind` names the call a user makes:

  session      session.SearchSession: one packed observation from pinned host
               memory (unpack, RFI mask, every trial DM, candidate lists)
  batch        batch.Batch: a few observations of uneven shape in one graph
  trials       search.search_trials on a filterbank already in HBM (one DM
               block of a survey plan)
  periodicity  search.periodicity of one host series
  raw_power    search.raw_power of one host series
  dedisperse   dedisperse.apply_trials: the series of a DM range, to the host
  fold_refine  fold.refine: a frequency grid of folds of one host series
  analyze      confirmation.analyze of the candidates of one observation
  gradient     fold.refine_gradient of nearby starting points
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pulsarsr_gb300 import batch, confirmation, dedisperse, fbank, fold, search, session, synth

K_DM = 4148.808  # dispersion constant, s MHz^2 pc^-1 cm^3


# ------------------------------------------------------------------ cases
def listed():
    return [
        # A short low-resolution observation on a coarse DM grid: a quick look.
        dict(name="session_quick", kind="session", nch=64, nbits=8, ns=1 << 18, tsamp=64e-6,
             fch1=1450.0, bw=100.0, dm_max=120.0, ntrials=61, min_hz=15.0, rfi=True),
        # The shape of a GBT L-band observation searched over DM 0-500.
        dict(name="session_gbt", kind="session", nch=96, nbits=4, ns=531000, tsamp=72e-6,
             fch1=1447.5, bw=96.0, dm_max=500.0, ntrials=2000, min_hz=15.0, rfi=True),
        # A float filterbank as the reference's synth command writes it.
        dict(name="session_f32", kind="session", nch=32, nbits=32, ns=65536, tsamp=250e-6,
             fch1=1500.0, bw=100.0, dm_max=120.0, ntrials=61, min_hz=10.0, rfi=True),
        # A wide 8-bit observation of odd length, DM steps of one sample.
        dict(name="session_wide", kind="session", nch=512, nbits=8, ns=1047799, tsamp=100e-6,
             fch1=1600.0, bw=400.0, dm_max=0.0, ntrials=700, min_hz=1.0, rfi=True),
        # A night's uneven observations searched by one graph launch.
        dict(name="batch_uneven", kind="batch", nobs=4, shapes=3, max_ns=1 << 19,
             max_trials=700),
        # One DM block of a survey-scale plan (4096 channels, harmonic sums to 32).
        dict(name="trials_survey", kind="trials", nch=4096, nbits=8, ns=1 << 21, tsamp=64e-6,
             fch1=1600.0, bw=400.0, dm_min=60.0, dm_step=0.375, ntrials=300, harmonics=32),
        # One series already at hand: the smallest search call.
        dict(name="periodicity_short", kind="periodicity", n=32583, tsamp=250e-6),
        # The spectrum of one long dedispersed series.
        dict(name="power_long", kind="raw_power", n=3000001, tsamp=64e-6, nch=96),
        # The series around a candidate's DM, to look at or to fold elsewhere.
        dict(name="series_block", kind="dedisperse", nch=96, nbits=4, ns=531000, tsamp=72e-6,
             fch1=1447.5, bw=96.0, dm_min=55.0, dm_step=0.25, ntrials=21),
        # fold::refine as the confirmation step runs it: 41 frequencies.
        dict(name="fold_refine", kind="fold_refine", n=263571, tsamp=72e-6, nch=96,
             period=0.0046214, steps=40, bins=64),
        # The confirmation step of a GBT-shaped search: five families.
        dict(name="analyze_gbt", kind="analyze", nch=96, nbits=4, ns=531000, tsamp=72e-6,
             fch1=1447.5, bw=96.0, dm_max=500.0, ntrials=2000, limit=5, bins=64),
        # Gradient refinement of one pulsar's candidates on float data.
        dict(name="gradient_group", kind="gradient", nch=256, nbits=32, ns=1 << 20,
             tsamp=64e-6, fch1=1500.0, bw=400.0, ncand=16, bins=128, subints=64),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _odd(rng, lo, hi):
    return int(_log(rng, lo, hi)) | rng.randrange(2)


def draw(rng):
    kind = rng.choice(["session", "session", "session", "batch", "trials", "periodicity",
                       "raw_power", "dedisperse", "fold_refine", "analyze", "gradient"])
    tsamp = rng.choice([64e-6, 72e-6, 100e-6, 128e-6, 250e-6])
    if kind == "session":
        nbits = rng.choice([1, 2, 4, 4, 8, 8, 8, 16, 32])
        c = dict(kind=kind, nch=_odd(rng, 16, 700), nbits=nbits, ns=_odd(rng, 1 << 16, 1 << 20),
                 tsamp=tsamp, fch1=rng.choice([1450.0, 1600.0, 800.0]), bw=rng.choice([100.0, 300.0]),
                 dm_max=0.0, ntrials=_odd(rng, 16, 1500), min_hz=rng.choice([1.0, 15.0]),
                 rfi=rng.random() < 0.8)
        # (trials x channels x samples of a drawn search stay below 2e11)
        while c["ntrials"] > 16 and c["nch"] * c["ns"] * c["ntrials"] > 2e11:
            c["ntrials"] //= 2
        return c
    if kind == "batch":
        return dict(kind=kind, nobs=rng.randrange(2, 6), shapes=rng.randrange(100, 10000),
                    max_ns=int(_log(rng, 1 << 18, 1 << 19)), max_trials=rng.randrange(250, 700))
    if kind == "trials":
        return dict(kind=kind, nch=rng.choice([1024, 2048, 3000, 4096]), nbits=8,
                    ns=_odd(rng, 1 << 19, 1 << 21), tsamp=64e-6, fch1=1600.0, bw=400.0,
                    dm_min=rng.uniform(0.0, 150.0), dm_step=rng.choice([0.05, 0.375, 0.5]),
                    ntrials=_odd(rng, 40, 250), harmonics=rng.choice([16, 32]))
    if kind == "periodicity":
        return dict(kind=kind, n=_odd(rng, 3000, 1 << 19), tsamp=tsamp)
    if kind == "raw_power":
        return dict(kind=kind, n=_odd(rng, 5000, 3 << 20), tsamp=tsamp, nch=_odd(rng, 16, 512))
    if kind == "dedisperse":
        return dict(kind=kind, nch=_odd(rng, 16, 300), nbits=rng.choice([2, 4, 8, 8, 16, 32]),
                    ns=_odd(rng, 1 << 17, 1 << 20), tsamp=tsamp, fch1=1447.5, bw=96.0,
                    dm_min=rng.uniform(0.0, 100.0), dm_step=rng.choice([0.25, 1.0]),
                    ntrials=rng.randrange(1, 60))
    if kind == "fold_refine":
        return dict(kind=kind, n=_odd(rng, 20000, 1 << 21), tsamp=tsamp, nch=_odd(rng, 16, 512),
                    period=_log(rng, 0.0015, 2.0), steps=rng.choice([20, 40, 80]),
                    bins=rng.choice([32, 64, 100, 128]))
    if kind == "analyze":
        return dict(kind=kind, nch=_odd(rng, 32, 256), nbits=rng.choice([4, 8]),
                    ns=_odd(rng, 1 << 17, 1 << 20), tsamp=tsamp, fch1=1447.5, bw=96.0,
                    dm_max=rng.uniform(60.0, 200.0), ntrials=_odd(rng, 61, 1500),
                    limit=rng.randrange(1, 6), bins=rng.choice([32, 64, 128]))
    return dict(kind=kind, nch=_odd(rng, 64, 512), nbits=rng.choice([8, 32]),
                ns=_odd(rng, 1 << 19, 1 << 21), tsamp=64e-6, fch1=1500.0, bw=400.0,
                ncand=rng.randrange(1, 17), bins=128, subints=64)


# ----------------------------------------------------------------- inputs
def _freqs(c):
    return c["fch1"] - np.arange(c["nch"]) * (c["bw"] / c["nch"])


def _delays(freqs, tsamp, dm):
    """Whole-sample delays, rounded half away from zero."""
    x = K_DM * dm * (1.0 / (freqs * freqs) - 1.0 / (freqs.max() ** 2)) / tsamp
    return np.floor(np.maximum(x, 0.0) + 0.5).astype(np.int64)


def _trials(c):
    """The case's DM plan, its largest delay at most a sixth of the samples.
    dm_max 0: steps of one sample across the band."""
    freqs = _freqs(c)
    span = K_DM * (1.0 / freqs.min() ** 2 - 1.0 / freqs.max() ** 2) / c["tsamp"]
    if "dm_step" in c:
        t = c["dm_min"] + c["dm_step"] * np.arange(c["ntrials"])
    else:
        hi = c["dm_max"] or (c["ntrials"] - 1) / span
        t = np.linspace(0.0, hi, c["ntrials"]) if c["ntrials"] > 1 else np.array([hi])
    return t * min(1.0, c["ns"] / 6.0 / max(span * t[-1], 1e-9))


def _rng(seed, salt):
    return np.random.default_rng([int(seed) & 0xffffffff, salt])


def _pulsars(c, seed, dm_hi, count=2):
    r = _rng(seed, 1)
    return [synth.Pulsar(float(np.exp(r.uniform(np.log(0.004), np.log(0.2)))),
                         float(r.uniform(0.1, 0.9) * dm_hi), 0.05, float(r.uniform(0.1, 0.4)))
            for _ in range(count)]


def _samples(c, seed, pulsars):
    """Time-major samples [ns][nch] on the GPU: noise with channel gains, the
    pulsars, two interfering channels and a broadband burst."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    nch, ns, nbits = c["nch"], c["ns"], c["nbits"]
    mean, sigma, hi = {1: (0.5, 0.6, 1), 2: (1.5, 0.8, 3), 4: (8.0, 2.0, 15), 8: (100.0, 10.0, 255),
                       16: (3000.0, 200.0, 65535), 32: (100.0, 10.0, None)}[nbits]
    r = _rng(seed, 2)
    gain = torch.tensor(1.0 + 0.2 * (2 * r.random(nch) - 1), device="cuda", dtype=torch.float32)
    loud = r.integers(0, nch, 2)
    burst = int(r.integers(0, max(ns - 1000, 1)))
    freqs = torch.tensor(_freqs(c), device="cuda", dtype=torch.float64)
    kind = torch.float32 if nbits == 32 else torch.int32 if nbits == 16 else torch.uint8
    out = torch.empty(ns, nch, device="cuda", dtype=kind)
    step = max(1, (1 << 25) // nch)
    for a in range(0, ns, step):
        b = min(ns, a + step)
        t = torch.arange(a, b, device="cuda", dtype=torch.float64)[:, None] * c["tsamp"]
        x = torch.randn(b - a, nch, device="cuda", generator=g)
        for p in pulsars:
            td = t - K_DM * p.dm * (freqs ** -2 - freqs.max() ** -2)
            ph = torch.remainder(td / p.period_s - p.phase, 1.0).float()
            d = torch.minimum(ph, 1.0 - ph)
            x += p.amplitude * torch.exp(-0.5 * (d / (p.duty / 2.355)) ** 2)
        x[:, int(loud[0])] += 2.0 * torch.sin(2 * math.pi * 60.0 * t[:, 0]).float()
        x[:, int(loud[1])] *= 3.0
        lo, up = max(burst, a), min(burst + 1000, b)
        if lo < up:
            x[lo - a:up - a] += 2.0
        v = mean + sigma * gain * x
        out[a:b] = v if hi is None else torch.clamp(torch.round(v), 0, hi).to(kind)
    return out


def _payload(samples, nbits):
    """The packed bytes (least significant bits first) in pinned host memory."""
    if nbits == 32:
        b = samples.contiguous().view(torch.uint8).reshape(-1)
    elif nbits == 16:
        s = samples.reshape(-1)
        b = torch.stack([s & 255, s >> 8], 1).to(torch.uint8).reshape(-1)
    elif nbits == 8:
        b = samples.reshape(-1)
    else:
        per = 8 // nbits
        s = samples.reshape(-1)
        s = torch.nn.functional.pad(s, (0, -s.numel() % per)).reshape(-1, per)
        b = torch.zeros(s.shape[0], device="cuda", dtype=torch.uint8)
        for j in range(per):
            b |= s[:, j] << (j * nbits)
    host = torch.empty(b.numel(), dtype=torch.uint8, pin_memory=True)
    host.copy_(b)
    return host.numpy()


def _header(c):
    return fbank.HeaderInfo(c["nch"], c["nbits"], c["tsamp"], c["fch1"], -c["bw"] / c["nch"], 0)


def _discovery(c, trials):
    return (c["ns"] - 2 * int(_delays(_freqs(c), c["tsamp"], float(trials[-1])).max())) // 2


def _rfi_block(c):
    return max(int(0.1 / c["tsamp"]), 32)


def _series(c, seed):
    """A dedispersed integer-sample series (f32 sums over channels) with a
    pulse train, as float32 on the host."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    r = _rng(seed, 3)
    period = c.get("period", float(np.exp(r.uniform(np.log(0.004), np.log(0.5)))))
    t = torch.arange(c["n"], device="cuda", dtype=torch.float64) * c["tsamp"]
    ph = torch.remainder(t / period - float(r.random()), 1.0).float()
    d = torch.minimum(ph, 1.0 - ph)
    x = torch.randn(c["n"], device="cuda", generator=g) + 0.5 * torch.exp(-0.5 * (d / 0.02) ** 2)
    if "nch" not in c:  # a normalised float series
        return x.cpu().numpy()
    return torch.round(8.0 * c["nch"] + 2.0 * math.sqrt(c["nch"]) * x).cpu().numpy()


def _batch_shapes(c):
    r = np.random.default_rng(c["shapes"])
    out = []
    for _ in range(c["nobs"]):
        nch = int(r.choice([64, 128, 256, 512, 1024]))
        ns = int(np.exp(r.uniform(np.log(1 << 18), np.log(c["max_ns"] + 1))))
        out.append(dict(nch=nch, nbits=8, ns=ns, tsamp=float(r.uniform(64e-6, 256e-6)),
                        fch1=1600.0, bw=400.0, dm_max=0.0,
                        ntrials=int(r.integers(200, c["max_trials"] + 1))))
    return out


def _device_fb(c, seed, pulsars, rfi):
    mean, sigma = {4: (8.0, 2.0), 8: (128.0, 16.0), 32: (0.0, 1.0)}[c["nbits"]]
    fb = synth.device(c["nch"], c["nbits"], c["ns"], c["tsamp"], c["fch1"], -c["bw"] / c["nch"],
                      seed=int(seed) & 0xffffffff, noise_mean=mean, noise_sigma=sigma,
                      gain_spread=0.1, pulsars=pulsars)
    if rfi:
        synth.inject_rfi(fb, int(seed) & 0xffffffff, nb_channels=max(c["nch"] // 100, 1),
                         nb_amplitude=3 * sigma, nb_hz=50.0, nbursts=4, burst_samples=781,
                         burst_amplitude=2 * sigma)
    return fb


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "session":
        t = _trials(c)
        cfg = search.Config(min_hz=c["min_hz"], max_hz=2000.0, threshold=8.0, max_candidates=32)
        s = session.SearchSession(_header(c), c["ns"], t, _discovery(c, t), cfg,
                                  _rfi_block(c) if c["rfi"] else 0, 8.0)
        x = _samples(c, seed, _pulsars(c, seed, t[-1]))
        return dict(kind=kind, s=s, payload=_payload(x, c["nbits"]), nch=c["nch"],
                    nblocks=-(-c["ns"] // _rfi_block(c)))
    if kind == "batch":
        cfg = search.Config(min_hz=1.0, max_hz=2000.0, threshold=8.0, max_candidates=32)
        obs, pay = [], []
        for i, q in enumerate(_batch_shapes(c)):
            t = _trials(q)
            obs.append(dict(header=_header(q), nsamples=q["ns"], trials=t,
                            discovery=_discovery(q, t), config=cfg, rfi_block=_rfi_block(q),
                            rfi_threshold=8.0))
            k = int(seed) * 16 + i
            pay.append(_payload(_samples(q, k, _pulsars(q, k, t[-1])), 8))
        return dict(kind=kind, b=batch.Batch(obs), payloads=pay)
    if kind == "trials":
        t = _trials(c)
        return dict(kind=kind, fb=_device_fb(c, seed, _pulsars(c, seed, t[-1], 4), True), t=t,
                    n=_discovery(c, t),
                    cfg=search.Config(min_hz=1.0, max_hz=2000.0, threshold=8.0, max_candidates=32,
                                      max_harmonics=c["harmonics"]))
    if kind in ("periodicity", "raw_power"):
        return dict(kind=kind, x=_series(c, seed), tsamp=c["tsamp"])
    if kind == "fold_refine":
        return dict(kind=kind, x=_series(c, seed), c=c)
    if kind == "dedisperse":
        t = _trials(c)
        x = _samples(c, seed, _pulsars(c, seed, t[-1]))
        if c["nbits"] < 8:  # whole bytes
            x = x[:x.shape[0] // 8 * 8]
        raw = synth.header_bytes(c["nch"], c["nbits"], c["tsamp"], c["fch1"], -c["bw"] / c["nch"])
        fb = fbank.decode(raw + _payload(x, c["nbits"]).tobytes())
        return dict(kind=kind, fb=fb, t=t, n=_length(c, t))
    if kind == "analyze":
        t = _trials(c)
        ps = _pulsars(c, seed, t[-1], c["limit"])
        r = _rng(seed, 4)
        cands = [(1 / p.period_s * (1 + 1e-6 * r.normal()), p.period_s,
                  float(t[np.argmin(np.abs(t - p.dm))]), int(h), float(r.uniform(9, 60)))
                 for p in ps for h in (1, 4, 16)]
        return dict(kind=kind, fb=_device_fb(c, seed, ps, False), t=t, c=c,
                    cands=np.array(cands, dtype=search.CAND_DTYPE))
    ps = _pulsars(c, seed, 150.0, 1)  # gradient
    fb = _device_fb(c, seed, ps, False)
    freqs = _freqs(c)
    n = c["ns"] - int(_delays(freqs, c["tsamp"], 200.0).max()) - 4
    step = c["tsamp"] / (K_DM * (1 / freqs.min() ** 2 - 1 / freqs.max() ** 2))
    r = _rng(seed, 5)
    res = 1.0 / (n * c["tsamp"])
    starts = [(1 / (1 / ps[0].period_s + r.uniform(-2, 2) * res / 20), 0.0,
               ps[0].dm + r.uniform(-2, 2) * step / 2) for _ in range(c["ncand"])]
    return dict(kind=kind, fb=fb, n=n, starts=starts, c=c, window=5 * step)


def _length(c, t):
    ns = c["ns"] // 8 * 8 if c["nbits"] < 8 else c["ns"]
    return ns - int(_delays(_freqs(c), c["tsamp"], float(t[-1])).max())


# -------------------------------------------------------------- one pass
def _lists(counts, cands, most):
    """The counts per trial and the candidates' fields, zero past the last one."""
    full = np.zeros(len(counts) * most, dtype=cands.dtype)
    full[:len(cands)] = cands
    return dict(counts=counts, **{k: full[k] for k in cands.dtype.names})


def _flags(n, at):
    f = np.zeros(n, np.uint8)
    f[at] = 1
    return f


def run(state):
    s, kind = state, state["kind"]
    if kind == "session":
        s["s"].load(s["payload"])
        s["s"].run()
        s["s"].sync()
        m = s["s"].mask()
        return dict(_lists(*s["s"].candidates(), 32), channels=_flags(s["nch"], m["channels"]),
                    blocks=_flags(s["nblocks"], m["blocks"]), masked=m["masked_fraction"])
    if kind == "batch":
        b = s["b"]
        for i, p in enumerate(s["payloads"]):
            b.load(i, p)
        b.run()
        b.sync()
        return [_lists(*b.candidates(i), 32) for i in range(b.n)]
    if kind == "trials":
        return _lists(*search.search_trials(s["fb"], s["t"], s["n"], s["cfg"]), 32)
    if kind == "periodicity":
        out = search.periodicity(s["x"], s["tsamp"], 0.0,
                                 search.Config(min_hz=1.0, max_hz=2000.0, threshold=8.0))
        return _lists(np.array([len(out)]), out, 32)
    if kind == "raw_power":
        return search.raw_power(s["x"])
    if kind == "dedisperse":
        return dedisperse.apply_trials(s["fb"], s["t"], s["n"], with_sums=True)
    if kind == "fold_refine":
        c = s["c"]
        p = fold.refine(s["x"], c["tsamp"], 1.0 / c["period"], 1.0 / (c["n"] * c["tsamp"]),
                        c["steps"], c["bins"])
        p["counts"] = p["counts"].astype(np.int64)
        return p
    if kind == "analyze":
        o = confirmation.analyze(s["fb"], s["t"], s["cands"], s["c"]["limit"], s["c"]["bins"])
        return _outcome(o.data)
    out, J, ev = fold.refine_gradient(s["fb"], s["n"], s["starts"], s["c"]["bins"],
                                      s["c"]["subints"], dm_window=s["window"])
    return dict({k: np.ascontiguousarray(out[k]) for k in out.dtype.names}, J=J,
                evals=ev.astype(np.int64))


def _outcome(data):
    """The numbers of a confirmation report, field by field over its candidates."""
    cs = data["candidates"]

    def meas(m):
        return [m["snr"], m["mean_difference"], m["standard_error"]]

    def samples(m):
        return [m["on_samples"], m["off_samples"]]

    per = [c["time_parts"] + c["subbands"] + [c["validation"], c["zero_dm_validation"]]
           for c in cs]
    return dict(
        refined_dm=np.array([c["refined_dm"] for c in cs]),
        period=np.array([[c["profile"]["period_s"], c["zero_dm_period_s"]] for c in cs]),
        snr=np.array([[c["profile"]["snr"], c["profile"]["reduced_chi_square"]] for c in cs]),
        bins=np.array([c["profile"]["bins"] for c in cs], np.float32),
        counts=np.array([c["profile"]["counts"] for c in cs], np.int64),
        window=np.array([[c["window"]["start_bin"], c["window"]["width_bins"]] for c in cs]),
        measured=np.array([[meas(m) for m in p] for p in per]),
        samples=np.array([[samples(m) for m in p] for p in per], np.int64),
        contrast=np.array([[c["dm_contrast"], c["dispersion_widths"]] for c in cs]),
        time_profiles=np.array([c["time_profiles"] for c in cs], np.float32),
        subband_profiles=np.array([c["subband_profiles"] for c in cs], np.float32),
        response=np.array([[q["discovery_profile_response"] for q in c["dm_response"]]
                           for c in cs]),
        accepted=np.array([int(c["accepted"]) for c in cs]))


# ------------------------------------------------------------------ costs
def _pow2(n):
    return 1 << (int(n) - 1).bit_length()


def _search_work(c, t):
    n = _discovery(c, t)
    N = 2 * _pow2(n)
    return dict(bytes=c["nch"] * c["ns"] * c["nbits"] / 8 + 40.0 * len(t),
                flops=len(t) * (float(c["nch"]) * n + 2.5 * N * math.log2(N)))


def work(case):
    c, kind = case, case["kind"]
    if kind in ("session", "trials"):
        return _search_work(c, _trials(c))
    if kind == "batch":
        w = [_search_work(q, _trials(q)) for q in _batch_shapes(c)]
        return dict(bytes=sum(x["bytes"] for x in w), flops=sum(x["flops"] for x in w))
    if kind in ("periodicity", "raw_power"):
        N = 2 * _pow2(c["n"])
        return dict(bytes=4.0 * c["n"] + (2.0 * N if kind == "raw_power" else 0.0),
                    flops=2.5 * N * math.log2(N))
    if kind == "dedisperse":
        t = _trials(c)
        n = _length(c, t)
        return dict(bytes=c["nch"] * c["ns"] * c["nbits"] / 8 + 4.0 * n * len(t),
                    flops=float(c["nch"]) * n * len(t))
    if kind == "fold_refine":
        return dict(bytes=4.0 * c["n"], flops=2.0 * c["n"] * (c["steps"] + 1))
    size = {4: 1, 8: 1, 32: 4}[c["nbits"]]
    if kind == "analyze":  # per family: 21 half-step DMs, 41 + 41 + 21 folds
        n = _discovery(c, _trials(c))
        return dict(bytes=float(c["nch"]) * c["ns"] * size,
                    flops=c["limit"] * (23.0 * c["nch"] * n + 2.0 * n * (103 + c["nch"])))
    return dict(bytes=float(c["nch"]) * c["ns"] * size, flops=4.0 * c["nch"] * c["ns"])


# ------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """Candidate lists, confirmation reports and refined timings are decisions
    on thresholds, with no value in 64 bits beside them: None."""
    c, kind = case, case["kind"]
    if kind == "raw_power":
        x = _series(c, seed).astype(np.float64)
        z = torch.from_numpy(x - x.mean()).cuda()
        return torch.fft.rfft(z, 2 * _pow2(c["n"])).abs().square()
    if kind == "dedisperse":
        t = _trials(c)
        n = _length(c, t)
        x = _samples(c, seed, _pulsars(c, seed, t[-1])).double()
        out = torch.zeros(len(t), n, device="cuda", dtype=torch.float64)
        for i, dm in enumerate(t):
            for ch, d in enumerate(_delays(_freqs(c), c["tsamp"], float(dm))):
                out[i] += x[int(d):int(d) + n, ch]
        return out, out.sum(1)
    if kind == "fold_refine":
        return _exact_refine(c, _series(c, seed).astype(np.float64))
    return None


def _exact_refine(c, x):
    n, bins, steps = c["n"], c["bins"], c["steps"]
    f0, span = 1.0 / c["period"], 1.0 / (n * c["tsamp"])
    t = np.arange(n) * c["tsamp"]
    best = None
    for i in range(steps + 1):
        p = 1.0 / (f0 - span + 2.0 * span * i / steps)
        q = t / p
        b = np.minimum(((q - np.trunc(q)) * bins).astype(np.int64), bins - 1)
        cnt = np.bincount(b, minlength=bins)
        v = np.bincount(b, x, bins) / np.maximum(cnt, 1)
        chi = (cnt * (v - x.mean()) ** 2).sum() / x.var() / ((cnt > 0).sum() - 1)
        if best is None or chi >= best[0]:
            best = (chi, p, v, cnt)
    chi, p, v, cnt = best
    off = np.sort(v[cnt > 0])[:max((cnt > 0).sum() * 3 // 4, 1)]
    snr = (v.max() - np.sort(v)[bins // 2]) / off.std()
    return dict(period_s=p, snr=snr, reduced_chi_square=chi, bins=v, counts=cnt)
