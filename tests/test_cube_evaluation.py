"""The cube's harmonic sums and adjoint over the forms their kernels split:
power-of-two and other bin counts, more harmonics than threads, rows that do not
fill a block, odd candidate counts and more candidates than a launch takes.
Bounds as in tests/test_refine_cube.py (f32 cells and rotations against the FP64
model)."""
import numpy as np
import pytest

import test_refine_cube as model


@pytest.mark.gpu
@pytest.mark.parametrize("bins,subints,nch,npoints", [
    (128, 64, 5, 16), (128, 10, 31, 65), (96, 7, 9, 3), (45, 12, 11, 2), (8, 1, 3, 1),
    (256, 5, 13, 130)])
def test_cube_objective_forms(gpu, monkeypatch, bins, subints, nch, npoints):
    from pulsarsr_gb300 import fold, synth
    monkeypatch.setattr(model, "B", bins)
    monkeypatch.setattr(model, "S", subints)
    P, Pd, DM = 0.0237, -1e-9, 57.3
    fb = synth.device(nch, 32, 1 << 16, 64e-6, 1500.0, -400.0 / nch, seed=5, noise_mean=0.0,
                      noise_sigma=1.0, pulsars=[synth.Pulsar(P, DM, 0.05, 0.5, phase=0.2,
                                                             pdot=Pd)])
    freqs = fb.header.frequencies()
    n = (1 << 16) - 3001
    ref = (P, Pd, DM)
    R, v = model.cube_f64(fb.data, freqs, 64e-6, n, ref)
    base = np.array(ref)
    rng = np.random.default_rng(bins)
    pts = [base + model.steps(freqs, 64e-6, n, base, 0.5) * rng.uniform(-1, 1, 3)
           for _ in range(npoints)]
    J, g = fold.refine_cube_objective(fb, n, ref, pts, bins, subints)
    for i, th in enumerate(pts):
        Jm, gm = model.objective_f64(R, v, freqs, 64e-6, n, ref, th)
        assert np.isclose(J[i], Jm, rtol=3e-6), (i, J[i], Jm)
        h = model.steps(freqs, 64e-6, n, th, 1.0)
        scale = np.abs(gm * h).max()
        assert np.allclose(g[i] * h, gm * h, rtol=0, atol=1e-3 * scale), (i, g[i] * h, gm * h)


@pytest.mark.gpu
def test_adjoint_of_more_harmonics_than_threads(gpu, monkeypatch):
    """512 harmonics: the adjoint against central differences of the device's own
    objective (the FP64 model does not share the f32 walk of 2.8 bins per sample
    that folds 1024 bins)."""
    from pulsarsr_gb300 import fold, synth
    bins, subints, nch = 1024, 3, 4
    monkeypatch.setattr(model, "B", 128)  # steps of 0.01 of a 128-bin bin
    P, Pd, DM = 0.0237, -1e-9, 57.3
    fb = synth.device(nch, 32, 1 << 16, 64e-6, 1500.0, -400.0 / nch, seed=5, noise_mean=0.0,
                      noise_sigma=1.0, pulsars=[synth.Pulsar(P, DM, 0.05, 0.5, phase=0.2,
                                                             pdot=Pd)])
    freqs = fb.header.frequencies()
    n = (1 << 16) - 3001
    ref = (P, Pd, DM)
    th = np.array(ref) + model.steps(freqs, 64e-6, n, np.array(ref), 0.3)
    h = model.steps(freqs, 64e-6, n, th, 1e-2)
    e = np.diag(h)
    J, g = fold.refine_cube_objective(fb, n, ref, [th] + [th + s * e[j] for j in range(3)
                                                          for s in (1, -1)], bins, subints)
    fd = (J[1::2] - J[2::2]) / 2.0
    scale = np.abs(g[0] * h).max()
    assert np.allclose(g[0] * h, fd, rtol=0, atol=2e-2 * scale), (g[0] * h, fd)
