"""The kernels behind the separable ones, and the two against each other.

A plan whose field is too wide for the separable row kernels, or whose memory does not hold
their scratch, runs the per-patch kernels at FFT sides 160 and 192 in FP32 and the unfused
path with its fused column stage elsewhere.  JUBIK_SEPARABLE=0 at plan creation gives every
plan those kernels.  They share no transform code with the separable ones, so each result is
compared with the float64 oracle and with the other kernels' result.

Tolerances are the tiers of the other parity tests: float64 1e-12 (gradient 1e-11), float32
1e-6, its gradient 3e-6 of the cancelling term R^T(d / lam); two results that each lie
within a tier lie within twice the tier of each other.
"""
import numpy as np
import pytest
import torch

import jubik_oracle as O
import jubik_gb300 as ju
from jubik_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu

F32, F64 = torch.float32, torch.float64

# (FFT side, patch stride, margin, patches per axis, modules)
SIDES = [(160, 48, 32, 3, 2), (192, 64, 32, 4, 2), (192, 64, 32, 3, 1), (256, 64, 64, 3, 2),
         (320, 128, 32, 3, 1), (384, 128, 64, 3, 2), (512, 128, 128, 2, 3)]


def _norm(a):
    return float(np.linalg.norm(np.asarray(a, np.float64).ravel()))


def _host(t):
    return t.detach().double().cpu().numpy().ravel()


def _results(inst, data, vec, dtype):
    plan = ju.ResponsePlan(inst.n_modules, inst.n_energies, inst.shape, inst.n_patches,
                           inst.margin, dtype=dtype)
    try:
        plan.set_psf(inst.psf).set_exposure(inst.exposure, inst.readmask).set_data(data)
        lam = plan.response(inst.sky)
        e, g = plan.energy_and_grad(inst.sky)
        again = plan.energy_and_grad(inst.sky)
        assert torch.equal(again[0], e) and torch.equal(again[1], g)
        return _host(lam), float(e), _host(g), _host(plan.response_vjp(vec))
    finally:
        plan.close()


@pytest.mark.parametrize("dtype", [F64, F32], ids=["f64", "f32"])
@pytest.mark.parametrize("side", SIDES, ids=lambda s: f"P{s[0]}M{s[4]}")
def test_both_kernels_match_the_oracle_and_each_other(cuda, side, dtype, monkeypatch):
    P, dx, margin, n, M = side
    nx = n * dx
    inst = synthetic.config2(nx=nx, dx=dx, margin=margin, n_modules=M, n_energies=1, seed=P + M)
    R = O.Response(O.Domain((1, nx, nx), (1.0, 1.0, 1.0)), inst.psf, n, margin, inst.exposure,
                   inst.readmask)
    lam = R(inst.sky)
    parts = [synthetic.poisson_data(l, 3 + i) for i, l in enumerate(lam)]
    data = np.concatenate(parts)
    vec = np.random.default_rng(P).normal(size=data.size)
    e_ref, g_ref = R.energy_and_grad(inst.sky, parts)
    cuts = np.cumsum([l.size for l in lam])[:-1]
    want = (np.concatenate(lam), e_ref, g_ref.ravel(),
            np.asarray(R.adjoint(np.split(vec, cuts))).ravel())
    cancel = _norm(R.adjoint([d / l for d, l in zip(parts, lam)]))
    tol = 1e-12 if dtype == F64 else 1e-6
    got = [_results(inst, data, vec, dtype)]
    monkeypatch.setenv("JUBIK_SEPARABLE", "0")
    got.append(_results(inst, data, vec, dtype))
    for a, b, f in ((got[0], want, 1), (got[1], want, 1), (got[0], got[1], 2)):
        assert _norm(a[0] - b[0]) < f * tol * _norm(want[0])
        assert abs(a[1] - b[1]) <= f * tol * abs(e_ref)
        if dtype == F64:
            assert _norm(a[2] - b[2]) < f * 1e-11 * _norm(g_ref)
        else:
            assert _norm(a[2] - b[2]) < f * 3e-6 * cancel
        assert _norm(a[3] - b[3]) < f * tol * _norm(want[3])
    # other kernels, so not the same bits
    assert not np.array_equal(got[0][0], got[1][0])


def test_run_lengths_without_the_separable_kernels(cuda, monkeypatch):
    """A run length set on a per-patch plan is the one its forward takes."""
    monkeypatch.setenv("JUBIK_SEPARABLE", "0")
    inst = synthetic.config2(nx=256, n_modules=2, n_energies=1, seed=4)
    plan = ju.ResponsePlan(2, 1, inst.shape, inst.n_patches, inst.margin, dtype=F32)
    try:
        plan.set_psf(inst.psf)
        out = {}
        for r in (1, 2, 4):
            plan.set_forward_run(r)
            assert plan.forward_run == r
            out[r] = _host(plan.psf_forward(inst.sky))
        for r in (2, 4):
            assert 0 < _norm(out[r] - out[1]) < 2e-7 * _norm(out[1])
        with pytest.raises(_lib.JubikUnsupported):
            ju.ResponsePlan(1, 1, inst.shape, inst.n_patches, inst.margin,
                            dtype=F32).set_forward_run(2)
    finally:
        plan.close()


@pytest.mark.parametrize("side", [(48, 16, 8), (224, 64, 48)], ids=["P48", "P224"])
def test_module_chunks_of_the_batched_transforms(cuda, side, monkeypatch):
    """FFT sides that no fused column stage covers give the same bits in one module chunk
    and in several, and the oracle's results."""
    P, dx, margin = side
    n, M = 3, 3
    inst = synthetic.config2(nx=n * dx, dx=dx, margin=margin, n_modules=M, n_energies=1, seed=P)
    R = O.Response(O.Domain((1, n * dx, n * dx), (1.0, 1.0, 1.0)), inst.psf, n, margin,
                   inst.exposure, inst.readmask)
    lam = R(inst.sky)
    parts = [synthetic.poisson_data(l, 3 + i) for i, l in enumerate(lam)]
    data = np.concatenate(parts)
    vec = np.random.default_rng(P).normal(size=data.size)
    _, g_ref = R.energy_and_grad(inst.sky, parts)
    one = _results(inst, data, vec, F64)
    assert _norm(one[0] - np.concatenate(lam)) < 1e-12 * _norm(np.concatenate(lam))
    assert _norm(one[2] - g_ref.ravel()) < 1e-11 * _norm(g_ref)
    for chunk in ("1", "2"):
        monkeypatch.setenv("JUBIK_PLAIN_CHUNK_MODULES", chunk)
        got = _results(inst, data, vec, F64)
        assert all(np.array_equal(a, b) for a, b in zip(got, one))
