"""The separable response at the edges of its geometry, against the float64 oracle.

Row spectra of every image row, column transforms per patch: fields that are no
multiple of the patch stride, odd strides (the last window starts early), odd
numbers of rows, one patch, more windows than a CTA holds at once, margins of
several strides (many overlapping patches), non-square fields, and every FFT
side of the separable kernels.

Tolerances are the tiers of the other parity tests: float64 1e-12 (gradient
1e-11), float32 1e-6; the float32 gradient R^T(1 - d/lam) is measured against the
cancelling term |R^T(d/lam)|, 3e-6.
"""
import numpy as np
import pytest
import torch

import jubik_oracle as O
import jubik_gb300 as ju
from jubik_gb300 import synthetic

F32, F64 = torch.float32, torch.float64

# (field, patches per axis, margin, modules, energies)
CASES = {
    "P160-18-windows-margin-19-strides": ((72, 72), 18, 76, 2, 1),
    "P160-17-windows": ((136, 136), 17, 72, 1, 2),
    "P192-odd-stride-clamped": ((189, 189), 3, 33, 3, 2),
    "P192-ragged-odd-field": ((197, 195), 3, 31, 2, 1),
    "P192-one-patch": ((64, 64), 1, 32, 1, 1),
    "P192-runs-of-4": ((256, 256), 4, 32, 9, 1),
    "P256-two-patches": ((101, 100), 2, 78, 2, 1),
    "P320-ragged": ((263, 262), 2, 29, 1, 2),
    "P384-three-patches": ((192, 192), 3, 128, 2, 1),
    "P512-one-patch": ((130, 130), 1, 126, 2, 1),
}


def _rel(a, b):
    a = a.detach().double().cpu().numpy() if isinstance(a, torch.Tensor) else np.asarray(a)
    a, b = a.ravel(), np.asarray(b, np.float64).ravel()
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _case(name):
    shape, n, margin, M, E = CASES[name]
    rng = np.random.default_rng(len(name))
    dx = shape[0] // n
    assert dx == shape[1] // n
    K = 2 * dx
    u = np.arange(K) - dx
    sig = rng.uniform(1.0, min(5.0, K / 6.0 + 0.6), size=(M, n * n, E, 1, 1))
    q = (u[:, None] - 0.3) ** 2 + 0.8 * (u[None, :] + 0.2) ** 2 + 0.2 * u[:, None] * u[None, :]
    psf = np.exp(-0.5 * q / sig ** 2) + 1e-4
    sky = np.exp(rng.normal(size=(E,) + shape))
    exposure = rng.uniform(0.5, 2.0, size=(M, E) + shape)
    keep = rng.random((M, E) + shape) > 0.05
    R = O.Response(O.Domain((E,) + shape, (1.0, 1.0, 1.0)), psf, n, margin, exposure * keep, keep,
                   pixel_area=0.7)
    return shape, n, margin, M, E, psf, sky, exposure * keep, keep, R, rng


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [F64, F32], ids=["f64", "f32"])
@pytest.mark.parametrize("name", list(CASES))
def test_edges_match_the_oracle(cuda, name, dtype):
    shape, n, margin, M, E, psf, sky, exposure, keep, R, rng = _case(name)
    lam = R(sky)
    data = [synthetic.poisson_data(l, 5 + i) for i, l in enumerate(lam)]
    e_ref, g_ref = R.energy_and_grad(sky, data)
    cancel = R.adjoint([d / l for d, l in zip(data, lam)])
    cot = rng.normal(size=(M, E) + shape)
    vec = rng.normal(size=sum(l.size for l in lam))
    v = rng.normal(size=sky.shape)
    plan = ju.ResponsePlan(M, E, shape, n, margin, dtype=dtype, pixel_area=0.7)
    try:
        plan.set_psf(psf).set_exposure(exposure, keep).set_data(np.concatenate(data))
        if "runs" in name and dtype == F32:
            plan.set_forward_run(4)
        tol = 1e-12 if dtype == F64 else 1e-6
        assert _rel(plan.psf_forward(sky), R.psf(sky)) < tol
        assert _rel(plan.psf_adjoint(cot), R.psf_adjoint(cot)) < tol
        assert _rel(plan.response(sky), np.concatenate(lam)) < tol
        parts = np.split(vec, np.cumsum([l.size for l in lam])[:-1])
        assert _rel(plan.response_vjp(vec), R.adjoint(parts)) < tol
        e, g = plan.energy_and_grad(sky)
        assert abs(float(e) - e_ref) <= tol * abs(e_ref)
        gd = g.double().cpu().numpy()
        if dtype == F64:
            assert _rel(gd, g_ref) < 1e-11
        else:
            assert np.linalg.norm(gd - g_ref) < 3e-6 * np.linalg.norm(cancel)
        assert _rel(plan.metric(None, v), R.metric(sky, v)) < 10 * tol
        e2, g2 = plan.energy_and_grad(sky)
        assert float(e2) == float(e) and torch.equal(g2, g)  # the same bits on every call
    finally:
        plan.close()


@pytest.mark.parametrize("name", list(CASES))
def test_cases_are_well_formed(name):
    """The oracle takes every case (CPU): finite, positive expected counts."""
    *_, sky, _, _, R, _ = _case(name)
    lam = np.concatenate(R(sky))
    assert np.all(np.isfinite(lam)) and np.all(lam > 0)


# (field side, patches per axis, margin, modules, energies): the library takes runs of
# 2 (P = 192, one module), 4 (P = 384, 1 and 3 modules) and no runs (odd n)
RUNS = [(1024, 16, 32, 1, 1), (1024, 8, 64, 1, 3), (1024, 8, 64, 3, 2), (448, 7, 32, 3, 2)]


@pytest.mark.gpu
@pytest.mark.parametrize("geom", RUNS, ids=lambda g: "x".join(map(str, g)))
def test_runs_of_the_library_match_float64(cuda, geom):
    """FP32 plans whose run length the library chooses, against a float64 plan."""
    nx, n, margin, M, E = geom
    rng = np.random.default_rng(nx + M)
    K = 2 * (nx // n)
    u = np.arange(K) - K // 2
    sig = rng.uniform(1.0, 5.0, size=(M, n * n, E, 1, 1))
    psf = np.exp(-0.5 * ((u[:, None] - 0.3) ** 2 + u[None, :] ** 2) / sig ** 2) + 1e-4
    sky = np.exp(rng.normal(size=(E, nx, nx)))
    data = rng.poisson(3.0, size=M * E * nx * nx).astype(np.int32)
    out = {}
    for dtype in (F64, F32):
        plan = ju.ResponsePlan(M, E, (nx, nx), n, margin, dtype=dtype)
        try:
            plan.set_psf(psf).set_data(data)
            lam = plan.response(sky)
            e, g = plan.energy_and_grad(sky)
            e2, g2 = plan.energy_and_grad(sky)
            assert float(e2) == float(e) and torch.equal(g2, g)
            out[dtype] = lam.double().cpu().numpy(), float(e), plan.metric(None, sky)
            out[dtype] += (plan.response_vjp(data / out[dtype][0].ravel()), g)
        finally:
            plan.close()
    (l64, e64, m64, c64, g64), (l32, e32, m32, _, g32) = out[F64], out[F32]
    assert _rel(l32, l64) < 1e-6
    assert abs(e32 - e64) <= 1e-6 * abs(e64)
    assert _rel(m32, m64.double().cpu().numpy()) < 1e-5
    assert float((g32.double() - g64).norm()) < 3e-6 * float(c64.norm())
