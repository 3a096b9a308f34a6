"""Separable row kernels off their usual paths: log-sky rows of a padded array, fields so
wide that a CTA holds fewer than sixteen sequences, and fields too wide for it.

The log-sky case is compared with the float64 oracle at the tiers of the other parity tests
(1e-12 and 1e-6; gradients 1e-11 and 3e-6 of the cancelling term).  The wide fields are
compared with the kernels that share no transform code with the separable ones
(JUBIK_SEPARABLE=0), FP64 against FP64 within twice the 1e-12 tier, and the too wide one FP64
against the separable FP32 response at 1e-6.
"""
import numpy as np
import pytest
import torch

import jubik_oracle as O
import jubik_gb300 as ju
from jubik_gb300 import synthetic

pytestmark = pytest.mark.gpu

F32, F64 = torch.float32, torch.float64


@pytest.mark.parametrize("dtype", [F64, F32], ids=["f64", "f32"])
@pytest.mark.parametrize("geom", [(48, 32, 3, 2, 2), (63, 33, 3, 2, 1), (64, 64, 3, 1, 2),
                                  (128, 32, 2, 2, 1), (128, 64, 2, 1, 1)],
                         ids=["P160", "P192-odd", "P256", "P320", "P384"])
def test_log_sky_of_a_padded_array(cuda, geom, dtype):
    dx, margin, n, M, E = geom
    nx = n * dx + 1  # an odd number of rows
    rng = np.random.default_rng(dx)
    K = 2 * dx
    u = np.arange(K) - dx
    psf = np.exp(-0.5 * ((u[:, None] - 0.3) ** 2 + u[None, :] ** 2)
                 / rng.uniform(1.0, 4.0, size=(M, n * n, E, 1, 1)) ** 2)
    s = rng.normal(0.5, 0.8, size=(E + 1, nx + 7, nx + 4))
    x = np.exp(s[:E, :nx, :nx])
    exposure = rng.uniform(0.5, 2.0, size=(M, E, nx, nx))
    keep = rng.random((M, E, nx, nx)) > 0.05
    R = O.Response(O.Domain((E, nx, nx), (1.0, 1.0, 1.0)), psf, n, margin, exposure * keep, keep,
                   pixel_area=0.4)
    lam = R(x)
    data = [synthetic.poisson_data(l, 31 + i) for i, l in enumerate(lam)]
    energy, gx = R.energy_and_grad(x, data)
    want = np.zeros_like(s)
    want[:E, :nx, :nx] = x * gx
    cancel = np.linalg.norm(x * R.adjoint([d / l for d, l in zip(data, lam)]))
    plan = ju.ResponsePlan(M, E, (nx, nx), n, margin, dtype=dtype, pixel_area=0.4)
    try:
        plan.set_psf(psf).set_exposure(exposure * keep, keep).set_data(np.concatenate(data))
        e, g = plan.energy_and_grad_logsky(s)
        assert abs(float(e) - energy) <= (1e-12 if dtype == F64 else 1e-6) * abs(energy)
        err = np.linalg.norm(g.double().cpu().numpy() - want)
        assert err < (1e-11 * np.linalg.norm(want) if dtype == F64 else 3e-6 * cancel)
        outside = np.ones(s.shape, bool)
        outside[:E, :nx, :nx] = False
        assert not g.cpu().numpy()[outside].any()
        alone, _ = plan.energy_and_grad_logsky(s, need_grad=False)
        assert float(alone) == float(e)
    finally:
        plan.close()


def _wide(nx, n, margin, dtype, dev):
    """A plan on a wide field, a sky and a cotangent."""
    K = 2 * (nx // n)
    gen = torch.Generator(device=dev)
    gen.manual_seed(nx + margin)
    u = torch.arange(K, device=dev, dtype=dtype) - K // 2
    sig = 1.0 + 4.0 * torch.rand((1, n * n, 1, 1), generator=gen, device=dev, dtype=F64)
    psf = torch.exp(-0.5 * ((u[:, None] - 0.3) ** 2 + u[None, :] ** 2) / sig.to(dtype) ** 2)
    sky = torch.rand((1, nx, nx), generator=gen, device=dev, dtype=F64) + 0.1
    cot = torch.randn((1, 1, nx, nx), generator=gen, device=dev, dtype=F64)
    plan = ju.ResponsePlan(1, 1, (nx, nx), n, margin, dtype=dtype)
    plan.set_psf(psf)
    return plan, sky, cot


# 4096 columns: eight sequences of side 320 beside the FP64 rows (340 values each), eight of 512
@pytest.mark.parametrize("margin", [32, 128], ids=["P320", "P512"])
def test_fewer_sequences_beside_wide_rows(cuda, margin, monkeypatch):
    out = []
    for separable in ("1", "0"):
        monkeypatch.setenv("JUBIK_SEPARABLE", separable)
        plan, sky, cot = _wide(4096, 32, margin, F64, cuda)
        try:
            out.append((plan.psf_forward(sky), plan.psf_adjoint(cot)))
        finally:
            plan.close()
    for a, b in zip(*out):
        assert not torch.equal(a, b)
        assert float((a - b).norm()) < 2e-12 * float(b.norm())


def test_too_wide_fields_run_the_unfused_path(cuda, monkeypatch):
    """6144 FP64 columns with the overlap-add's compensation do not fit in shared memory."""
    nx, n, margin = 6144, 64, 32  # side 256
    plan, sky, cot = _wide(nx, n, margin, F64, cuda)
    try:
        wide = plan.psf_forward(sky), plan.psf_adjoint(cot)
        size = plan.workspace_bytes
    finally:
        plan.close()
    monkeypatch.setenv("JUBIK_SEPARABLE", "0")
    plan, _, _ = _wide(nx, n, margin, F64, cuda)
    try:
        assert plan.workspace_bytes == size
        assert torch.equal(plan.psf_forward(sky), wide[0])
        assert torch.equal(plan.psf_adjoint(cot), wide[1])
    finally:
        plan.close()
    monkeypatch.delenv("JUBIK_SEPARABLE")
    plan, _, _ = _wide(nx, n, margin, F32, cuda)
    try:
        for a, b in ((plan.psf_forward(sky), wide[0]), (plan.psf_adjoint(cot), wide[1])):
            assert float((a.double() - b).norm()) < 1e-6 * float(b.norm())
    finally:
        plan.close()
