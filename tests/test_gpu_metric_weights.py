"""The quotients of a likelihood pass are those of the division, bit for bit.

A likelihood pass forms the metric weight eps^2 / lam and the residual's d / lam from one
reciprocal.  Two other passes divide: ``metric(x, v)`` forms the weight of a fresh lam in
the image pass, and ``poisson_energy`` the gradient 1 - d / lam of a lam vector, whose
transpose is the plan's gradient at unit exposure.  The lam of all three has the same bits,
so the results must have the same bits too: at FFT side 96 (the fused kernels' likelihood
pass) and at 160 .. 384 (the separable rows').

The scales of exposure and sky take the quotients through the range of the short form, over
its limits and to where eps^2 is nearly subnormal.
"""
import numpy as np
import pytest
import torch

import jubik_gb300 as ju
from jubik_gb300 import _lib
from jubik_gb300.plan import ptr, stream_handle

# (field, patches per axis, margin): FFT sides 96, 160, 192, 256, 384
GEOMETRIES = {96: (128, 4, 16), 160: (144, 3, 32), 192: (512, 8, 32), 256: (192, 3, 64),
              384: (256, 2, 64)}
# (exposure, sky): eps^2 and lam = eps * sky inside the limits 1e-18 .. 1e18, at and beyond them
SCALES = [(1.0, 1.0), (2e3, 2e-3), (1e-8, 1.0), (1e-9, 1e9), (9e8, 1e-8), (1e9, 1e8),
          (1e-18, 1e2), (3e-19, 1e8), (1e17, 1.0), (1e-17, 1e-2)]


def _case(side):
    nx, n, margin = GEOMETRIES[side]
    rng = np.random.default_rng(side)
    u = np.arange(2 * (nx // n)) - nx // n
    sig = rng.uniform(0.8, 2.0, size=(2, n * n, 1, 1, 1))
    psf = np.exp(-0.5 * (u[:, None] ** 2 + u[None, :] ** 2) / sig ** 2) + 1e-6
    plan = ju.ResponsePlan(2, 1, (nx, nx), n, margin, dtype=torch.float32)
    assert plan.P == side
    return plan.set_psf(psf), nx, rng


def _tensor(a, dev, dtype=torch.float32):
    return torch.as_tensor(a, dtype=dtype, device=dev)


@pytest.mark.gpu
@pytest.mark.parametrize("side", list(GEOMETRIES))
def test_metric_weights(cuda, side):
    plan, nx, rng = _case(side)
    try:
        v = _tensor(rng.normal(size=(1, nx, nx)), cuda)
        for eps, flux in SCALES:
            plan.set_exposure(_tensor(eps * np.exp(rng.uniform(-0.7, 0.7, (2, 1, nx, nx))), cuda))
            plan.set_data(rng.poisson(2.0, size=2 * nx * nx).astype(np.int32))
            x = _tensor(flux * np.exp(rng.normal(size=(1, nx, nx))), cuda)
            of_image = plan.metric(x, v)
            plan.energy_and_grad(x, need_grad=False)
            assert torch.equal(plan.metric(None, v), of_image), (eps, flux)
            assert bool(torch.isfinite(of_image).all())
    finally:
        plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("side", list(GEOMETRIES))
def test_residuals(cuda, side):
    plan, nx, rng = _case(side)
    try:
        for flux, top in ((1.0, 5), (1e-8, 3), (1e9, 2 ** 31 - 1), (1e-17, 2), (1e17, 9)):
            x = _tensor(flux * np.exp(rng.normal(size=(1, nx, nx))), cuda)
            d = _tensor(rng.integers(0, top, size=2 * nx * nx, endpoint=True), cuda, torch.int32)
            plan.set_data(d)
            lam = plan.response(x)
            res = torch.empty_like(lam)
            e = torch.empty((), dtype=torch.float64, device=cuda)
            _lib.call("jubik_poisson_energy", ptr(lam), ptr(d), lam.numel(), _lib.F32, ptr(e),
                      ptr(res), stream_handle(plan.device))
            _, g = plan.energy_and_grad(x)
            assert torch.equal(g, plan.response_vjp(res)), flux
    finally:
        plan.close()
