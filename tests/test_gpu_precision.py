"""The separable kernels are no less accurate than the per-patch ones.

At FFT sides 160 and 192 the per-patch kernels (``path="fused_unit"``) transform every
patch by itself and add the patches exactly, in two words.  The separable kernels add
vertically overlapping patches before the row transforms, so that a row transform's rounding
is no longer averaged over the patches; two-word sums, exact window weights and PSF spectra
that take back the transforms' gain have to make up for it.  Both are compared with the
float64 oracle on the same FP32 inputs: the separable error may exceed the per-patch one by
5 % at most, the scatter of the ratio of two errors between inputs.  (The gradient and the
metric product follow from these two maps; 1 / lam lets a few faint pixels decide their
errors, whose ratio scatters by a factor of two.)
"""
import numpy as np
import pytest
import torch

import jubik_oracle as O
import jubik_gb300 as ju
from jubik_gb300 import synthetic

# (field, patches per axis, margin, modules, energies); 398 and 249: no whole strides
CASES = {"P192": (384, 6, 32, 2, 1), "P192-one-module": (384, 6, 32, 1, 2),
         "P192-ragged": (398, 6, 30, 3, 1), "P160": (288, 6, 32, 3, 1),
         "P160-odd-stride": (249, 5, 31, 2, 1)}


def _err(a, b):
    a = a.detach().double().cpu().numpy().ravel()
    b = np.asarray(b, np.float64).ravel()
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CASES))
def test_errors_do_not_exceed_the_per_patch_kernels(cuda, name):
    nx, n, margin, M, E = CASES[name]
    rng = np.random.default_rng(nx + M)
    K = 2 * (nx // n)
    u = np.arange(K) - K // 2

    def f32(a):
        return np.asarray(a, np.float32).astype(np.float64)

    sig = rng.uniform(1.0, 5.0, size=(M, n * n, E, 1, 1))
    q = (u[:, None] - 0.3) ** 2 + 0.8 * (u[None, :] + 0.2) ** 2
    psf = f32((1.0 + q / sig ** 2) ** -2.5)
    smooth = np.stack([synthetic.grf((nx, nx), rng, mean=1.0) for _ in range(E)])
    sky = f32(np.exp(smooth))
    exposure = f32(rng.uniform(0.5, 2.0, size=(M, E, nx, nx)))
    keep = np.ones((M, E, nx, nx), bool)
    R = O.Response(O.Domain((E, nx, nx), (1.0, 1.0, 1.0)), psf, n, margin, exposure, keep)
    lam = R(sky)
    vec = [f32(rng.normal(size=l.size)) for l in lam]
    want = {"response": np.concatenate(lam), "vjp": R.adjoint(vec)}
    errors = {}
    for path in ("fused_unit", "auto"):
        plan = ju.ResponsePlan(M, E, (nx, nx), n, margin, dtype=torch.float32, path=path)
        try:
            plan.set_psf(psf).set_exposure(exposure, keep)
            got = {"response": plan.response(sky), "vjp": plan.response_vjp(np.concatenate(vec))}
            errors[path] = {k: _err(got[k], want[k]) for k in want}
        finally:
            plan.close()
    for k in want:
        assert errors["auto"][k] <= 1.05 * errors["fused_unit"][k], (k, errors)
