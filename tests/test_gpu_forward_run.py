"""``forward_run`` reports the run length that the forward takes, and 1 is always obeyed.

One-module plans and plans at FFT side 384 take runs by the library's choice; longer runs
than 1 are a setting of module-shared FP32 plans at side 192 only, but runs of 1 can be asked
of every plan.  A run sums the rows of its patches in another order, so the response's bits
tell which length ran.
"""
import numpy as np
import pytest
import torch

import jubik_gb300 as ju
from jubik_gb300 import _lib

pytestmark = pytest.mark.gpu

# (field, patches per axis, margin, modules, energies): enough patches for runs on a GPU of
# this class (more than two waves of CTAs)
RUNS = [(1024, 16, 32, 1, 1), (1024, 16, 32, 1, 3), (1024, 8, 64, 1, 3), (1024, 8, 64, 3, 2)]


@pytest.mark.parametrize("geom", RUNS, ids=lambda g: "x".join(map(str, g)))
def test_reported_run_is_the_one_taken(cuda, geom):
    nx, n, margin, M, E = geom
    rng = np.random.default_rng(nx + M)
    K = 2 * (nx // n)
    u = np.arange(K) - K // 2
    psf = np.exp(-0.5 * (u[:, None] ** 2 + u[None, :] ** 2)
                 / rng.uniform(1.0, 5.0, size=(M, n * n, 1, 1)) ** 2)
    sky = torch.as_tensor(np.exp(rng.normal(size=(E, nx, nx))), dtype=torch.float32, device=cuda)
    plan = ju.ResponsePlan(M, E, (nx, nx), n, margin, dtype=torch.float32)
    try:
        plan.set_psf(psf)
        assert plan.forward_run in (2, 4)
        chosen = plan.psf_forward(sky)
        plan.set_forward_run(1)
        assert plan.forward_run == 1
        single = plan.psf_forward(sky)
        assert not torch.equal(single, chosen)
        assert float((single - chosen).norm()) < 2e-7 * float(chosen.norm())
        with pytest.raises(_lib.JubikUnsupported):
            plan.set_forward_run(2)
        assert plan.forward_run == 1
        plan.set_forward_run(0)
        assert plan.forward_run in (2, 4)
        assert torch.equal(plan.psf_forward(sky), chosen)
    finally:
        plan.close()


def test_plans_without_runs_report_1(cuda):
    for shape, n, margin, dtype in (((128, 128), 4, 16, torch.float32),
                                    ((448, 448), 7, 32, torch.float32),
                                    ((1024, 1024), 16, 32, torch.float64)):
        plan = ju.ResponsePlan(1, 1, shape, n, margin, dtype=dtype)
        try:
            assert plan.forward_run == 1
            assert plan.set_forward_run(1).forward_run == 1
        finally:
            plan.close()


# (field, modules, energies, the library's run): FFT side 192 in strides of 64 rows.  A CTA of
# the forward's columns holds a run of patches and 8 of 96 columns, and an SM four CTAs; the
# longest of 4 and 2 that makes 1.5 waves (2 with fewer than three modules) is taken.
WAVES = [(1024, 7, 3, 4), (768, 3, 2, 2), (512, 7, 3, 2), (512, 2, 3, 1), (512, 3, 1, 1),
         (1024, 2, 1, 2)]


@pytest.mark.parametrize("geom", WAVES, ids=lambda g: "x".join(map(str, g)))
def test_library_choice_follows_the_waves(cuda, geom):
    nx, M, E, run = geom
    n, sms = nx // 64, torch.cuda.get_device_properties(cuda).multi_processor_count
    least = 1.5 if M >= 3 else 2.0
    fits = [r for r in (4, 2) if E * n * (n // r) * 12 / (4.0 * sms) >= least]
    if sms == 152:
        assert (fits or [1])[0] == run
    plan = ju.ResponsePlan(M, E, (nx, nx), n, 32, dtype=torch.float32)
    try:
        assert plan.forward_run == (fits or [1])[0]
    finally:
        plan.close()
