"""Grouped passes at FFT sides 160 and 192, whose plans run the separable kernels alone.

A grouped pass runs the fused kernels on these plans, with buffers that a plan gets when it
first joins a group.  Problems of one and of several modules at both sides against the
float64 oracle, at the FP32 tiers of the parity tests (1e-6; the gradient 3e-6 of the
cancelling term R^T(d / lam)), and the path choice for grouped passes.
"""
import numpy as np
import pytest
import torch

import jubik_oracle as O
import jubik_gb300 as ju
from jubik_gb300 import synthetic

pytestmark = pytest.mark.gpu

# (stride, margin, patches per axis, modules, energies): sides 192, 192, 192, 160, 160
GEOMETRIES = [(64, 32, 3, 1, 2), (64, 32, 4, 2, 1), (60, 36, 3, 3, 2), (48, 32, 3, 1, 1),
              (48, 32, 4, 2, 2)]


@pytest.fixture(scope="module")
def problems():
    insts, refs = [], []
    for k, (dx, margin, n, M, E) in enumerate(GEOMETRIES):
        inst = synthetic.config2(nx=n * dx, dx=dx, margin=margin, n_modules=M, n_energies=E, seed=k)
        R = O.Response(O.Domain((E, n * dx, n * dx), (1.0, 1.0, 1.0)), inst.psf, n, margin,
                       inst.exposure, inst.readmask)
        lam = R(inst.sky)
        data = [synthetic.poisson_data(l, 60 + 7 * k + i) for i, l in enumerate(lam)]
        e, g = R.energy_and_grad(inst.sky, data)
        cancel = np.linalg.norm(R.adjoint([d / l for d, l in zip(data, lam)]))
        insts.append(inst)
        refs.append(dict(data=np.concatenate(data), energy=e, grad=g, cancel=cancel))
    return insts, refs


def test_grouped_passes_match_the_oracle(cuda, problems):
    insts, refs = problems
    b = ju.ProblemBatch(insts, dtype=torch.float32, n_streams=2)
    try:
        b.set_data([r["data"] for r in refs])
        before = [p.workspace_bytes for p in b.plans]
        b.energy_and_grad()
        assert [p.workspace_bytes for p in b.plans] == before
        assert b.group()
        # four classes: (192 and 160) x (one module, several)
        assert b.launches_per_pass() == 4 + 2 * (2 + 4)
        grown = [p.workspace_bytes for p in b.plans]
        assert all(g > w for g, w in zip(grown, before))
        assert b.group() and [p.workspace_bytes for p in b.plans] == grown
        first = None
        for run in ("eager", "graph", "again"):
            if run == "graph":
                b.capture()
            for t in b.grad:
                t.fill_(float("nan"))
            e, g = b.energy_and_grad() if run == "eager" else b.replay()
            torch.cuda.synchronize()
            bits = [e.clone()] + [t.clone() for t in g]
            first = first or bits
            assert all(torch.equal(p, q) for p, q in zip(bits, first)), run
            for k, r in enumerate(refs):
                assert abs(float(e[k]) - r["energy"]) <= 1e-6 * abs(r["energy"]), (run, k)
                err = np.linalg.norm(g[k].double().cpu().numpy() - r["grad"])
                assert err < 3e-6 * r["cancel"], (run, k)
        # one plan's pass after grouped ones: its own kernels, and the metric weights of either
        for k, (plan, r) in enumerate(zip(b.plans, refs)):
            v = torch.ones_like(b.x[k])
            grouped = plan.metric(None, v)
            e1, g1 = plan.energy_and_grad(b.x[k])
            assert abs(float(e1) - r["energy"]) <= 1e-6 * abs(r["energy"])
            assert np.linalg.norm(g1.double().cpu().numpy() - r["grad"]) < 3e-6 * r["cancel"]
            assert float((plan.metric(None, v) - grouped).norm()) < 1e-5 * float(grouped.norm())
    finally:
        b.close()


def test_autotune_for_grouped_passes_times_what_groups(cuda, problems):
    insts, refs = problems
    plain = synthetic.config2(nx=48, dx=16, margin=8, n_modules=1, n_energies=1)  # side 48
    b = ju.ProblemBatch(insts + [plain], dtype=torch.float32, n_streams=2)
    try:
        lam = b.expected_counts()
        b.set_data([r["data"] for r in refs] + [synthetic.poisson_data(lam[-1], 1)])
        chosen = b.autotune(reps=2, grouped=True)
        assert set(chosen) == {160, 192, 48}
        for side in (160, 192):  # the unfused path does not group
            assert set(b.timings[side]) == {"fused", "fused_unit"}
            assert chosen[side] in ("fused", "fused_unit")
        assert set(b.timings[48]) == {"plain"}
        e, _ = b.energy_and_grad()
        for k, r in enumerate(refs):
            assert abs(float(e[k]) - r["energy"]) <= 1e-6 * abs(r["energy"])
    finally:
        b.close()
