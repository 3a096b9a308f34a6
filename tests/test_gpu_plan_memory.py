"""Plans within a bound of device memory (JUBIK_PLAN_MEMORY_MB, read at plan creation).

A plan that does not fit with the separable kernels' scratch takes kernels that need less,
whichever of its allocations is the one that fails; one that fits with neither raises
MemoryError.  What a plan took without the separable kernels (JUBIK_SEPARABLE=0) it fits in
with them.  Results of bounded plans agree with those of an unbounded one within twice the
tier of the precision (1e-12, 1e-6; gradients 1e-11 and 3e-6 of the cancelling term, which
for these sums is the gradient of constant counts).
"""
import numpy as np
import pytest
import torch

import jubik_gb300 as ju

pytestmark = pytest.mark.gpu

F32, F64 = torch.float32, torch.float64

# (dtype, field, patches per axis, margin, modules)
CASES = {"f32-P192-M1": (F32, 256, 4, 32, 1), "f32-P192-M3": (F32, 256, 4, 32, 3),
         "f64-P192-M2": (F64, 192, 3, 32, 2), "f32-P384-M2": (F32, 256, 2, 64, 2),
         "f32-P160-M7": (F32, 144, 3, 32, 7)}


class _Problem:
    def __init__(self, name):
        self.dtype, self.nx, self.n, self.margin, self.M = CASES[name]
        rng = np.random.default_rng(len(name))
        u = np.arange(2 * (self.nx // self.n)) - self.nx // self.n
        sig = rng.uniform(1.0, 4.0, size=(self.M, self.n ** 2, 1, 1, 1))
        self.psf = np.exp(-0.5 * (u[:, None] ** 2 + u[None, :] ** 2) / sig ** 2)
        self.sky = np.exp(rng.normal(size=(1, self.nx, self.nx)))
        self.data = rng.poisson(2.0, size=self.M * self.nx ** 2).astype(np.int32)

    def run(self, monkeypatch, mb=None):
        """(workspace, response, gradient, metric product) of a plan under the bound."""
        if mb is None:
            monkeypatch.delenv("JUBIK_PLAN_MEMORY_MB", raising=False)
        else:
            monkeypatch.setenv("JUBIK_PLAN_MEMORY_MB", f"{mb:.6f}")
        plan = ju.ResponsePlan(self.M, 1, (self.nx, self.nx), self.n, self.margin,
                               dtype=self.dtype)
        monkeypatch.delenv("JUBIK_PLAN_MEMORY_MB", raising=False)
        try:
            size = plan.workspace_bytes
            plan.set_psf(self.psf)
            lam = plan.response(self.sky)
            if mb is not None:  # (the counts' buffers belong to the bound too)
                return (size, lam.double().cpu().numpy())
            plan.set_data(self.data)
            g = plan.energy_and_grad(self.sky)[1]
            return (size, lam.double().cpu().numpy(), g.double().cpu().numpy(),
                    plan.metric(None, self.sky).double().cpu().numpy())
        finally:
            plan.close()


@pytest.mark.parametrize("name", list(CASES))
def test_bounded_plans_run_or_raise(cuda, name, monkeypatch):
    prob = _Problem(name)
    full = prob.run(monkeypatch)
    tol = 2e-12 if prob.dtype == F64 else 2e-6
    failed = False
    for share in np.linspace(1.0, 0.25, 26):
        mb = (share * full[0] + 64) / 1e6
        try:
            got = prob.run(monkeypatch, mb)
        except MemoryError as err:
            assert "JUBIK_PLAN_MEMORY_MB" in str(err)
            failed = True
            continue
        assert not failed, "a smaller bound fits where a larger one did not"
        assert got[0] <= mb * 1e6
        assert np.linalg.norm(got[1] - full[1]) < tol * np.linalg.norm(full[1])
    assert failed  # a quarter of the workspace holds neither


@pytest.mark.parametrize("name", list(CASES))
def test_memory_of_the_former_kernels_is_enough(cuda, name, monkeypatch):
    prob = _Problem(name)
    full = prob.run(monkeypatch)
    monkeypatch.setenv("JUBIK_SEPARABLE", "0")
    former = prob.run(monkeypatch)
    monkeypatch.delenv("JUBIK_SEPARABLE")
    got = prob.run(monkeypatch, (former[0] + 64) / 1e6)
    assert got[0] <= former[0] + 64
    tol = 2e-12 if prob.dtype == F64 else 2e-6
    assert np.linalg.norm(got[1] - full[1]) < tol * np.linalg.norm(full[1])


@pytest.mark.parametrize("name", list(CASES))
def test_workspace(cuda, name, monkeypatch):
    """The separable scratch takes two buffers, the slabs' and the rows'.  Against the former
    kernels' workspace it weighs most with one module, which had no module-shared buffers:
    4/3 of a spectrum per unit beside the spectrum itself, 1 + 4/3 over 1 + 5/9."""
    prob = _Problem(name)
    full = prob.run(monkeypatch)
    monkeypatch.setenv("JUBIK_SEPARABLE", "0")
    assert full[0] <= 1.5 * prob.run(monkeypatch)[0]


def test_longer_slabs_keep_captured_graphs_valid(cuda):
    """A shorter run takes larger slabs; a graph captured before goes on with its own."""
    rng = np.random.default_rng(3)
    nx, n = 256, 4
    u = np.arange(128) - 64
    psf = np.exp(-0.5 * (u[:, None] ** 2 + u[None, :] ** 2) / rng.uniform(
        1.0, 4.0, size=(2, n * n, 1, 1, 1)) ** 2)
    plan = ju.ResponsePlan(2, 1, (nx, nx), n, 32, dtype=F32)
    try:
        plan.set_psf(psf)
        x = torch.as_tensor(np.exp(rng.normal(size=(1, nx, nx))), dtype=F32, device=cuda)
        out = torch.empty((2, 1, nx, nx), dtype=F32, device=cuda)
        want = {}
        for r in (4, 1):
            plan.set_forward_run(r)
            want[r] = plan.psf_forward(x, out=out).clone()
        plan.set_forward_run(4)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            plan.psf_forward(x, out=out)
        plan.set_forward_run(1)
        assert torch.equal(plan.psf_forward(x, out=out), want[1])
        graph.replay()
        assert torch.equal(out, want[4])
    finally:
        plan.close()
