"""Separable plans that take their modules in chunks: the same bits, with less memory.

JUBIK_PLAIN_CHUNK_MODULES bounds the modules in flight of a plan of the plain path, and a
plan of either path that does not fit with all of them at once takes one at a time.  The
adjoint's module sum and the likelihood's sums go from chunk to chunk, so every result has
the bits of an unchunked plan.
"""
import numpy as np
import pytest
import torch

import jubik_gb300 as ju

pytestmark = pytest.mark.gpu

F32, F64 = torch.float32, torch.float64

# (field, patches per axis, margin, modules, energies): FFT sides 160, 192 (runs), 256, 384
CASES = {"P160": (249, 5, 31, 3, 1), "P192-ragged": (197, 3, 31, 5, 2),
         "P192": (256, 4, 32, 5, 1), "P256": (192, 3, 64, 4, 1), "P384": (256, 2, 64, 3, 2)}


class _Run:
    def __init__(self, name, dtype, path):
        nx, n, margin, M, E = CASES[name]
        rng = np.random.default_rng(nx)
        u = np.arange(2 * (nx // n)) - nx // n
        sig = rng.uniform(1.0, 4.0, size=(M, n * n, E, 1, 1))
        psf = np.exp(-0.5 * (u[:, None] ** 2 + u[None, :] ** 2) / sig ** 2)
        full = (M, E, nx, nx)
        keep = rng.random(full) > 0.03
        x = np.exp(rng.normal(size=(E, nx, nx)))
        self.plan = plan = ju.ResponsePlan(M, E, (nx, nx), n, margin, dtype=dtype, path=path,
                                           pixel_area=0.7)
        try:
            self.size = plan.workspace_bytes
            plan.set_psf(psf).set_exposure(rng.uniform(0.5, 2.0, size=full), keep)
            plan.set_data(rng.poisson(2.0, size=int(keep.sum())).astype(np.int32))
            out = [plan.psf_forward(x), plan.psf_adjoint(rng.normal(size=full)), plan.response(x),
                   plan.response_vjp(rng.normal(size=int(keep.sum())))]
            out += list(plan.energy_and_grad(x))
            out += [plan.energy_and_grad(x, need_grad=False)[0], plan.metric(None, x),
                    plan.metric(0.5 * x, x)]
            out += list(plan.energy_and_grad_logsky(np.pad(np.log(x), ((0, 1), (0, 3), (0, 5)))))
            self.bits = [t.cpu() for t in out]
        finally:
            plan.close()


def _same(a, b):
    return all(torch.equal(p, q) for p, q in zip(a.bits, b.bits))


@pytest.mark.parametrize("dtype", [F64, F32], ids=["f64", "f32"])
@pytest.mark.parametrize("name", list(CASES))
def test_chunks_give_the_same_bits(cuda, name, dtype, monkeypatch):
    whole = _Run(name, dtype, "plain")
    assert all(bool(torch.isfinite(t).all()) for t in whole.bits)
    sizes = []
    for modules in (2, 1):
        monkeypatch.setenv("JUBIK_PLAIN_CHUNK_MODULES", str(modules))
        part = _Run(name, dtype, "plain")
        assert _same(part, whole)
        sizes.append(part.size)
    assert sizes[1] < sizes[0]
    if CASES[name][3] >= 5:  # (the sums between chunks weigh as much as a module's slabs)
        assert sizes[0] < whole.size


@pytest.mark.parametrize("path,dtype", [("auto", F32), ("plain", F32), ("auto", F64)])
def test_plans_short_of_memory_take_one_module_at_a_time(cuda, path, dtype, monkeypatch):
    whole = _Run("P192", dtype, path)
    monkeypatch.setenv("JUBIK_PLAIN_CHUNK_MODULES", "1")
    least = _Run("P192", dtype, "plain")
    monkeypatch.delenv("JUBIK_PLAIN_CHUNK_MODULES")
    assert least.size < whole.size
    monkeypatch.setenv("JUBIK_PLAN_MEMORY_MB", f"{(whole.size - 64) / 1e6:.6f}")
    plan = ju.ResponsePlan(5, 1, (256, 256), 4, 32, dtype=dtype, path=path)
    try:
        assert plan.workspace_bytes <= least.size
        rng = np.random.default_rng(1)
        u = np.arange(128) - 64
        psf = np.exp(-0.5 * (u[:, None] ** 2 + u[None, :] ** 2)
                     / rng.uniform(1.0, 4.0, size=(5, 16, 1, 1, 1)) ** 2)
        x = np.exp(rng.normal(size=(1, 256, 256)))
        got = plan.set_psf(psf).psf_forward(x), plan.psf_adjoint(plan.psf_forward(x))
    finally:
        plan.close()
    monkeypatch.delenv("JUBIK_PLAN_MEMORY_MB")
    plan = ju.ResponsePlan(5, 1, (256, 256), 4, 32, dtype=dtype, path=path)
    try:
        assert plan.workspace_bytes == whole.size
        plan.set_psf(psf)
        assert torch.equal(plan.psf_forward(x), got[0])
        assert torch.equal(plan.psf_adjoint(got[0]), got[1])
    finally:
        plan.close()
