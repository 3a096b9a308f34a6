"""The calls whose time matters to a user of the response, and their exact results.

An inference run spends its time in a few calls: the Poisson energy with its
gradient (the minimiser's step), the metric product (every conjugate-gradient
iteration of an MGVI sample), the response itself (mock data, posterior
checks) and its transpose.  The cases below take them at the geometries of the
demo configurations and benchmark workloads of this repository, from a single
small field to seven telescope modules at 1024^2, in float32 (the throughput
tier) and float64 (the reference's own precision, the default of
``build_psf_op`` and ``linpatch_convolve`` on numpy-like input).

A geometry is a square field of ``nx`` pixels cut into ``n`` x ``n`` patches of
stride ``nx // n`` with an FFT side of ``2 (nx // n) + 2 margin``, ``M`` modules
and ``E`` energy bins.
"""
import math

import numpy as np
import torch

import jubik_gb300 as ju
from jubik_gb300 import sky as jsky


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def listed():
    return [
        # the minimiser's step on a full survey field: seven telescope modules, 1024^2, three
        # energy bins, 16 x 16 patches (FFT side 192)
        dict(name="like_1024_m7", kind="likelihood", nx=1024, n=16, margin=32, M=7, E=3,
             dtype="float32"),
        # the eROSITA demo configuration: two modules, 512^2, 8 x 8 patches
        dict(name="like_512_m2", kind="likelihood", nx=512, n=8, margin=32, M=2, E=3,
             dtype="float32"),
        # the smallest field of the benchmark: one module, one energy, FFT side 96; launches and
        # latency count
        dict(name="like_256_m1", kind="likelihood", nx=256, n=8, margin=16, M=1, E=1,
             dtype="float32"),
        # the Chandra demo configuration: one observation, 4 x 4 wide patches (FFT side 320)
        dict(name="like_chandra_512", kind="likelihood", nx=512, n=4, margin=32, M=1, E=3,
             dtype="float32"),
        # seven modules with patches twice as wide (FFT side 384)
        dict(name="like_wide_1024_m7", kind="likelihood", nx=1024, n=8, margin=64, M=7, E=3,
             dtype="float32"),
        # one conjugate-gradient iteration's metric product at a fixed expansion point
        dict(name="metric_1024_m7", kind="metric", nx=1024, n=16, margin=32, M=7, E=3,
             dtype="float32"),
        # expected counts of a field whose side is no multiple of its odd patch stride
        dict(name="response_700_m5", kind="response", nx=700, n=11, margin=33, M=5, E=2,
             dtype="float32"),
        # back-projection of data-space noise, one module (the draw of an MGVI sample)
        dict(name="vjp_1024_m1", kind="vjp", nx=1024, n=16, margin=32, M=1, E=3,
             dtype="float32"),
        # the PSF operator at its default precision, differentiated: forward and backward
        dict(name="psfop_512_m2_f64", kind="psf_op", nx=512, n=8, margin=32, M=2, E=3,
             dtype="float64"),
        # the drop-in patch convolution of a small image at the reference's precision
        dict(name="linpatch_256_f64", kind="linpatch", nx=256, n=8, margin=16, M=1, E=1,
             dtype="float64"),
        # the step in the coordinates of the diffuse sky model: two correlated fields on the
        # padded grid, through exp and the response of the demo field
        dict(name="sky_512_m2", kind="sky", nx=512, n=8, margin=32, M=2, E=3, dtype="float32"),
        # sixteen independent fields of uneven size in one grouped pass
        dict(name="batch_16", kind="batch", nx=512, n=16, margin=16, M=1, E=3, dtype="float32",
             count=16),
    ]


# ------------------------------------------------------------------ geometry
def _side(c):
    return 2 * (c["nx"] // c["n"]) + 2 * c["margin"]


def _largest_prime(v):
    p, big = 2, 1
    while v > 1:
        while v % p == 0:
            big, v = p, v // p
        p += 1
    return big


def _fields(c):
    """The geometries (nx, n, margin, M, E) a case evaluates: one, or the batch's."""
    if c["kind"] != "batch":
        return [(c["nx"], c["n"], c["margin"], c["M"], c["E"])]
    rng = np.random.default_rng(7 * c["nx"] + c["count"])
    out = []
    for _ in range(c["count"]):
        # field sides spread over 128 .. nx, FFT sides 64 and 128, 4 to 16 patches an axis
        side = math.exp(rng.uniform(math.log(128), math.log(max(160, c["nx"]))))
        P = 64 if side < 360 else 128
        margin = int(rng.integers(3, P // 6)) * 2
        dx = P // 2 - margin
        n = min(16, max(4, int(round(side / dx))))
        out.append((n * dx, n, margin, c["M"], int(rng.integers(1, c["E"] + 1))))
    return out


def _work_one(nx, n, margin, M, E, size, forward, adjoint):
    """Bytes and floating point operations of the response (and / or its transpose).  Rows
    of vertically overlapping patches are rows of the same image, so an image row is
    transformed once per patch column; columns are transformed once per patch."""
    P = 2 * (nx // n) + 2 * margin
    K = 2 * (nx // n)
    lg = 5.0 * math.log2(P)
    row = 0.5 * P * lg                      # a real row of P points
    cols = 0.5 * P * P * lg                 # P / 2 complex columns
    units = M * E * n * n
    one = units * (cols + 3 * P * P) + E * n * n * cols + (M + 1) * E * n * nx * row
    sides = int(forward) + int(adjoint)
    psf = M * n * n * E * K * K * size
    return sides * one, psf


def work(case):
    size = 4 if case["dtype"] == "float32" else 8
    kind = case["kind"]
    total = {"bytes": 0.0, "flops": 0.0}
    for nx, n, margin, M, E in _fields(case):
        fwd = kind != "vjp"
        adj = kind not in ("response", "linpatch")
        flops, psf = _work_one(nx, n, margin, M, E, size, fwd, adj)
        sky, img = E * nx * nx * size, M * E * nx * nx * size
        b = psf + sky
        if kind in ("likelihood", "batch"):
            b += 2 * img + sky                      # exposure, counts; gradient
        elif kind == "metric":
            b += img + sky                          # weights; product
        elif kind in ("response", "vjp"):
            b += 2 * img                            # exposure; readout vector
        elif kind == "psf_op":
            b += 2 * img + sky
        elif kind == "linpatch":
            b += img
        elif kind == "sky":
            s = _padded(nx)
            b += 2 * img + 2 * sky + 2 * 3 * 2 * s * s * size
            flops += 2 * 5.0 * s * s * math.log2(s * s)
        total["bytes"] += b
        total["flops"] += flops
    return total


def draw(rng):
    """One more case of the same ranges: kinds, precisions, fields of 128 to 1024 pixels, 3 to
    16 patches an axis, margins of the demo configurations' rule and around it."""
    top = max(work(c)["flops"] for c in listed() if c["dtype"] == "float32")
    kinds = ["likelihood"] * 5 + ["metric", "metric", "response", "vjp", "psf_op", "linpatch", "sky",
                                  "batch"]
    while True:
        kind = rng.choice(kinds)
        if kind == "batch":
            return dict(kind=kind, nx=int(2 ** rng.uniform(8.0, 9.2)), n=16, margin=16, M=1,
                        E=rng.randint(1, 3), dtype="float32", count=rng.randint(4, 24))
        f64 = kind in ("psf_op", "linpatch") or rng.random() < 0.15
        nx = int(2 ** rng.uniform(7.0, 9.3 if f64 else 10.0))
        n = rng.randint(3, 16)
        M = 1 if kind == "linpatch" else rng.choice([1, 1, 2, 3, 5, 7])
        E = rng.randint(1, 3)
        dx = nx // n
        if dx < 8 or dx > 140:
            continue
        margin = max(2, math.ceil(nx * rng.uniform(0.03, 0.08)))
        if rng.random() < 0.7:  # a margin chosen for the FFT: the next side that is a multiple of 32
            P = -(-(2 * dx + 2 * margin) // 32) * 32
            margin = P // 2 - dx
        P = 2 * dx + 2 * margin
        c = dict(kind=kind, nx=nx, n=n, margin=margin, M=M, E=E,
                 dtype="float64" if f64 else "float32")
        if P > 512 or _largest_prime(P) > 13 or 2 * dx > P:
            continue
        # float64 arithmetic is slow on this GPU: a drawn float64 case stays small
        if work(c)["flops"] > (0.03 if f64 else 1.0) * top:
            continue
        return c


# ------------------------------------------------------------------ inputs
def _dtype(c):
    return torch.float32 if c["dtype"] == "float32" else torch.float64


def _gen(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _padded(nx):
    """The padded grid of the sky model: the demo configurations' padding ratio, rounded up to
    a product of 2, 3, 5, 7 and 11."""
    s = int(nx * 1.1075)
    while _largest_prime(s) > 11:
        s += 1
    return s


def _modes(s):
    """Fourier-mode length index of every pixel of an s x s grid, and the lengths."""
    i = np.minimum(np.arange(s), s - np.arange(s))
    k2, index = np.unique(i[:, None] ** 2 + i[None, :] ** 2, return_inverse=True)
    dev = _device()
    return (torch.as_tensor(index.reshape(s, s), device=dev).long(),
            torch.as_tensor(np.sqrt(k2) / s, device=dev, dtype=torch.float64))


def _grf(g, E, nx, std):
    """Log-sky: a Gaussian random field with P(k) ~ (1 + (k / 0.05)^2)^-2."""
    dev = _device()
    k = torch.fft.fftfreq(nx, device=dev, dtype=torch.float64)
    pk = (1.0 + (k[:, None] ** 2 + k[None, :] ** 2) / 0.05 ** 2) ** -1
    w = torch.randn((E, nx, nx), generator=g, device=dev, dtype=torch.float64)
    s = torch.fft.ifft2(torch.fft.fft2(w) * pk).real
    s = (s - s.mean(dim=(-2, -1), keepdim=True)) / s.std(dim=(-2, -1), keepdim=True)
    return std * s


def _sky(g, E, nx):
    """Expected photon flux: diffuse emission on a flat background, a few counts per pixel at
    the exposures below."""
    return 2e-3 * (torch.exp(_grf(g, E, nx, 1.0)) + 0.3)


def _psf(g, nx, n, M, E, dtype):
    """(M, n^2, E, K, K) Moffat kernels that widen off axis, turned per module."""
    dev = _device()
    dx = nx // n
    K = 2 * dx
    turn = float(torch.rand((), generator=g, device=dev)) * 2 * math.pi
    k = torch.arange(n * n, device=dev)
    cen = torch.stack([(k % n) * dx + dx // 2, (k // n) * dx + dx // 2], 1).double()
    r = (cen - nx / 2.0).norm(dim=1)
    r = r / r.max().clamp_min(1e-9)
    off = torch.arange(K, device=dev, dtype=torch.float64) - dx
    u, v = off[:, None], off[None, :]
    out = torch.empty((M, n * n, E, K, K), dtype=dtype, device=dev)
    top = min(8.0, K / 8.0)
    for m in range(M):
        th = turn + math.radians(51.4) * m
        a = (math.cos(th) * u + math.sin(th) * v)[None]
        b = (-math.sin(th) * u + math.cos(th) * v)[None] / 0.8
        for e in range(E):
            fwhm = (2.0 + (top - 2.0) * r) * (1.0 + 0.1 * e)
            alpha = fwhm / (2.0 * math.sqrt(2.0 ** (1 / 2.5) - 1.0))
            q = (1.0 + (a * a + b * b) / (alpha ** 2)[:, None, None]) ** -2.5
            out[m, :, e] = (q / q.sum(dim=(-2, -1), keepdim=True)).to(dtype)
    return out


def _exposure(g, nx, M, E, dtype):
    """Vignetted exposure maps and read-out masks with 1 % of the pixels missing."""
    dev = _device()
    c = torch.arange(nx, device=dev, dtype=torch.float64) - nx / 2 + 0.5
    r2 = c[:, None] ** 2 + c[None, :] ** 2
    level = 1e3 + 1e3 * torch.arange(M, device=dev, dtype=torch.float64) / 6.0
    ex = level[:, None, None, None] * (1.0 - 0.3 * r2 / r2.max())
    bad = torch.rand((M, nx * nx), generator=g, device=dev).topk(nx * nx // 100).indices
    keep = torch.ones((M, nx * nx), dtype=torch.bool, device=dev).scatter_(1, bad, False)
    keep = keep.reshape(M, 1, nx, nx)
    full = (M, E, nx, nx)
    return (ex * keep).expand(full).to(dtype).contiguous(), keep.expand(full).contiguous()


def _inputs(c, geo, seed):
    """Everything a call on one field works on, from the seed alone."""
    nx, n, margin, M, E = geo
    dt, g = _dtype(c), _gen(seed)
    truth = _sky(g, E, nx)
    x = (truth * torch.exp(0.2 * _grf(g, E, nx, 1.0))).to(dt)   # a position near the truth
    psf = _psf(g, nx, n, M, E, dt)
    ex, keep = _exposure(g, nx, M, E, dt)
    # counts of the true sky behind a 3 pixel blur (the data of a real instrument do not
    # come from this code either)
    k = torch.fft.fftfreq(nx, device=x.device, dtype=torch.float64)
    blur = torch.exp(-2.0 * (math.pi * 3.0) ** 2 * (k[:, None] ** 2 + k[None, :] ** 2))
    mean = torch.fft.ifft2(torch.fft.fft2(truth) * blur).real.clamp_min(0)
    lam = ex.double() * mean[None]
    counts = torch.poisson(lam.float(), generator=g).to(torch.int32)
    tangent = torch.randn((E, nx, nx), generator=g, device=x.device, dtype=torch.float64).to(dt)
    cot = torch.randn((M, E, nx, nx), generator=g, device=x.device, dtype=torch.float64).to(dt)
    return dict(x=x, psf=psf, ex=ex, keep=keep, counts=counts, tangent=tangent, cot=cot)


def _plan(c, geo, i):
    nx, n, margin, M, E = geo
    p = ju.ResponsePlan(M, E, (nx, nx), n, margin, dtype=_dtype(c))
    p.set_psf(i["psf"])
    p.set_exposure(i["ex"], i["keep"])
    return p


class _Field:
    """One field of a batch, with the attributes ProblemBatch reads."""

    def __init__(self, geo, i):
        nx, self.n_patches, self.margin, self.n_modules, self.n_energies = geo
        self.shape, self.pixel_area = (nx, nx), 1.0
        self.sky = i["x"].cpu().numpy()
        self.psf, self.exposure, self.readmask = i["psf"], i["ex"], i["keep"]


def _sky_inputs(c, seed):
    """Amplitude spectrum, excitations and offsets of two correlated fields."""
    s, dt, dev = _padded(c["nx"]), _dtype(c), _device()
    g = _gen(seed + 5)
    _, k = _modes(s)
    amp = (1.0 + (k / 0.05) ** 2) ** -1
    amp[0] = 0.0
    amp = torch.stack([amp, 0.3 * amp]) * (9.0 / s)
    xi = torch.randn((2, s, s), generator=g, device=dev, dtype=torch.float64)
    off = torch.tensor([math.log(3e-3), -0.5], device=dev, dtype=torch.float64)
    return amp.to(dt), xi.to(dt), off.to(dt)


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    geos = _fields(c)
    if kind == "batch":
        ins = [_inputs(c, geo, seed * 100 + j) for j, geo in enumerate(geos)]
        b = ju.ProblemBatch([_Field(geo, i) for geo, i in zip(geos, ins)], dtype=_dtype(c))
        b.set_data([i["counts"][i["keep"]].cpu().numpy() for i in ins])
        b.group()
        return dict(kind=kind, batch=b)
    geo = geos[0]
    nx, n, margin, M, E = geo
    i = _inputs(c, geo, seed)
    dom = ju.Domain((E, nx, nx), (1.0, 1.0, 1.0))
    if kind == "linpatch":
        return dict(kind=kind, x=i["x"], kernel=i["psf"][0], domain=dom, n=n, margin=margin)
    if kind == "psf_op":
        op = ju.build_psf_op(dom, n, margin, dtype=_dtype(c))
        op(i["x"], i["psf"])  # the program holds the operator with its kernels set
        return dict(kind=kind, op=op, x=i["x"].requires_grad_(True), kernel=i["psf"],
                    cot=i["cot"])
    p = _plan(c, geo, i)
    st = dict(kind=kind, plan=p, x=i["x"])
    if kind in ("likelihood", "metric", "sky"):
        p.set_data(i["counts"][i["keep"]])
    if kind == "metric":
        p.energy_and_grad(i["x"], need_grad=False)
        st["v"] = i["tangent"]
    if kind == "vjp":
        st["cot"] = i["cot"][i["keep"]]
    if kind == "sky":
        s = _padded(nx)
        e_lo = np.array([0.2, 0.6, 1.2])[:E]
        e_hi = np.array([0.6, 1.2, 2.3])[:E]
        st["sky"] = jsky.CorrelatedFieldSky(
            (s, s), 1.0, n_fields=2, crop=(nx, nx),
            coefficients=jsky.diffuse_coefficients(e_lo, e_hi, 1.0), dtype=_dtype(c))
        st["amp"], st["xi"], st["off"] = _sky_inputs(c, seed)
    return st


def run(state):
    kind = state["kind"]
    if kind == "batch":
        e, g = state["batch"].energy_and_grad()
        return {"energy": e.to(torch.float32), "grad": list(g)}
    if kind == "linpatch":
        return ju.linpatch_convolve(state["x"], state["domain"], state["kernel"], state["n"],
                                    state["margin"])
    if kind == "psf_op":
        y = state["op"](state["x"], state["kernel"])
        (g,) = torch.autograd.grad(y, state["x"], state["cot"])
        return {"image": y.detach(), "grad": g}
    p = state["plan"]
    if kind == "likelihood":
        # the minimiser keeps the energy in its own precision, that of the position
        e, g = p.energy_and_grad(state["x"])
        return {"energy": e.to(g.dtype), "grad": g}
    if kind == "metric":
        return p.metric(None, state["v"])
    if kind == "response":
        return p.response(state["x"])
    if kind == "vjp":
        return p.response_vjp(state["cot"])
    e, dxi, damp, doff = state["sky"].energy_and_grad(p, state["amp"], state["xi"], state["off"])
    return {"energy": e.to(dxi.dtype), "dxi": dxi, "damp": damp, "doff": doff}


# ------------------------------------------------------------------ exact results
class _Exact:
    """The response of one field in float64 torch: patch windows with bilinear weights,
    circular convolution of side P with the normalised kernel, overlap-add and crop."""

    def __init__(self, geo, psf):
        self.nx, self.n, self.margin, self.M, self.E = geo
        self.dx = self.nx // self.n
        self.K = 2 * self.dx
        self.P = self.K + 2 * self.margin
        half = self.dx // 2
        top = self.nx + 2 * half - self.K
        self.start = [min(i * self.dx, top) - half for i in range(self.n)]  # window rows
        dev = psf.device
        a = torch.linspace(0, 1, self.dx, dtype=torch.float64, device=dev) if self.dx > 1 else \
            torch.zeros(1, dtype=torch.float64, device=dev)
        b = torch.cat([a, a.flip(0)])
        self.w = b[:, None] * b[None, :]
        self.psf = psf
        self.pad = self.P + self.dx  # wide enough for every window

    def _spectrum(self, m, e):
        k = self.psf[m, :, e].double()
        k = k / k.sum(dim=(-2, -1), keepdim=True)
        big = torch.zeros((self.n * self.n, self.P, self.P), dtype=torch.float64, device=k.device)
        big[:, :self.K, :self.K] = k
        return torch.fft.rfft2(torch.roll(big, (-self.dx, -self.dx), (-2, -1)))

    def _cut(self, img, size, lead):
        p = torch.nn.functional.pad(img, (self.pad,) * 4)
        o = self.pad - lead
        return torch.stack([p[self.start[k % self.n] + o:self.start[k % self.n] + o + size,
                              self.start[k // self.n] + o:self.start[k // self.n] + o + size]
                            for k in range(self.n * self.n)])

    def _add(self, patches, size, lead):
        full = self.nx + 2 * self.pad
        p = torch.zeros((full, full), dtype=torch.float64, device=patches.device)
        o = self.pad - lead
        for k in range(self.n * self.n):
            r, c = self.start[k % self.n] + o, self.start[k // self.n] + o
            p[r:r + size, c:c + size] += patches[k]
        return p[self.pad:self.pad + self.nx, self.pad:self.pad + self.nx]

    def forward(self, x):
        out = torch.empty((self.M, self.E, self.nx, self.nx), dtype=torch.float64,
                          device=x.device)
        for e in range(self.E):
            z = torch.nn.functional.pad(self._cut(x[e].double(), self.K, 0) * self.w,
                                        (self.margin,) * 4)
            f = torch.fft.rfft2(z)
            for m in range(self.M):
                y = torch.fft.irfft2(f * self._spectrum(m, e), s=(self.P, self.P))
                out[m, e] = self._add(y, self.P, self.margin)
        return out

    def adjoint(self, c):
        out = torch.empty((self.E, self.nx, self.nx), dtype=torch.float64, device=c.device)
        mg = self.margin
        for e in range(self.E):
            s = 0
            for m in range(self.M):
                f = torch.fft.rfft2(self._cut(c[m, e].double(), self.P, mg))
                s = s + f * self._spectrum(m, e).conj()
            y = torch.fft.irfft2(s, s=(self.P, self.P))
            out[e] = self._add(y[:, mg:mg + self.K, mg:mg + self.K] * self.w, self.K, 0)
        return out


def _exact_likelihood(ex, i, x):
    """(energy, gradient in x) of one field's Poisson likelihood."""
    eps, keep = i["ex"].double(), i["keep"]
    lam = eps * ex.forward(x)
    d = i["counts"].double()
    one = torch.ones((), dtype=torch.float64, device=lam.device)
    lam = torch.where(keep, lam, one)
    energy = torch.where(keep, lam - d * torch.log(lam), 0 * one).sum()
    return energy, ex.adjoint(torch.where(keep, eps * (1.0 - d / lam), 0 * one))


def _hartley(v):
    f = torch.fft.fft2(v)
    return f.real + f.imag


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    geos = _fields(c)
    if kind == "batch":
        es, gs = [], []
        for j, geo in enumerate(geos):
            i = _inputs(c, geo, seed * 100 + j)
            e, g = _exact_likelihood(_Exact(geo, i["psf"]), i, i["x"])
            es.append(e)
            gs.append(g)
        return {"energy": torch.stack(es), "grad": gs}
    geo = geos[0]
    i = _inputs(c, geo, seed)
    ex = _Exact(geo, i["psf"])
    eps, keep = i["ex"].double(), i["keep"]
    if kind == "linpatch":
        return ex.forward(i["x"])[0]
    if kind == "psf_op":
        return {"image": ex.forward(i["x"]), "grad": ex.adjoint(i["cot"])}
    if kind == "likelihood":
        e, g = _exact_likelihood(ex, i, i["x"])
        return {"energy": e, "grad": g}
    if kind == "metric":
        lam = eps * ex.forward(i["x"])
        w = torch.where(keep, eps * eps / torch.where(keep, lam, lam * 0 + 1), lam * 0)
        return ex.adjoint(w * ex.forward(i["tangent"]))
    if kind == "response":
        return (eps * ex.forward(i["x"]))[keep]
    if kind == "vjp":
        return ex.adjoint(torch.where(keep, eps * i["cot"].double(), eps * 0))
    # the diffuse sky: log-sky = field_0 + log-energy x field_1 on the data corner
    nx, E = geo[0], geo[4]
    s = _padded(nx)
    amp, xi, off = (t.double() for t in _sky_inputs(c, seed))
    pd, _ = _modes(s)
    e_lo, e_hi = np.array([0.2, 0.6, 1.2])[:E], np.array([0.6, 1.2, 2.3])[:E]
    coef = torch.as_tensor(np.stack([np.ones(E), 0.5 * np.log(e_hi * e_lo)], 1), device=xi.device)
    a = amp[:, pd]
    fields = off[:, None, None] + _hartley(a * xi)
    sky = torch.exp(torch.einsum("eb,bxy->exy", coef, fields[:, :nx, :nx]))
    energy, g = _exact_likelihood(ex, i, sky)
    gf = torch.zeros_like(xi)
    gf[:, :nx, :nx] = torch.einsum("eb,exy->bxy", coef, g * sky)
    h = _hartley(gf)
    damp = torch.stack([torch.zeros_like(amp[b]).index_add_(0, pd.reshape(-1),
                                                            (xi[b] * h[b]).reshape(-1))
                        for b in range(2)])
    return {"energy": energy, "dxi": a * h, "damp": damp, "doff": gf.sum(dim=(-2, -1))}
