"""Performance cases: what programs written on this framework have it do.

Every case goes through the public entry points (CpaSpace, autograd.transform,
GaussianLogLikelihood, remap / remap_ssd) over the unit domain, with theta
drawn from the Gaussian prior, points uniform in the domain, images of
Gaussian-smoothed noise, and integration to time 1 unless the case says
otherwise.  A case's "kind" selects the call:

  plain      one theta at a time, points given one call at a time: theta ->
             Avees -> calc_T_fwd (and calc_T_inv and a remapped image when the
             points are an image's pixel grid) -- the reference's own usage.
  batch      many theta in one call (tables_from_theta + calc_T_batched),
             uniform or ragged point sets, reference or exact scheme.
  grad       one training step's forward and backward through
             autograd.transform with a squared-distance loss.
  register   one likelihood evaluation of many registration chains
             (GaussianLogLikelihood.batch), the work of a Metropolis step.
  remap      remap + Gaussian SSD of a batch of image pairs through given maps.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from cpabdiffeo_b200 import _lib
from cpabdiffeo_b200.autograd import transform
from cpabdiffeo_b200.cpa_space import CpaSpace
from cpabdiffeo_b200.registration import GaussianLogLikelihood, remap, remap_ssd
from cpabdiffeo_b200.space import Prior, build_space

DEV = "cuda"


def listed():
    return [
        # one small call, where launches and the host path count: a contour or a set of landmarks through one theta
        dict(name="plain_2d_f64_1000", kind="plain", nC="4x4", tess="I", prec="f64", n=1000, dt=0.02, nT=50, nODE=100),
        # the plain synthesis configuration: 512 x 512 pixel centres forward and inverse, and the image remapped
        dict(name="plain_2d_f64_512x512", kind="plain", nC="4x4", tess="I", prec="f64", H=512, W=512, dt=0.02, nT=50,
             nODE=100),
        # the batched 1D configuration: signals of 1e3 to 1e5 samples warped by 4096 theta (88 M points)
        dict(name="batch_1d_exact_f32", kind="batch", nC="100", tess="II", prec="f32", scheme="exact", N=4096,
             lo=1000, hi=100000, tuned=True, dt=0.02, nT=50, nODE=100),
        # the same path at full precision, a smaller batch
        dict(name="batch_1d_exact_f64", kind="batch", nC="100", tess="II", prec="f64", scheme="exact", N=512, lo=1000,
             hi=100000, tuned=True, dt=0.02, nT=50, nODE=100),
        # the batched 2D workload: 64 cells, point sets of one size
        dict(name="batch_2d_ref_f32", kind="batch", nC="4x4", tess="I", prec="f32", scheme="ref", N=1024, lo=8192,
             hi=8192, tuned=True, dt=0.02, nT=50, nODE=100),
        # the same with hitting times at the cell faces
        dict(name="batch_2d_exact_f32", kind="batch", nC="4x4", tess="I", prec="f32", scheme="exact", N=512, lo=8192,
             hi=8192, tuned=True, dt=0.02, nT=50, nODE=100),
        # what a server launches: requests of odd sizes in a fine 2D space, launch shape left at its defaults
        dict(name="ragged_2d_8x8_f32", kind="batch", nC="8x8", tess="I", prec="f32", scheme="ref", N=48, lo=1003,
             hi=99991, tuned=False, dt=0.02, nT=50, nODE=100),
        # the same in 3D: tetrahedra, 320 cells
        dict(name="ragged_3d_4x4x4_f32", kind="batch", nC="4x4x4", tess="I", prec="f32", scheme="ref", N=24, lo=1003,
             hi=99991, tuned=False, dt=0.02, nT=50, nODE=100),
        # the 3D gradient configuration at a tenth of its size: dense grids, FP32
        dict(name="grad_3d_f32", kind="grad", nC="4x4x4", tess="I", prec="f32", N=8, n=262144, dt=0.02, nT=50,
             nODE=100),
        # a 2D alignment's training step at full precision
        dict(name="grad_2d_f64", kind="grad", nC="4x4", tess="I", prec="f64", N=16, n=4096, dt=0.02, nT=50, nODE=100),
        # the likelihoods of one Metropolis step of 256 registration chains
        dict(name="register_2d_f32", kind="register", nC="4x4", tess="I", prec="f32", N=256, H=256, W=256, dt=0.02,
             nT=50, nODE=100),
        # 256 image pairs compared through stored maps
        dict(name="remap_ssd_f32", kind="remap", prec="f32", N=256, H=256, W=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "batch", "batch", "batch", "grad", "register", "remap"])
    prec = rng.choice(["f32", "f32", "f64"])
    flow = dict(dt=0.02, nT=50, nODE=100) if rng.random() < 0.7 else \
        rng.choice([dict(dt=0.05, nT=20, nODE=10), dict(dt=0.1, nT=10, nODE=30), dict(dt=0.01, nT=100, nODE=10)])
    dim = rng.choice([1, 2, 2, 3])
    if kind == "register":
        dim = 2
    if dim == 1:
        space = dict(nC=str(rng.choice([16, 37, 64, 100, 256])), tess="II")
    elif dim == 2:
        space = dict(nC=rng.choice(["2x2", "4x4", "5x3", "8x8"]), tess=rng.choice(["I", "I", "I", "II"]))
    else:
        space = rng.choice([dict(nC="2x2x2", tess="I"), dict(nC="4x4x4", tess="I"), dict(nC="4x4x4", tess="II")])
    if kind == "plain":
        if rng.random() < 0.5 and dim == 2:
            return dict(kind=kind, prec=prec, H=rng.randint(64, 512), W=rng.randint(64, 512), **space, **flow)
        return dict(kind=kind, prec=prec, n=_log_int(rng, 1000, 300000), **space, **flow)
    if kind == "batch":
        scheme = "exact" if dim == 1 or rng.random() < 0.3 else "ref"
        lo = _log_int(rng, 500, 4000)
        return dict(kind=kind, prec=prec, scheme=scheme, N=_log_int(rng, 4, 200), lo=lo,
                    hi=lo if rng.random() < 0.3 else lo * rng.randint(2, 20), tuned=rng.random() < 0.5, **space, **flow)
    if kind == "grad":
        return dict(kind=kind, prec=prec, N=_log_int(rng, 1, 16), n=_log_int(rng, 1000, 12000), **space, **flow)
    if kind == "register":
        return dict(kind=kind, prec=prec, N=_log_int(rng, 1, 64), H=rng.randint(64, 256), W=rng.randint(64, 256), **space,
                    **flow)
    return dict(kind=kind, prec=prec, N=_log_int(rng, 8, 256), H=rng.randint(64, 256), W=rng.randint(64, 256))


# ---------------------------------------------------------------- inputs


def _grid(case):
    return tuple(int(k) for k in case["nC"].split("x"))


def _dtype(case):
    return torch.float32 if case["prec"] == "f32" else torch.float64


def _flow(case):
    return dict(dt=case["dt"], nTimeSteps=case["nT"], nStepsODEsolver=case["nODE"])


def _prior_args(dim):
    return (0.15, 0.5) if dim == 3 else (0.1, 1.0)


@functools.lru_cache(maxsize=None)
def _space(nC, tess, prec, tuned):
    """The space a program keeps: its basis, handle and launch shape."""
    g = tuple(int(k) for k in nC.split("x"))
    sp = CpaSpace([0.0] * len(g), [1.0] * len(g), g, tess=tess, device=DEV,
                  precision=torch.float32 if prec == "f32" else torch.float64)
    if tuned:  # what autotune.tune settles on for large batches
        sp.set_launch(block=256 if len(g) == 1 else 128, tile_pts=2048, cell_sort=True)
    return sp


@functools.lru_cache(maxsize=None)
def _prior_factor(nC, tess):
    g = tuple(int(k) for k in nC.split("x"))
    p = Prior.create(build_space(len(g), g, tess), *_prior_args(len(g)))
    w, V = np.linalg.eigh(p.cov_cpa)
    return torch.as_tensor(V * np.sqrt(np.clip(w, 0, None)), device=DEV)


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _thetas(case, N, gen):
    F = _prior_factor(case["nC"], case["tess"])
    return torch.randn((N, F.shape[1]), dtype=torch.float64, device=DEV, generator=gen) @ F.T


def _uniform(shape, dtype, gen):
    return torch.rand(shape, dtype=dtype, device=DEV, generator=gen)


def _images(N, H, W, gen, sigma=8.0):
    """Uniform noise smoothed by a Gaussian (reflecting borders), float32 [N, H, W]."""
    r = min(int(4 * sigma), H - 1, W - 1)
    k = torch.exp(-0.5 * (torch.arange(-r, r + 1, device=DEV, dtype=torch.float32) / sigma) ** 2)
    k = k / k.sum()
    x = torch.nn.functional.pad(_uniform((N, 1, H, W), torch.float32, gen), (r, r, r, r), mode="reflect")
    out = torch.zeros((N, 1, H + 2 * r, W), device=DEV)
    for i in range(2 * r + 1):
        out += k[i] * x[..., i:i + W]
    x, out = out, torch.zeros((N, 1, H, W), device=DEV)
    for i in range(2 * r + 1):
        out += k[i] * x[:, :, i:i + H]
    return out[:, 0].contiguous()


def _pixel_centres(H, W, dtype):
    y = (torch.arange(H, device=DEV, dtype=torch.float64) + 0.5) / H
    x = (torch.arange(W, device=DEV, dtype=torch.float64) + 0.5) / W
    return torch.stack([x.expand(H, W), y[:, None].expand(H, W)], -1).reshape(H * W, 2).to(dtype).contiguous()


def _inputs(case, seed):
    """Everything of a case that its seed decides."""
    gen, dt = _generator(seed), _dtype(case)
    kind = case["kind"]
    if kind == "plain":
        s = dict(theta=_thetas(case, 1, gen)[0])
        if "H" in case:
            s["pts"] = _pixel_centres(case["H"], case["W"], dt)
            s["img"] = _images(1, case["H"], case["W"], gen)[0]
        else:
            s["pts"] = _uniform((case["n"], len(_grid(case))), dt, gen)
        return s
    if kind == "batch":
        N, lo, hi = case["N"], case["lo"], case["hi"]
        # sizes spread evenly over the logarithm of their range, in an order of the seed's
        u = np.random.default_rng(seed).permutation((np.arange(N) + 0.5) / N)
        sizes = np.floor(lo * (hi / lo) ** u + 1e-9).astype(np.int64)
        offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
        return dict(theta=_thetas(case, N, gen), offsets=torch.as_tensor(offs, device=DEV), total=int(offs[-1]),
                    pts=_uniform((int(offs[-1]), len(_grid(case))), dt, gen))
    if kind == "grad":
        N, n, dim = case["N"], case["n"], len(_grid(case))
        side = round(n ** (1.0 / dim))
        if side ** dim == n:  # a dense grid's centres, the same for every theta
            ax = (torch.arange(side, device=DEV, dtype=torch.float64) + 0.5) / side
            one = torch.stack([a.reshape(-1) for a in torch.meshgrid(*[ax] * dim, indexing="ij")], -1)
        else:
            one = _uniform((n, dim), torch.float64, gen)
        pts = one.repeat(N, 1).to(dt)
        # FP32 programs keep FP32 parameters; the target is a smooth displacement of the points
        theta = _thetas(case, N, gen).to(dt)
        phase = _uniform((N, 1, dim), torch.float64, gen)
        disp = 0.03 * torch.sin(2 * math.pi * (pts.reshape(N, n, dim).double() + phase))
        return dict(theta=theta, pts=pts, target=(pts + disp.reshape(-1, dim)).to(dt).contiguous())
    N, H, W = case["N"], case["H"], case["W"]
    src = _images(N, H, W, gen)
    dst = torch.roll(src, (1, 2), (1, 2)) + 0.02 * torch.randn((N, H, W), device=DEV, generator=gen)
    if kind == "register":
        return dict(theta=_thetas(case, N, gen), src=src, dst=dst.contiguous())
    shift = 0.05 * torch.sin(2 * math.pi * (_pixel_centres(H, W, torch.float64) + _uniform((N, 1, 2), torch.float64, gen)))
    maps = (_pixel_centres(H, W, torch.float64) + shift).to(dt)
    return dict(map=maps.contiguous(), src=src, dst=dst.contiguous())


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    kind = case["kind"]
    if kind == "remap":
        return s
    s["space"] = sp = _space(case["nC"], case["tess"], case["prec"], bool(case.get("tuned", False)))
    s["flow"] = _flow(case)
    if kind == "plain":
        s["fwd"] = torch.empty_like(s["pts"])
        if "H" in case:
            s["inv"] = torch.empty_like(s["pts"])
            s["warped"] = torch.empty_like(s["img"])
    elif kind == "batch":
        s["out"] = torch.empty_like(s["pts"])
        s["scheme"] = _lib.SCHEME_EXACT if case["scheme"] == "exact" else _lib.SCHEME_REF
        if case["lo"] == case["hi"]:
            s["offsets"] = None
    elif kind == "grad":
        s["theta"].requires_grad_(True)
    elif kind == "register":
        s["ll"] = GaussianLogLikelihood(sp, s["src"], s["dst"], 0.05, params_flow_int=_flow(case), precision=_dtype(case))
    return s


# ---------------------------------------------------------------- one pass


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "remap":
        H, W = case["H"], case["W"]
        return remap_ssd(state["map"], state["src"], state["dst"], 0.05, pixel_map=(W, -0.5, H, -0.5))
    sp = state["space"]
    if kind == "plain":
        sp.theta2Avees(state["theta"])
        sp.update_pat()
        sp.calc_T_fwd(pts=state["pts"], out=state["fwd"], **state["flow"])
        if "H" not in case:
            return state["fwd"]
        sp.calc_T_inv(pts=state["pts"], out=state["inv"], **state["flow"])
        remap(state["inv"], state["img"], out=state["warped"], pixel_map=(case["W"], -0.5, case["H"], -0.5))
        return state["fwd"], state["inv"], state["warped"]
    if kind == "batch":
        tables = sp.tables_from_theta(state["theta"], case["dt"], 1)
        return sp.calc_T_batched(tables, state["pts"], state["out"], offsets=state["offsets"], scheme=state["scheme"],
                                 **state["flow"])
    if kind == "grad":
        theta = state["theta"]
        theta.grad = None
        y = transform(theta.double(), state["pts"], sp, **state["flow"])
        (0.5 * (y - state["target"]).square().sum()).backward()
        return y.detach(), theta.grad
    # the FP32 mode's likelihood is specified to 1e-6 relative: an FP32 chain keeps it as float32
    return state["ll"].batch(state["theta"]).to(_dtype(case))


# ---------------------------------------------------------------- what a pass cannot do without


def work(case):
    kind = case["kind"]
    el = 4 if case["prec"] == "f32" else 8
    if kind == "remap":
        px = case["N"] * case["H"] * case["W"]
        return dict(bytes=px * (2 * el + 8), flops=px * 14)
    g = _grid(case)
    dim = len(g)
    nC = int(np.prod(g)) * (1 if case["tess"] == "II" else 4 if dim == 2 else 5)
    # a point's transform: at least one affine map and cell lookup in each cell it visits, about two per point and cell
    per_point = 4 * (2 * dim * (dim + 1) + 8 * dim)
    D = nC * dim * (dim + 1)

    def tables(N):  # theta in, one product with the basis and one exponential per cell
        return dict(bytes=N * D * 8, flops=N * (D * 2 * dim + nC * 12 * 2 * dim ** 3))

    if kind == "plain":
        n = case["n"] if "n" in case else case["H"] * case["W"]
        t = tables(1)
        both = 2 if "H" in case else 1
        return dict(bytes=t["bytes"] + n * (dim * el * (1 + both) + (8 if both == 2 else 0)),
                    flops=t["flops"] + n * per_point * both)
    t = tables(case["N"])
    if kind == "batch":
        lo, hi = case["lo"], case["hi"]
        n = case["N"] * (lo if lo == hi else (hi - lo) / math.log(hi / lo))
        return dict(bytes=t["bytes"] + 2 * n * dim * el, flops=t["flops"] + n * per_point)
    if kind == "grad":
        n = case["N"] * case["n"]
        return dict(bytes=2 * t["bytes"] + 3 * n * dim * el, flops=2 * t["flops"] + 3 * n * per_point)
    n = case["N"] * case["H"] * case["W"]
    return dict(bytes=t["bytes"] + n * 8, flops=t["flops"] + n * (per_point + 14))


# ---------------------------------------------------------------- the same in 64 bits, in plain torch


def _cells(u, g, tess):
    """Cell of points u in box units [n, dim] (u[:, k] in [0, g[k]])."""
    n = torch.as_tensor(g, device=u.device, dtype=u.dtype)
    k = torch.minimum(u.floor().clamp(min=0), n - 1)
    f = u - k
    k = k.long()
    box, stride = torch.zeros_like(k[:, 0]), 1
    for i, m in enumerate(g):
        box = box + k[:, i] * stride
        stride *= m
    if tess == "II":
        return box
    if len(g) == 2:
        x, y = f[:, 0], f[:, 1]
        a, b = x < y, 1 - x < y
        return box * 4 + torch.where(a, torch.where(b, 2, 3), torch.where(b, 1, 0))
    odd = ((k[:, 0] ^ k[:, 1] ^ k[:, 2]) & 1).bool()
    x, y, z = torch.where(odd, f[:, 1], f[:, 0]), torch.where(odd, 1 - f[:, 0], f[:, 1]), f[:, 2]
    tet = torch.where(-x - y + z >= 0, 1, torch.where(x + y + z - 2 >= 0, 2, torch.where(
        -x + y - z >= 0, 3, torch.where(x - y - z >= 0, 4, 0))))
    return box * 5 + tet


class _Flow64:
    """The reference scheme (closed-form steps kept while the point stays in its
    cell, else midpoint sub-steps) for N instances, in float64."""

    def __init__(self, case, theta, sign=1, nODE=None):
        self.g, self.tess = _grid(case), case["tess"]
        self.dim, self.N = len(self.g), theta.shape[0]
        self.nT, self.nODE = case["nT"], nODE or case["nODE"]
        self.dt, self.h = case["dt"], case["dt"] / self.nODE
        B = torch.as_tensor(build_space(self.dim, self.g, self.tess).B, device=DEV)
        self.theta = theta
        self.A = sign * (theta.double() @ B.T).reshape(self.N, -1, self.dim, self.dim + 1)
        self.nC = self.A.shape[1]
        X = torch.nn.functional.pad(self.A * self.dt, (0, 0, 0, 1))
        self.T = torch.linalg.matrix_exp(X)[..., :self.dim, :]
        self.Af = self.A.detach().reshape(-1, self.dim, self.dim + 1)
        self.Tf = self.T.detach().reshape(-1, self.dim, self.dim + 1)
        self.scale = torch.as_tensor([float(k) for k in self.g], device=DEV, dtype=torch.float64)

    def cell(self, p, inst):
        return _cells(p * self.scale, self.g, self.tess) + inst * self.nC

    @staticmethod
    def affine(M, c, p):
        m = M[c]
        return (m[..., :-1] @ p[..., None])[..., 0] + m[..., -1]

    def substep(self, p, inst):
        c = self.cell(p, inst)
        pm = p + self.h / 2 * self.affine(self.Af, c, p)
        return p + self.h * self.affine(self.Af, c, pm), c, pm

    def step(self, p, inst):
        """One time step: (end, cell, kept)."""
        c = self.cell(p, inst)
        q = self.affine(self.Tf, c, p)
        kept = self.cell(q, inst) == c
        left = (~kept).nonzero()[:, 0]
        if left.numel():
            r, ri = p[left], inst[left]
            for _ in range(self.nODE):
                r = self.substep(r, ri)[0]
            q = q.index_copy(0, left, r)
        return q, c, kept

    def run(self, p, inst):
        p = p.double()
        for _ in range(self.nT):
            p = self.step(p, inst)[0]
        return p

    def grad(self, p, inst, gout):
        """dLoss/dtheta for dLoss/dT(p) = gout(T(p)); returns (T(p), gradient)."""
        starts, p = [], p.double()
        for _ in range(self.nT):
            starts.append(p)
            p = self.step(p, inst)[0]
        g = gout(p)
        GA, GT = torch.zeros_like(self.Af), torch.zeros_like(self.Tf)

        def outer(a, x):
            return a[:, :, None] * torch.nn.functional.pad(x, (0, 1), value=1.0)[:, None, :]

        for q in reversed(starts):
            c = self.cell(q, inst)
            kept = self.cell(self.affine(self.Tf, c, q), inst) == c
            k, f = kept.nonzero()[:, 0], (~kept).nonzero()[:, 0]
            GT.index_add_(0, c[k], outer(g[k], q[k]))
            gn = (self.Tf[c][..., :-1].transpose(1, 2) @ g[..., None])[..., 0]
            if f.numel():
                r, ri, trail = q[f], inst[f], []
                for _ in range(self.nODE):
                    e, ce, pm = self.substep(r, ri)
                    trail.append((r, ce, pm))
                    r = e
                gf = g[f]
                for r, ce, pm in reversed(trail):
                    LT = self.Af[ce][..., :-1].transpose(1, 2)
                    a = self.h * gf
                    d = (LT @ a[..., None])[..., 0]
                    b = self.h / 2 * d
                    GA.index_add_(0, ce, outer(a, pm) + outer(b, r))
                    gf = gf + d + (LT @ b[..., None])[..., 0]
                gn = gn.index_copy(0, f, gf)
            g = gn
        dtheta, = torch.autograd.grad([self.A, self.T], [self.theta], [GA.reshape(self.A.shape), GT.reshape(self.T.shape)])
        return p, dtheta


def _exact_1d(case, theta, pts, inst):
    """The flow of a piecewise-affine velocity on [0, 1] across cell boundaries."""
    f = _Flow64(case, theta)
    n, out = f.nC, torch.empty_like(pts, dtype=torch.float64)
    for s in range(0, pts.shape[0], 1 << 24):
        x, i = pts[s:s + (1 << 24), 0].double(), inst[s:s + (1 << 24)]
        y = x.clone()
        c = torch.clamp((x * n).floor(), 0, n - 1).long()
        t = torch.full_like(x, f.dt * f.nT)
        idx = torch.arange(x.numel(), device=DEV)
        while idx.numel():
            m = f.Af[i * n + c]
            a, b = m[:, 0, 0], m[:, 0, 1]
            v = a * x + b
            to = torch.where(v > 0, c + 1, c - 1)
            xe = torch.where(v > 0, c + 1, c).double() / n
            ratio = (a * xe + b) / v
            tau = torch.where(a.abs() > 1e-8, torch.log(ratio) / a, (xe - x) / b)
            go = (v.abs() > 1e-8) & (to >= 0) & (to < n) & (ratio > 0) & (tau < t)
            z = a * t
            end = x + t * v * torch.where(z.abs() > 1e-12, torch.expm1(z) / z, torch.ones_like(z))
            y[idx[~go]] = end[~go].clamp(0, 1)
            idx, x, t, c, i = idx[go], xe[go], (t - tau)[go], to[go], i[go]
        out[s:s + (1 << 24), 0] = y
    return out


def _bilinear64(img, px, py):
    """img [N, H, W] at pixel coordinates [N, P], zero outside, float64."""
    N, H, W = img.shape
    flat = img.reshape(N, -1).double()
    c0, r0 = px.floor(), py.floor()
    fx, fy = px - c0, py - r0

    def tap(r, c):
        inside = (r >= 0) & (r < H) & (c >= 0) & (c < W)
        i = r.clamp(0, H - 1).long() * W + c.clamp(0, W - 1).long()
        return torch.where(inside, flat.gather(1, i), torch.zeros_like(px))

    top = (1 - fx) * tap(r0, c0) + fx * tap(r0, c0 + 1)
    bot = (1 - fx) * tap(r0 + 1, c0) + fx * tap(r0 + 1, c0 + 1)
    return (1 - fy) * top + fy * bot


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "remap":
        N, H, W = s["src"].shape
        m = s["map"].double()
        w = _bilinear64(s["src"], m[..., 0] * W - 0.5, m[..., 1] * H - 0.5)
        return -0.5 / 0.05 ** 2 * (w - s["dst"].reshape(N, -1).double()).square().sum(1)
    if kind == "plain":
        th, p = s["theta"][None], s["pts"]
        inst = torch.zeros(p.shape[0], dtype=torch.long, device=DEV)
        fwd = _Flow64(case, th).run(p, inst)
        if "H" not in case:
            return fwd
        inv = _Flow64(case, th, sign=-1).run(p, inst)
        H, W = case["H"], case["W"]
        w = _bilinear64(s["img"][None], inv[None, :, 0] * W - 0.5, inv[None, :, 1] * H - 0.5)
        return fwd, inv, w.reshape(H, W)
    if kind == "batch":
        offs = s["offsets"]
        inst = torch.repeat_interleave(torch.arange(case["N"], device=DEV), offs[1:] - offs[:-1])
        if case["scheme"] == "ref":
            return _Flow64(case, s["theta"]).run(s["pts"], inst)
        if len(_grid(case)) == 1:
            return _exact_1d(case, s["theta"], s["pts"], inst)
        # the flow itself, as ten times finer sub-steps give it: good enough to judge FP32, not FP64
        return _Flow64(case, s["theta"], nODE=1000).run(s["pts"], inst) if case["prec"] == "f32" else None
    N = case["N"]
    if kind == "grad":
        inst = torch.repeat_interleave(torch.arange(N, device=DEV), case["n"])
        target = s["target"].double()
        th = s["theta"].double().requires_grad_(True)
        y, g = _Flow64(case, th).grad(s["pts"], inst, lambda p: p - target)
        return y, g
    H, W = case["H"], case["W"]
    inst = torch.repeat_interleave(torch.arange(N, device=DEV), H * W)
    p = _Flow64(case, s["theta"], sign=-1).run(_pixel_centres(H, W, torch.float64).repeat(N, 1), inst).reshape(N, H * W, 2)
    w = _bilinear64(s["src"], p[..., 0] * W - 0.5, p[..., 1] * H - 0.5)
    return -0.5 / 0.05 ** 2 * (w - s["dst"].reshape(N, -1).double()).square().sum(1)
