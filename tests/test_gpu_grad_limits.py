"""Gradients through calc_T of the largest spaces that the tables allow (two of
dim (dim + 1) doubles per cell in 227 KB), and a status just above: dLoss/dA and
dLoss/dx against torch's through the same steps in FP64, one cell's matrix
exponential per step.  1e-10 of the largest entry: some 30 steps, rounded
differently (1e-16 each, sums of a few hundred terms)."""
import ctypes as C

import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"
DT, NT, NODE = 0.004, 6, 4


def _cell(x, nCs):
    c, stride = torch.zeros(len(x), dtype=torch.long), 1
    for k, n in enumerate(nCs):
        c += torch.floor(x[:, k] * n).long().clamp(0, n - 1) * stride
        stride *= n
    return c


def _forward(A, x, nCs):
    """calc_T step by step; the branch of every step from its values."""
    dim = len(nCs)
    ext = lambda p: torch.cat([p, torch.ones_like(p[:, :1])], 1)[:, :, None]
    T = torch.linalg.matrix_exp(torch.cat([DT * A, torch.zeros_like(A[:, :1])], 1))[:, :dim]
    for _ in range(NT):
        c = _cell(x, nCs)
        q = (T[c] @ ext(x))[:, :, 0]
        p, h = x, DT / NODE
        for _ in range(NODE):
            M = A[_cell(p, nCs)]
            mid = p + 0.5 * h * (M @ ext(p))[:, :, 0]
            p = p + h * (M @ ext(mid))[:, :, 0]
        x = torch.where((_cell(q, nCs) == c)[:, None], q, p)
    return x


def _run(nCs, prec, n=300):
    dim, nC = len(nCs), int(np.prod(nCs))
    L, h = _lib.load(), C.c_void_p()
    pad = (3 - dim)
    _lib.check(L.cpab_ctx_create(C.byref(h), dim, 2, (C.c_int * 3)(*nCs, *[1] * pad),
                                 (C.c_double * 3)(*[1.0 / k for k in nCs], *[1.0] * pad)))
    rng = np.random.default_rng(11)
    A = torch.as_tensor(rng.normal(0, 0.3, (1, nC, dim, dim + 1)), device=DEV)
    x = torch.as_tensor(rng.uniform(0, 1, (n, dim)), device=DEV).to(prec)
    w = torch.as_tensor(rng.normal(0, 1, (n, dim)), device=DEV).to(prec)
    sA, T, gA, gx = torch.empty_like(A), torch.empty_like(A), torch.empty_like(A), torch.empty_like(x)
    p, s = _lib.ptr, _lib.stream_ptr()
    _lib.check(L.cpab_expm(h, p(A), 1, DT, 1, p(sA), p(T), s), h)
    ws = torch.empty(L.cpab_grad_ref_workspace_bytes(h, 1, n, NT, 1), dtype=torch.uint8, device=DEV)
    st = L.cpab_grad_theta_ref(h, None, 0, p(sA), p(T), 1, p(x), n, p(w), 0 if prec == torch.float64 else 1, DT, NT, NODE,
                               1, 1, None, p(gx), p(gA), None, p(ws), ws.numel(), s)
    torch.cuda.synchronize()
    _lib.check(L.cpab_ctx_destroy(h))
    return st, A, x, w, gA, gx


# (FP32 not in 1D: with 7264 cells some of the 1800 step ends lie within float rounding of a vertex)
@pytest.mark.parametrize("nCs,prec,tol", [((7264,), torch.float64, 1e-10)] + [
    (nCs, *p) for nCs in ((49, 49), (48, 48), (11, 11, 10)) for p in ((torch.float64, 1e-10), (torch.float32, 1e-4))])
def test_largest_spaces(nCs, prec, tol):
    st, A, x, w, gA, gx = _run(nCs, prec)
    assert st == 0
    a, y = A[0].cpu().requires_grad_(True), x.double().cpu().requires_grad_(True)
    (_forward(a, y, nCs) * w.double().cpu()).sum().backward()
    ea = (gA[0].cpu() - a.grad).abs().max().item() / a.grad.abs().max().item()
    ex = (gx.double().cpu() - y.grad).abs().max().item() / y.grad.abs().max().item()
    print(nCs, prec, f"dA {ea:.1e} dx {ex:.1e}")
    assert ea < tol and ex < tol


@pytest.mark.parametrize("nCs", [(7265,), (2422, 1), (1211, 1, 1)])
def test_a_status_above(nCs):
    st, *_ = _run(nCs, torch.float64)
    assert st == 10  # CPAB_UNSUPPORTED
