"""FP64 gradients through calc_T of points that move along a facet, which the
adjoint takes step by step in the reference's arithmetic (careful_point), among
others that it takes in jumps: dLoss/dA and dLoss/dx against torch's through the
same steps.  1e-10 of the largest entry: some 30 steps, rounded differently."""
import ctypes as C

import numpy as np
import pytest
import torch

import test_gpu_grad_limits as G
from cpabdiffeo_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("nT,nODE", [(6, 4), (40, 20)])  # 40 steps: longer than the list of moves kept at once
@pytest.mark.parametrize("nCs", [(4, 4), (4, 2, 2)])
def test_points_along_a_facet(nCs, nT, nODE, monkeypatch):
    monkeypatch.setattr(G, "NT", nT)
    monkeypatch.setattr(G, "NODE", nODE)
    dim, nC, n = len(nCs), int(np.prod(nCs)), 600
    rng = np.random.default_rng(17)
    A = rng.normal(0, 0.3, (nC, dim, dim + 1))
    A[np.isin(np.arange(nC) % 4, (1, 2)), 0] = 0.0  # v_x = 0 beside the plane x = 1/2: points stay on it, to the bit
    x = rng.uniform(0.05, 0.95, (n, dim))
    x[::3, 0] = 0.5
    L, h, pad = _lib.load(), C.c_void_p(), 3 - dim
    _lib.check(L.cpab_ctx_create(C.byref(h), dim, 2, (C.c_int * 3)(*nCs, *[1] * pad),
                                 (C.c_double * 3)(*[1.0 / k for k in nCs], *[1.0] * pad)))
    dA, dx, w = (torch.as_tensor(a, device=DEV) for a in (A, x, rng.normal(0, 1, (n, dim))))
    sA, T, gA, gx = torch.empty_like(dA), torch.empty_like(dA), torch.empty_like(dA), torch.empty_like(dx)
    p, s = _lib.ptr, _lib.stream_ptr()
    _lib.check(L.cpab_expm(h, p(dA), 1, G.DT, 1, p(sA), p(T), s), h)
    ws = torch.empty(L.cpab_grad_ref_workspace_bytes(h, 1, n, nT, 1) + 16 * dA.numel() * 8, dtype=torch.uint8, device=DEV)
    _lib.check(L.cpab_grad_theta_ref(h, None, 0, p(sA), p(T), 1, p(dx), n, p(w), 0, G.DT, nT, nODE, 1, 1, None, p(gx), p(gA),
                                     None, p(ws), ws.numel(), s), h)
    _lib.check(L.cpab_ctx_destroy(h))
    a, y = dA.cpu().requires_grad_(True), dx.cpu().requires_grad_(True)
    end = G._forward(a, y, nCs)
    assert (end[::3, 0] == 0.5).all()
    (end * w.cpu()).sum().backward()
    ea = (gA.cpu() - a.grad).abs().max().item() / a.grad.abs().max().item()
    ex = (gx.cpu() - y.grad).abs().max().item() / y.grad.abs().max().item()
    print(nCs, nT, f"dA {ea:.1e} dx {ex:.1e}")
    assert ea < 1e-10 and ex < 1e-10
