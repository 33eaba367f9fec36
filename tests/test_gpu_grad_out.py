"""cpab_grad_theta_ref's out: the points calc_T takes its input to, bit for bit --
the map that the gradient is of, so without the clamp of a 1D space, into any
buffer (the input itself too) and whatever the context's launch options."""
import ctypes as C

import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib
from cpabdiffeo_b200.cpa_space import CpaSpace
from cpabdiffeo_b200.space import Prior

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("prec", [torch.float64, torch.float32])
@pytest.mark.parametrize("nCs", [(5,), (3, 2)])
@pytest.mark.parametrize("n", [37, 60000])
def test_out(nCs, prec, n):
    dim, nT, nODE, dt, N = len(nCs), 20, 10, 0.05, 2
    rng = np.random.default_rng(4)
    sp = CpaSpace([0.0] * dim, [1.0] * dim, nCs, tess="II", zero_v_across_bdry=[False] * dim, device=DEV)
    theta = torch.as_tensor(rng.normal(0, 0.5, (N, sp.d)), device=DEV)
    A, T = sp.tables_from_theta(theta, dt, 1)
    x = torch.as_tensor(rng.uniform(0, 1, (N * n, dim)), device=DEV).to(prec)
    w = torch.as_tensor(rng.normal(0, 1, (N * n, dim)), device=DEV).to(prec)
    c, p, s = sp._ctx, _lib.ptr, _lib.stream_ptr()
    c.check(c.lib.cpab_set_clamp(c.h, 0, 0.0, 1.0))
    want = sp.calc_T_batched((A, T), x, torch.empty_like(x), dt=dt, nTimeSteps=nT, nStepsODEsolver=nODE)
    assert want.min() < 0 or want.max() > 1
    c.check(c.lib.cpab_set_clamp(c.h, 1, 0.0, 1.0))
    sp.set_launch(tile_pts=65536, cell_sort=True)
    ws = torch.empty(c.lib.cpab_grad_ref_workspace_bytes(c.h, N, n, nT, 1), dtype=torch.uint8, device=DEV)

    def grad(pts, out):
        gA = torch.empty_like(A)
        gx = torch.empty_like(x)
        c.check(c.lib.cpab_grad_theta_ref(c.h, None, 0, p(A), p(T), N, p(pts), n, p(w), 0 if prec == torch.float64 else 1,
                                          dt, nT, nODE, 1, 1, p(out), p(gx), p(gA), None, p(ws), ws.numel(), s))
        return gA, gx

    out, same = torch.empty_like(x), x.clone()
    gA, gx = grad(x, out)
    assert torch.equal(out, want)
    gA2, gx2 = grad(same, same)
    assert torch.equal(same, want) and torch.equal(gx, gx2)
    assert (gA - gA2).abs().max() <= 1e-6 * gA.abs().max()  # sums in any order


@pytest.mark.parametrize("nCs,tess", [((20,), "II"), ((4, 4), "I"), ((5, 3), "I"), ((3, 7), "II"), ((3, 3, 3), "I"),
                                      ((2, 3, 5), "II"), ((16, 16), "I")])
@pytest.mark.parametrize("n", [4000, 150000])  # all at once; with the slow ones left for later
@pytest.mark.parametrize("closed", [True, False])
def test_fp32_adjoint_follows_calc_T(nCs, tess, n, closed):
    """FP32: with room for all its sums the adjoint's own forward ends where calc_T does, bit for bit: points
    anywhere, half of them on faces, edges, corners and diagonals of boxes, some past the domain."""
    dim, nT, nODE, dt = len(nCs), 50, 100, 0.02
    rng = np.random.default_rng(14)
    sp = CpaSpace([0.0] * dim, [1.0] * dim, nCs, tess=tess, zero_v_across_bdry=[closed] * dim, device=DEV)
    A, T = sp.tables_from_theta(torch.as_tensor(Prior.create(sp.geo, 0.15, 0.5).sample(1, rng), device=DEV), dt, 1)
    x = rng.uniform(-0.1, 1.1, (n, dim))
    on = (rng.integers(0, np.asarray(nCs) + 1, (n, dim)) + rng.choice([0.0, 0.25, 0.5, 0.75], (n, dim))) / np.asarray(nCs)
    x[::2] = np.where(on <= 1, on, x)[::2]
    x = torch.as_tensor(x, device=DEV).float()
    w, out, gx, gA = torch.ones_like(x), torch.empty_like(x), torch.empty_like(x), torch.empty_like(A)
    c, p = sp._ctx, _lib.ptr
    c.check(c.lib.cpab_set_clamp(c.h, 0, 0.0, 1.0))
    want = sp.calc_T_batched((A, T), x, torch.empty_like(x), dt=dt, nTimeSteps=nT, nStepsODEsolver=nODE)
    ws = torch.empty(c.lib.cpab_grad_ref_workspace_bytes(c.h, 1, n, nT, 1) + 16 * sp.D * 8, dtype=torch.uint8, device=DEV)
    c.check(c.lib.cpab_grad_theta_ref(c.h, None, 0, p(A), p(T), 1, p(x), n, p(w), 1, dt, nT, nODE, 1, 1, p(out), p(gx), p(gA),
                                      None, p(ws), ws.numel(), _lib.stream_ptr()))
    off = (out != want).any(1)
    print(nCs, tess, n, closed, f"{off.sum().item()} differ, at most {(out - want).abs().max().item():.1e}")
    assert not off.any()
