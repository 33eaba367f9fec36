"""cpab_grad_theta_ref's out: the points calc_T takes its input to, bit for bit --
the map that the gradient is of, so without the clamp of a 1D space, into any
buffer (the input itself too) and whatever the context's launch options."""
import ctypes as C

import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib
from cpabdiffeo_b200.cpa_space import CpaSpace

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
