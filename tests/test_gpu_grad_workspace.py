"""The reference-scheme gradient with any workspace: the least asked for (few
points: shorter composed steps), some more (instances a few at a time) and all
that it puts to use give the same gradients.  FP64, the same map rounded
differently over up to 5000 steps (1e-16 each, grown by the flow): 1e-9."""
import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib
from cpabdiffeo_b200.cpa_space import CpaSpace
from cpabdiffeo_b200.space import Prior

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("nCs,tess", [((20,), "II"), ((4, 4), "I"), ((2, 2, 2), "I")])
@pytest.mark.parametrize("n", [3, 500])
def test_any_workspace(nCs, tess, n):
    dim, N, nT, nODE, dt = len(nCs), 7, 50, 100, 0.02
    rng = np.random.default_rng(13)
    sp = CpaSpace([0.0] * dim, [1.0] * dim, nCs, tess=tess, device=DEV)
    A, T = sp.tables_from_theta(torch.as_tensor(Prior.create(sp.geo, 0.15, 0.5).sample(N, rng), device=DEV), dt, 1)
    x = torch.as_tensor(rng.uniform(0, 1, (N * n, dim)), device=DEV)
    w = torch.as_tensor(rng.normal(0, 1, (N * n, dim)), device=DEV)
    c, p, one = sp._ctx, _lib.ptr, 16 * sp.D * 8
    got = []
    for ck, more in ((nT, 0), (1, 0), (nT, one), (nT, 2 * one + 8), (nT, one // 16 + 255), (nT, 3 * one), (nT, N * one), (nT, 100 * one)):
        least = c.lib.cpab_grad_ref_workspace_bytes(c.h, N, n, nT, ck)
        ws = torch.full((least + more + 256,), 255, dtype=torch.uint8, device=DEV)  # NaN everywhere
        gA, gx = torch.empty_like(A), torch.empty_like(x)
        c.check(c.lib.cpab_grad_theta_ref(c.h, None, 0, p(A), p(T), N, p(x), n, p(w), 0, dt, nT, nODE, 1, ck, None, p(gx),
                                          p(gA), None, p(ws), least + more, _lib.stream_ptr()))
        assert (ws[least + more:] == 255).all()
        got.append((gA, gx))
    for gA, gx in got:
        assert (gA - got[-1][0]).abs().max() <= 1e-9 * got[-1][0].abs().max()
        assert (gx - got[-1][1]).abs().max() <= 1e-9 * got[-1][1].abs().max()
