"""The adjoint of calc_T through composed steps (cpab_grad.cu): the same points
with every table level and with level 0 alone -- one step per move, lists
longer than kept at once, replayed from saved states and from before them --
give the same gradients.

Few points leave no room for sums of the levels above 0; the same points among
many others (of zero loss) have them.  FP64: the two are the same map, rounded
differently over up to 1400 steps (1e-16 each, grown by the flow): 1e-9
relative.  FP32: 2e-3, the FP32 adjoint's against the FP64 one."""
import numpy as np
import pytest
import torch

from cpabdiffeo_b200.autograd import transform
from cpabdiffeo_b200.cpa_space import CpaSpace
from cpabdiffeo_b200.space import Prior

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("prec,tol", [(torch.float64, 1e-9), (torch.float32, 2e-3)])
@pytest.mark.parametrize("nT,nODE,T", [(50, 100, 1.0), (7, 3, 0.3), (1, 1, 0.02), (1400, 4, 1.0)])
@pytest.mark.parametrize("nCs,tess", [((20,), "II"), ((4, 4), "I"), ((5, 3), "I"), ((3, 4), "II"), ((2, 2, 2), "I"),
                                      ((3, 2, 2), "II")])
def test_levels_equal_single_steps(nCs, tess, nT, nODE, T, prec, tol):
    dim, rng = len(nCs), np.random.default_rng(8)
    sp = CpaSpace([0.0] * dim, [1.0] * dim, nCs, tess=tess, device=DEV, precision=prec)
    theta = torch.as_tensor(Prior.create(sp.geo, 0.15, 0.5).sample(2, rng), device=DEV)
    few = min(37, sp.nC * (dim + 1) - 1)  # below one sum per cell: level 0 alone
    many = 40 * sp.nC * (dim + 1)         # room for every level
    x = torch.as_tensor(rng.uniform(0.02, 0.98, (2, many, dim)), device=DEV, dtype=prec)
    w = torch.as_tensor(rng.standard_normal((2, many, dim)), device=DEV, dtype=prec)
    w[:, few:] = 0
    p = dict(dt=T / nT, nTimeSteps=nT, nStepsODEsolver=nODE)

    def grads(n):
        th = theta.clone().requires_grad_(True)
        xx = x[:, :n].reshape(-1, dim).clone().requires_grad_(True)
        (transform(th, xx, sp, **p) * w[:, :n].reshape(-1, dim)).sum().backward()
        return th.grad, xx.grad.reshape(2, n, dim)[:, :few].double()

    (t0, x0), (t1, x1) = grads(few), grads(many)
    assert torch.isfinite(t0).all() and t0.abs().max() > 0
    assert ((t0 - t1).abs().max() / t0.abs().max()).item() < tol
    assert ((x0 - x1).abs().max() / x0.abs().max()).item() < tol
