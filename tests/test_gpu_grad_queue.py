"""The gradient of many points by one launch, where warps leave slow points for
later, against the sums of launches so small that they do not: FP64, whose
sums differ by rounding alone: n = 3e5 terms of random sign, partial sums of
some sqrt(n) terms' size, each addition off by 1.1e-16 of that at random, in all
3e-11 of a term or 1e-13 of the sum; 1e-11 of the largest entry leaves room for
entries with larger partial sums."""
import numpy as np
import pytest
import torch

from cpabdiffeo_b200.autograd import transform
from cpabdiffeo_b200.cpa_space import CpaSpace
from cpabdiffeo_b200.space import Prior

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("nCs,tess", [((100,), "II"), ((4, 4), "I"), ((3, 4), "II"), ((2, 2, 2), "I")])
@pytest.mark.parametrize("extra", [-1, 0, 1, 33])
def test_many_points_equal_few(nCs, tess, extra):
    dim = len(nCs)
    rng = np.random.default_rng(12)
    sp = CpaSpace([0.0] * dim, [1.0] * dim, nCs, tess=tess, device=DEV)
    theta = torch.as_tensor(Prior.create(sp.geo, 0.15, 0.5).sample(1, rng), device=DEV)
    n = torch.cuda.get_device_properties(0).multi_processor_count * 2048 + extra  # more than a launch's threads
    x = torch.as_tensor(rng.uniform(0, 1, (n, dim)), device=DEV)
    w = torch.as_tensor(rng.normal(size=(n, dim)), device=DEV)
    p = dict(dt=0.05, nTimeSteps=20, nStepsODEsolver=10)

    def grad(lo, hi):
        th = theta.clone().requires_grad_(True)
        y = x[lo:hi].clone().requires_grad_(True)
        (transform(th, y, sp, **p) * w[lo:hi]).sum().backward()
        return th.grad, y.grad

    gt, gx = grad(0, n)
    few = 20000
    parts = [grad(lo, min(lo + few, n)) for lo in range(0, n, few)]
    want = sum(t for t, _ in parts)
    assert torch.equal(gx, torch.cat([y for _, y in parts]))
    assert (gt - want).abs().max().item() <= 1e-11 * want.abs().max().item()
