"""The 1D exact scheme in FP32 for points that end next to zero, against the
FP64 walk, relative to the results themselves: 1e-5 of max(|y|, 1e-6), the
mode's bound (the evaluation's roundings, a few 6e-8, times the logarithm of how
far the interval's results spread, below 20)."""
import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib
from cpabdiffeo_b200.cpa_space import CpaSpace
from cpabdiffeo_b200.space import Prior

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("nC", [2, 16, 100, 600])
def test_relative_error(nC, sign):
    rng = np.random.default_rng(nC)
    sp = CpaSpace([0.0], [1.0], (nC,), device=DEV)
    N, n = 64, 4096
    theta = torch.as_tensor(Prior.create(sp.geo, 0.1, 1.0).sample(N, rng), device=DEV)
    x = torch.as_tensor(10.0 ** rng.uniform(-7, 0, (N * n, 1)), dtype=torch.float32, device=DEV)
    p = dict(dt=0.02, nTimeSteps=50, nStepsODEsolver=10, scheme=_lib.SCHEME_EXACT)
    tables = sp.tables_from_theta(theta, p["dt"], sign)
    y32, y64 = torch.empty_like(x), torch.empty_like(x.double())
    sp.calc_T_batched(tables, x, y32, **p)
    sp.calc_T_batched(tables, x.double(), y64, **p)
    rel = ((y32.double() - y64).abs() / y64.abs().clamp(min=1e-6)).max().item()
    print(nC, sign, rel)
    assert rel <= 1e-5
