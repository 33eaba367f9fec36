"""The exact scheme's exits by fixed-degree polynomials (slow flows) and by the
general ones: the flow is the same whatever the sub-step's length, so runs on
both sides of the line between the two, h |L| = 0.03, agree.

Tolerance: each exit's rounding, a few 1e-16, grows by at most exp(|L| T) (T =
1, |L| < 9) until the end, < 1e-11.  A path that leaves a cell and comes back
within one long sub-step is not seen there; its end moves by at most the square
of what it does in that sub-step.  Allowed for 1 % of the points."""
import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib
from cpabdiffeo_b200.cpa_space import CpaSpace
from cpabdiffeo_b200.space import Prior

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("nCs,tess", [((4, 4), "I"), ((3, 4), "II"), ((2, 2, 2), "I"), ((3, 2, 2), "II")])
def test_sub_step_lengths_agree(nCs, tess):
    dim, nT, dt = len(nCs), 10, 0.1
    rng = np.random.default_rng(6)
    sp = CpaSpace([0.0] * dim, [1.0] * dim, nCs, tess=tess, device=DEV)
    theta = torch.as_tensor(Prior.create(sp.geo, 0.15, 0.5).sample(1, rng), device=DEV)
    tables = sp.tables_from_theta(theta, dt, 1)
    A = tables[0].reshape(sp.nC, dim, dim + 1)[:, :, :dim]
    scale = 8.0 / A.abs().sum(2).amax().item()  # |L| = 8
    tables = sp.tables_from_theta(theta * scale, dt, 1)
    x = torch.as_tensor(rng.uniform(0.02, 0.98, (4001, dim)), device=DEV)
    ends = {}
    for nODE in (400, 64, 24):  # h |L| = 0.002, 0.0125, 0.033
        ends[nODE] = torch.empty_like(x)
        cnt = torch.zeros(_lib.CNT_N, dtype=torch.int64, device=DEV)
        sp.calc_T_batched(tables, x, ends[nODE], scheme=_lib.SCHEME_EXACT, counters=cnt, dt=dt, nTimeSteps=nT,
                          nStepsODEsolver=nODE)
        assert cnt[_lib.CNT_CROSSINGS] > 400  # exits are what this is about
    for nODE in (64, 24):
        err = (ends[nODE] - ends[400]).abs().amax(1)
        print(nCs, tess, nODE, err.quantile(0.99).item(), err.max().item())
        assert err.quantile(0.99).item() < 1e-11
