"""FP64 calc_T in phases (large launches) against the lane scheduler (small
launches) and the oracle: the same steps in the same order, so equal bits and
equal counters."""
import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib
from cpabdiffeo_b200.cpa_space import CpaSpace
from cpabdiffeo_b200.space import Prior

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("tile_pts", [100, 1023, 2048, 5000])
@pytest.mark.parametrize("nT,nODE", [(50, 10), (1, 1), (5, 3)])
@pytest.mark.parametrize("nCs,tess", [((100,), "II"), ((5, 3), "I"), ((3, 4), "II"), ((2, 2, 2), "I"), ((4, 2, 2), "II")])
def test_phases_equal_lane_scheduler(nCs, tess, nT, nODE, tile_pts):
    dim = len(nCs)
    rng = np.random.default_rng(9)
    sp = CpaSpace([0.0] * dim, [1.0] * dim, nCs, tess=tess, device=DEV)
    sp.set_launch(tile_pts=tile_pts)
    sizes = [0, 1, 1023, 1024, 1025, 2049, 7000, 9000]  # in all above 128 points per SM of any part made so far
    N, n = len(sizes), sum(sizes)
    theta = torch.as_tensor(Prior.create(sp.geo, 0.15, 0.5).sample(N, rng), device=DEV)
    x = rng.uniform(-0.02, 1.02, (n, dim))
    x[:: 7] = np.clip(np.round(x[:: 7] * 4) / 4, 0, 1)  # faces and corners
    x[5] = np.nan
    pts = torch.as_tensor(x, device=DEV)
    off = np.concatenate([[0], np.cumsum(sizes)])
    p = dict(dt=1.0 / nT, nTimeSteps=nT, nStepsODEsolver=nODE)
    tables = sp.tables_from_theta(theta, p["dt"], 1)
    got, want = torch.empty_like(pts), torch.empty_like(pts)
    c_got, c_want = (torch.zeros(_lib.CNT_N, dtype=torch.int64, device=DEV) for _ in range(2))
    sp.calc_T_batched(tables, pts, got, offsets=torch.as_tensor(off, device=DEV), counters=c_got, **p)
    for i in range(N):
        for a in range(off[i], off[i + 1], 4000):
            b = min(a + 4000, off[i + 1])
            one = tuple(t[i: i + 1].contiguous() for t in tables)
            out = torch.empty_like(pts[a:b])
            sp.calc_T_batched(one, pts[a:b].contiguous(), out, counters=c_want, **p)
            want[a:b] = out
    assert torch.equal(got.view(torch.int64), want.view(torch.int64))
    assert c_got.tolist() == c_want.tolist()
    # uniform, one instance: the line between the two routes
    n0 = torch.cuda.get_device_properties(0).multi_processor_count * 128
    y = torch.as_tensor(rng.uniform(0, 1, (n0, dim)), device=DEV)
    one = tuple(t[7:8].contiguous() for t in tables)
    a, b = torch.empty_like(y), torch.empty_like(y[:-1])
    sp.calc_T_batched(one, y, a, **p)
    sp.calc_T_batched(one, y[:-1].contiguous(), b, **p)
    assert torch.equal(a[:-1], b)
