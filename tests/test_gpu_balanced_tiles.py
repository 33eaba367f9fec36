"""Tiles that share a small launch's points out evenly: totals on both sides of
one and of two tiles per CTA, uniform and ragged with empty instances.  A
point's result does not depend on its tile: equal bits."""
import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib
from cpabdiffeo_b200.cpa_space import CpaSpace
from cpabdiffeo_b200.space import Prior

pytestmark = pytest.mark.gpu
DEV = "cuda"
CTAS, TILE = 3, 96


@pytest.mark.parametrize("scheme", [_lib.SCHEME_REF, _lib.SCHEME_EXACT])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("N", [1, 5, 40])
@pytest.mark.parametrize("total", [1, 63, 200, CTAS * TILE, CTAS * TILE + 1, 2 * CTAS * TILE - 1, 2 * CTAS * TILE, 2000])
def test_any_total(total, N, dtype, scheme):
    rng = np.random.default_rng(total + N)
    sp = CpaSpace([0.0, 0.0], [1.0, 1.0], (4, 4), tess="I", device=DEV)
    theta = torch.as_tensor(Prior.create(sp.geo, 0.1, 1.0).sample(N, rng), device=DEV)
    p = dict(dt=0.1, nTimeSteps=10, nStepsODEsolver=10)
    tables = sp.tables_from_theta(theta, p["dt"], 1)
    cut = np.sort(rng.integers(0, total + 1, N - 1))  # some instances empty
    off = np.concatenate([[0], cut, [total]]).astype(np.int64)
    x = torch.as_tensor(rng.uniform(0, 1, (total, 2)), dtype=dtype, device=DEV)
    want = torch.empty_like(x)
    for i in range(N):
        one = tuple(t[i: i + 1].contiguous() for t in tables)
        if off[i + 1] > off[i]:
            out = torch.empty_like(x[off[i]: off[i + 1]])
            sp.calc_T_batched(one, x[off[i]: off[i + 1]].contiguous(), out, scheme=scheme, **p)
            want[off[i]: off[i + 1]] = out
    sp.set_launch(tile_pts=TILE, max_ctas=CTAS)
    got = torch.full_like(x, float("nan"))
    sp.calc_T_batched(tables, x, got, offsets=torch.as_tensor(off, device=DEV), scheme=scheme, **p)
    assert torch.equal(got, want)
    # uniform: the first instances' points, as many for each
    n = total // N
    if n:
        a, b = torch.full_like(x[: n * N], float("nan")), torch.empty_like(x[: n * N])
        sp.calc_T_batched(tables, x[: n * N].contiguous(), a, scheme=scheme, **p)
        sp.calc_T_batched(tables, x[: n * N].contiguous(), b, offsets=torch.arange(N + 1, device=DEV) * n, scheme=scheme,
                          **p)
        assert torch.equal(a, b)
