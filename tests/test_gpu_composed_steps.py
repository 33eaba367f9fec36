"""FP32 calc_T through composed steps (cpabdiffeo_b200/csrc/cpab_jump.cuh) against
the FP64 mode, which is bit-exact to the reference: step counts at and between
the table levels, every level spacing, anisotropic boxes, points on faces,
corners and outside the domain.

Tolerance: 1e-5 (the FP32 mode's).  A point that lands within float rounding of
a cell's face may be judged inside by one precision and outside by the other;
it then takes sub-steps instead of a closed-form step, which differ by the
sub-steps' own error -- allowed for 0.2 % of the points, up to 1e-3."""
import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib
from cpabdiffeo_b200.cpa_space import CpaSpace
from cpabdiffeo_b200.space import Prior

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _points(rng, sp, n):
    top, dim = np.asarray(sp.XMAXS), sp.dim
    inc = top / np.asarray(sp.nCs)
    x = rng.uniform(-0.02, 1.02, (n, dim)) * top
    # a quarter on faces, edges and corners of boxes, inside the domain (outside, the velocity jumps there, and
    # rounding alone says which side a point is on)
    faces = rng.integers(0, np.asarray(sp.nCs) + 1, (n // 4, dim)) * inc
    x[: n // 4] = np.where(rng.uniform(size=faces.shape) < 0.5, faces, np.clip(x[: n // 4], 0, top))
    return x.astype(np.float32)


@pytest.mark.parametrize("scheme", [_lib.SCHEME_REF, _lib.SCHEME_SIMPLE, _lib.SCHEME_EXACT])
@pytest.mark.parametrize("nT,nODE,T", [(50, 100, 1.0), (1, 1, 0.005), (7, 33, 0.7), (64, 16, 1.0), (3, 300, 0.1)])
@pytest.mark.parametrize("nCs,tess,top", [((100,), "II", (1.0,)), ((4, 4), "I", (1.0, 1.0)), ((5, 3), "I", (1.0, 2.0)),
                                          ((3, 4), "II", (1.0, 1.0)), ((12, 12), "I", (1.0, 1.0)),
                                          ((2, 2, 2), "I", (1.0, 1.0, 1.0)), ((2, 3, 2), "I", (1.0, 2.0, 1.0)),
                                          ((4, 2, 2), "II", (1.0, 1.0, 1.0))])
def test_fp32_equals_fp64(nCs, tess, top, nT, nODE, T, scheme):
    dim = len(nCs)
    if dim == 1 and scheme == _lib.SCHEME_EXACT:
        pytest.skip("1D has its own exact kernel")
    rng = np.random.default_rng(3)
    sp = CpaSpace([0.0] * dim, list(top), nCs, tess=tess, device=DEV)
    theta = Prior.create(sp.geo, 0.15, 0.5).sample(2, rng)
    dt = T / nT
    tables = sp.tables_from_theta(torch.as_tensor(theta, device=DEV), dt, 1)
    n = 3001
    x = _points(rng, sp, 2 * n)
    if scheme == _lib.SCHEME_EXACT:  # hitting times are defined inside the domain
        x = np.clip(x, 0, np.asarray(top)).astype(np.float32)
    p = dict(dt=dt, nTimeSteps=nT, nStepsODEsolver=nODE, scheme=scheme)
    got, want = (torch.empty((2 * n, dim), dtype=d, device=DEV) for d in (torch.float32, torch.float64))
    cnt = torch.zeros(_lib.CNT_N, dtype=torch.int64, device=DEV)
    sp.calc_T_batched(tables, torch.as_tensor(x, device=DEV), got, counters=cnt, **p)
    sp.calc_T_batched(tables, torch.as_tensor(x.astype(np.float64), device=DEV), want, **p)
    err = (got.double() - want).abs().amax(1)
    c = cnt.tolist()
    assert c[_lib.CNT_POINTS] == 2 * n
    if scheme != _lib.SCHEME_SIMPLE:  # every time step is kept or redone with nODE sub-steps
        assert c[_lib.CNT_FAST] + c[_lib.CNT_FALLBACK] == 2 * n * nT
        assert c[_lib.CNT_SUBSTEPS] == c[_lib.CNT_FALLBACK] * nODE
    off = (err > 1e-5 * max(top)).double().mean().item()
    print(nCs, tess, nT, nODE, scheme, f"max {err.max().item():.2e} beyond 1e-5: {off:.2e}")
    assert off <= 2e-3 and err.max().item() < 1e-3 * max(top)


@pytest.mark.parametrize("nCs", [(16, 16), (24, 24), (48, 48)])
def test_wide_spaces_and_nan(nCs):
    """Many cells: sparser table levels, down to single steps; a NaN point stays NaN and alone."""
    rng = np.random.default_rng(4)
    sp = CpaSpace([0.0, 0.0], [1.0, 1.0], nCs, tess="II", device=DEV)
    A = torch.as_tensor(rng.normal(0, 0.2, (1, sp.D)), device=DEV)  # any piecewise-affine field
    x = rng.uniform(0, 1, (4096, 2)).astype(np.float32)
    x[17] = np.nan
    p = dict(dt=0.02, nTimeSteps=20, nStepsODEsolver=20)
    tables = sp.tables_from_A(A, p["dt"])
    got, want = (torch.empty((4096, 2), dtype=d, device=DEV) for d in (torch.float32, torch.float64))
    sp.calc_T_batched(tables, torch.as_tensor(x, device=DEV), got, **p)
    sp.calc_T_batched(tables, torch.as_tensor(x.astype(np.float64), device=DEV), want, **p)
    assert torch.isnan(got[17]).all()
    keep = torch.ones(4096, dtype=torch.bool, device=DEV)
    keep[17] = False
    err = (got.double() - want)[keep].abs().amax(1)
    # the field jumps across faces, so a point at a face may part: allow 1 %
    assert (err > 1e-5).double().mean().item() <= 1e-2


@pytest.mark.parametrize("nCs", [(16, 16), (24, 24), (6, 6, 6), (1500, 1)])
def test_cell_sorting_changes_nothing(nCs):
    """FP32 ignores it: the same table levels, so the same bits."""
    dim = len(nCs)
    rng = np.random.default_rng(5)
    sp = CpaSpace([0.0] * dim, [1.0] * dim, nCs, tess="II", device=DEV)
    tables = sp.tables_from_A(torch.as_tensor(rng.normal(0, 0.2, (1, sp.D)), device=DEV), 0.02)
    x = torch.as_tensor(rng.uniform(0, 1, (20000, dim)), dtype=torch.float32, device=DEV)
    got = []
    for sort, tile in ((False, 2048), (True, 2048), (True, 16384)):
        sp.set_launch(tile_pts=tile, cell_sort=sort)
        got.append(sp.calc_T_batched(tables, x, torch.empty_like(x), dt=0.02, nTimeSteps=50, nStepsODEsolver=100))
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
