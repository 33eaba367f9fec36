"""The 1D exact scheme in FP32 (intervals of the flow map, cpab_exact1d.cu) against
the FP64 mode's walk, which is tested against the reference's closed form: cell
counts on both sides of the rule, forward and inverse, fields with sources,
sinks, zero and constant cells, jumps at vertices and NaN, points at vertices
and outside, ragged ranges cut anywhere.

Tolerance: 1e-6, the FP32 mode's against the closed form; where a field
stretches by G, the float input's own rounding (3e-8 G) on top."""
import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib
from cpabdiffeo_b200.cpa_space import CpaSpace
from cpabdiffeo_b200.space import Prior

pytestmark = pytest.mark.gpu
DEV = "cuda"
P = dict(dt=0.02, nTimeSteps=50, nStepsODEsolver=10)


def _run(sp, A, x, offs, dt, sign=1):
    tables = sp.tables_from_A(A, dt, sign)
    p = dict(P, dt=dt)
    out = []
    for d in (torch.float32, torch.float64):
        y = torch.full(x.shape, float("nan"), dtype=d, device=DEV)
        cnt = torch.zeros(_lib.CNT_N, dtype=torch.int64, device=DEV)
        sp.calc_T_batched(tables, x.to(d), y, offsets=offs, scheme=_lib.SCHEME_EXACT, counters=cnt, **p)
        out.append((y.double(), cnt.cpu().numpy()))
    return out


def _points(rng, nC, n):
    x = rng.uniform(0, 1, n)
    x[: n // 8] = rng.integers(0, nC + 1, n // 8) / nC
    x[n // 8: n // 8 + 4] = [-0.25, 0.0, 1.0, 1.5]
    return torch.as_tensor(x[:, None].astype(np.float32), device=DEV)


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("nC", [2, 7, 16, 100, 256, 600, 700])
def test_prior_fields(nC, sign):
    rng = np.random.default_rng(nC)
    sp = CpaSpace([0.0], [1.0], (nC,), device=DEV)
    N = 5
    theta = Prior.create(sp.geo, 0.1, 1.0).sample(N, rng) if sp.d else np.zeros((N, 0))
    A = torch.as_tensor(theta @ sp.geo.B.T, device=DEV).reshape(N, -1)
    sizes = np.array([0, 1, 3001, 1023, 20000])
    offs = torch.as_tensor(np.concatenate([[0], np.cumsum(sizes)]), device=DEV)
    x = _points(rng, nC, int(sizes.sum()))
    (got, c32), (want, c64) = _run(sp, A, x, offs, 0.02, sign)
    assert c32[_lib.CNT_POINTS] == sizes.sum() and c32[_lib.CNT_FAILED] == 0
    # cells visited: points within float rounding of an interval's end may count one more or less
    assert abs(int(c32[_lib.CNT_FAST]) - int(c64[_lib.CNT_FAST])) <= 1e-3 * c64[_lib.CNT_FAST] + 8
    slope = float(torch.exp(A.reshape(N, nC, 2)[..., 0].abs().amax() * 1.0).clamp(max=1e4))
    assert (got - want).abs().max().item() <= 1e-6 + 3e-8 * slope


@pytest.mark.parametrize("nC", [8, 100])
@pytest.mark.parametrize("kind", ["zero", "constant", "source_sink", "steep", "jumps", "nan"])
def test_made_fields(nC, kind):
    rng = np.random.default_rng(5)
    sp = CpaSpace([0.0], [1.0], (nC,), device=DEV)
    xv = np.linspace(0, 1, nC + 1)
    v = {"zero": 0 * xv, "constant": np.where((xv > 0) & (xv < 1), 0.3, 0.0), "source_sink": 0.2 * np.sin(7 * np.pi * xv),
         "steep": np.sin(2 * np.pi * xv) * 2.0, "jumps": 0 * xv, "nan": 0.3 * np.sin(3 * np.pi * xv)}[kind]
    a = np.diff(v) * nC
    A = np.stack([a, v[:-1] - a * xv[:-1]], 1)
    if kind == "jumps":
        A = rng.normal(0, 0.3, (nC, 2))
    if kind == "nan":
        A[nC // 2] = np.nan
    x = _points(rng, nC, 8000)
    (got, c32), (want, c64) = _run(sp, torch.as_tensor(A.reshape(1, -1), device=DEV), x, None, 0.02)
    assert c32[_lib.CNT_POINTS] == 8000 and c32[_lib.CNT_NAN] == c64[_lib.CNT_NAN]
    ok = torch.isfinite(want)
    assert torch.equal(ok, torch.isfinite(got))
    err = (got - want).abs()[ok]
    slope = float(np.exp(min(np.nanmax(np.abs(A[:, 0])), 9.0)))
    if kind == "jumps":  # a point at a vertex may be on the other side of the jump
        assert (err > 1e-6 + 3e-8 * slope).double().mean().item() < 0.15
    else:
        assert err.max().item() <= 1e-6 + 3e-8 * slope
