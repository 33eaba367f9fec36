"""The 1D exact scheme in FP32, how its points are shared out (cpab_exact1d.cu):
instances of a few points, around the size from which intervals are built, cut
into equal parts or ranges, empty ones among them -- every point against the
FP64 mode, and an instance alone the same bits as in any batch.

Tolerance: 1e-6, the FP32 mode's against the closed form, and the float input's
rounding where the field stretches (see test_gpu_exact1d_intervals.py)."""
import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib
from cpabdiffeo_b200.cpa_space import CpaSpace
from cpabdiffeo_b200.space import Prior

pytestmark = pytest.mark.gpu
DEV = "cuda"
P = dict(dt=0.02, nTimeSteps=50, nStepsODEsolver=10, scheme=_lib.SCHEME_EXACT)


@pytest.mark.parametrize("nC", [7, 100])
@pytest.mark.parametrize("N,n", [(1, 1), (1, 63), (3, 1023), (3, 1024), (5, 1025), (300, 33), (700, 10), (2000, 3), (2, 70001),
                                 (600, 4097)])
def test_uniform_and_ragged(nC, N, n):
    rng = np.random.default_rng(N + n)
    sp = CpaSpace([0.0], [1.0], (nC,), device=DEV)
    sA, T = sp.tables_from_theta(torch.as_tensor(Prior.create(sp.geo, 0.1, 1.0).sample(N, rng), device=DEV), P["dt"], 1)
    x = torch.as_tensor(rng.uniform(0, 1, (N * n, 1)).astype(np.float32), device=DEV)
    slope = float(torch.exp(sA.reshape(N, nC, 2)[..., 0].abs().amax()).clamp(max=1e4))
    new = lambda d=torch.float32, k=N * n: torch.full((k, 1), float("nan"), dtype=d, device=DEV)
    want = sp.calc_T_batched((sA, T), x.double(), new(torch.float64), **P)
    cnt = torch.zeros(_lib.CNT_N, dtype=torch.int64, device=DEV)
    got = sp.calc_T_batched((sA, T), x, new(), counters=cnt, **P)
    assert cnt[_lib.CNT_POINTS].item() == N * n
    assert (got.double() - want).abs().max().item() <= 1e-6 + 3e-8 * slope
    # the same as ragged, with empty instances between
    offs = torch.arange(N + 1, device=DEV, dtype=torch.int64).repeat_interleave(2)[1:] * n
    twice = tuple(t.repeat_interleave(2, 0).contiguous() for t in (sA, T))
    assert torch.equal(sp.calc_T_batched(twice, x, new(), offsets=offs.contiguous(), **P), got)
    for i in {0, N // 2, N - 1}:
        s = slice(i * n, (i + 1) * n)
        alone = sp.calc_T_batched((sA[i:i + 1], T[i:i + 1]), x[s].contiguous(), new(k=n), **P)
        assert torch.equal(alone, got[s])
