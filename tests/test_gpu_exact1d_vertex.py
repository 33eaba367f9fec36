"""The 1D exact scheme: points that start exactly on the far vertex of a cell they
leave slowly.  The tables of crossings to skip (FP64) and of the flow map's
intervals (FP32) are built from a point 1e-12 inside the cell, whose exit is
1e-12 / v earlier; end times between the two must not be taken for a crossing
more.  Against the closed form.

Tolerance, FP32: 1e-6, the mode's.  FP64: 1e-9: x + b/a = v/a = 2.5e-7 carries a rounding of 5.5e-17, 2.2e-10 of
it; the time through the cell, log(.)/a, is off by 2.5 times that, the position
by the velocity 0.5 on top: 3e-10."""
import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib
from cpabdiffeo_b200.cpa_space import CpaSpace

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("prec,tol,n", [(torch.float64, 1e-9, 4), (torch.float32, 1e-6, 4), (torch.float32, 1e-6, 4000)])
@pytest.mark.parametrize("sign", [1, -1])
def test_slow_far_vertex(oracle_mod, sign, prec, tol, n):
    v0, a = 1e-7, 0.4
    # right: cell 1 from v0 at 0.25 to 0.1, cell 2 at 0.1, cell 3 at 0.5; left: the mirror image
    A = np.array([[0.0, 0.1], [a, v0 - 0.25 * a], [0.0, 0.1], [0.0, 0.5]])
    x0 = 0.25
    if sign < 0:  # x -> 1 - x: v -> -v(1 - x) = a x - (a + b)
        A = np.stack([A[:, 0], -(A[:, 0] + A[:, 1])], 1)[::-1].copy()
        x0 = 0.75
    through = np.log((a * 0.25 + v0) / v0) / a + 0.25 / 0.1
    sp = CpaSpace([0.0], [1.0], (4,), device=DEV)
    x = np.resize(np.array([[x0], [x0 + sign * 1e-3], [0.3], [0.6]]).astype(np.float32), (n, 1)).astype(np.float64)
    for T in through + np.linspace(-1.5e-5, 2e-6, 23):
        tables = sp.tables_from_A(torch.as_tensor(A.reshape(1, -1), device=DEV), T / 50)
        y = torch.empty((n, 1), dtype=prec, device=DEV)
        sp.calc_T_batched(tables, torch.as_tensor(x, device=DEV).to(prec), y, scheme=_lib.SCHEME_EXACT, dt=T / 50, nTimeSteps=50,
                          nStepsODEsolver=10)
        want, failed = oracle_mod.closed_form_1d(A, 4, x, T / 50 * 50)
        assert failed == 0
        err = np.abs(y.cpu().numpy().ravel() - np.asarray(want).ravel())
        assert err.max() < tol, (T - through, err[:4])
