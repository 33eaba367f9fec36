"""FP64 calc_T of 3D type I spaces with boxes of any shape -- the reference clamps
z with the x box's size, inside the domain or beyond its top -- bit for bit the
reference's steps, one at a time (tests/jump_host.cpp)."""
import ctypes as C

import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib
from cpabdiffeo_b200.cpa_space import CpaSpace
from cpabdiffeo_b200.space import Prior
from test_jump_host import _points, lib  # noqa: F401

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [2000, 60000])  # lanes for themselves; phase by phase
@pytest.mark.parametrize("closed", [True, False])
@pytest.mark.parametrize("nCs", [(4, 2, 3), (2, 2, 4), (3, 3, 2), (5, 1, 1)])
def test_bits(lib, nCs, closed, n):  # noqa: F811
    nT, nODE, dt = 50, 20, 0.02
    rng = np.random.default_rng(16)
    sp = CpaSpace([0.0] * 3, [1.0] * 3, nCs, tess="I", zero_v_across_bdry=[closed] * 3, device=DEV)
    A, T = sp.tables_from_theta(torch.as_tensor(Prior.create(sp.geo, 0.15, 0.5).sample(1, rng), device=DEV), dt, 1)
    x = _points(rng, nCs, (1.0,) * 3, n, 0.3)
    y = sp.calc_T_batched((A, T), torch.as_tensor(x, device=DEV), torch.empty((n, 3), dtype=torch.float64, device=DEV), dt=dt,
                          nTimeSteps=nT, nStepsODEsolver=nODE)
    hA, hT, got, want = A.cpu().numpy(), T.cpu().numpy(), np.empty_like(x), np.empty_like(x)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    assert lib.jump_walk(3, 1, (C.c_int * 3)(*nCs), (C.c_double * 3)(*sp.geo.incs), 0, p(hA), p(hT), p(x), p(got), p(want),
                         C.c_long(n), nT, nODE, C.c_double(dt), 31) == 1
    np.testing.assert_array_equal(y.cpu().numpy(), want)
