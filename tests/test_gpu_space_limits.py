"""FP32 calc_T of the largest spaces, whose tables leave no room for the warps'
queues, against single steps in the reference's arithmetic (tests/jump_host.cpp):
1e-5, the FP32 mode's tolerance.  The field jumps from cell to cell, so a point
within float rounding of a face may part: 1 % allowed (some 20 steps, each 1e-7
of a cell's share of the points)."""
import ctypes as C

import numpy as np
import pytest
import torch

from cpabdiffeo_b200 import _lib
from test_jump_host import lib  # noqa: F401

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("block", [32, 256])
@pytest.mark.parametrize("nCs", [(14525,), (4841, 1), (4780, 1), (2420, 1, 1), (605, 2, 2)])
def test_largest_spaces(lib, nCs, block):  # noqa: F811
    dim, nC, n = len(nCs), int(np.prod(nCs)), 5000
    rng = np.random.default_rng(9)
    L, h = _lib.load(), C.c_void_p()
    nc, inc = (C.c_int * 3)(*(list(nCs) + [1] * (3 - dim))), (C.c_double * 3)(*[1.0 / k for k in nCs], *[1.0] * (3 - dim))
    _lib.check(L.cpab_ctx_create(C.byref(h), dim, 2, nc, inc))
    _lib.check(L.cpab_set_launch(h, block, 0, 0), h)
    dt, nT, nODE = 0.001, 20, 5
    A = rng.normal(0, 0.05, (nC, dim, dim + 1))
    x = rng.uniform(0, 1, (n, dim)).astype(np.float32)
    dA, dx = torch.as_tensor(A, device=DEV), torch.as_tensor(x, device=DEV)
    sA, T, y = torch.empty_like(dA), torch.empty_like(dA), torch.empty_like(dx)
    p, s = _lib.ptr, _lib.stream_ptr()
    _lib.check(L.cpab_expm(h, p(dA), 1, dt, 1, p(sA), p(T), s), h)
    _lib.check(L.cpab_calc_T(h, p(sA), p(T), p(dx), p(y), n, 1, 0, dt, nT, nODE, None, s), h)
    hp = lambda a: a.ctypes.data_as(C.c_void_p)
    x64, hT, got, want = x.astype(np.float64), T.cpu().numpy(), np.empty((n, dim)), np.empty((n, dim))
    assert lib.jump_walk(dim, 2, nc, inc, 1, hp(A), hp(hT), hp(x64), hp(got), hp(want), C.c_long(n), nT, nODE,
                         C.c_double(dt), 31) == 1
    err = np.abs(y.cpu().numpy() - want).max(1)
    _lib.check(L.cpab_ctx_destroy(h))
    print(nCs, block, f"max {err.max():.2e} beyond 1e-5: {(err > 1e-5).mean():.2e}")
    assert (err > 1e-5).mean() <= 1e-2
