"""The largest spaces that calc_T and the likelihoods take: the cell tables (A
and T, or the two level 0 maps in FP32) within an SM's 227 KB.  The entry points
are called for no points, or with too small a workspace, so they return before
any launch.  CPU only."""
import ctypes as C

import pytest

from cpabdiffeo_b200 import _lib

OK, NO_MEMORY, UNSUPPORTED = 0, 5, 10
BASE = 1 << 20  # aligned; never read
F64, F32 = 0, 1
LIMIT = 227 * 1024


@pytest.fixture
def ctx():
    lib, made = _lib.load(), []

    def make(dim, tess, nCs):
        h = C.c_void_p()
        n = (C.c_int * 3)(*(list(nCs) + [1] * (3 - dim)))
        inc = (C.c_double * 3)(*[1.0 / k for k in n])
        assert lib.cpab_ctx_create(C.byref(h), dim, tess, n, inc) == OK
        made.append(h)
        return h

    yield lib, make
    for h in made:
        lib.cpab_ctx_destroy(h)


def _cells(dim, prec):
    """Most cells: two tables of dim (dim + 1) entries each and 48 bytes of bookkeeping."""
    return (LIMIT - 48) // (2 * dim * (dim + 1) * (8 if prec == F64 else 4))


@pytest.mark.parametrize("scheme", [0, 1])
@pytest.mark.parametrize("prec", [F64, F32])
@pytest.mark.parametrize("dim", [1, 2, 3])
def test_calc_T(ctx, dim, prec, scheme):
    lib, make = ctx
    n = _cells(dim, prec)
    for cells, want in ((n, OK), (n + 1, OK if (prec, scheme) == (F32, 1) else UNSUPPORTED)):  # (one map there)
        h = make(dim, 2, [cells] + [1] * (dim - 1))
        st = lib.cpab_calc_T(h, BASE, BASE, BASE, BASE, 0, prec, scheme, 0.02, 50, 100, None, None)
        assert st == want, (cells, lib.cpab_last_error_string(h))


@pytest.mark.parametrize("tess,nCs", [(1, (34, 34)), (2, (69, 69))])
def test_wide_2d_spaces(ctx, tess, nCs):
    lib, make = ctx
    assert lib.cpab_calc_T(make(2, tess, nCs), BASE, BASE, BASE, BASE, 0, F32, 0, 0.02, 50, 100, None, None) == OK


@pytest.mark.parametrize("prec", [F64, F32])
def test_likelihoods(ctx, prec):
    lib, make = ctx
    el = 8 if prec == F64 else 4
    # the smallest tile: 256 pixels of 16 bytes or voxels of 24, and a sum of each 32
    for dim, tile in ((2, 256 * 16 + 8 * 8), (3, 256 * 24 + 8 * 8)):
        n = (LIMIT - tile) // (2 * dim * (dim + 1) * el)
        for cells, want in ((n, NO_MEMORY), (n + 1, UNSUPPORTED)):
            h = make(dim, 2, [cells] + [1] * (dim - 1))
            lib.cpab_set_launch(h, 0, 0, 64)
            args = [h, BASE, BASE, 1, BASE, BASE] + [64] * dim + [0.05, prec, 0.02, 50, 100, BASE, None, None, 0, None, None]
            st = (lib.cpab_register_ll if dim == 2 else lib.cpab_register3d_ll)(*args)
            assert st == want, (dim, cells, lib.cpab_last_error_string(h))


@pytest.mark.parametrize("scheme", [0, 1])
@pytest.mark.parametrize("dim,nCs", [(1, (100,)), (2, (4, 4)), (2, (69, 70)), (3, (4, 4, 4))])
def test_fp32_needs_no_room_to_sort(ctx, dim, nCs, scheme):
    """FP32 launches ignore cell sorting: it takes nothing from the space or the tile."""
    lib, make = ctx
    h = make(dim, 2, nCs)
    lib.cpab_set_cell_sort(h, 1)
    for tile in (2048, 65536):
        lib.cpab_set_launch(h, 0, 0, tile)
        st = lib.cpab_calc_T(h, BASE, BASE, BASE, BASE, 0, F32, scheme, 0.02, 50, 100, None, None)
        assert st == OK, (tile, lib.cpab_last_error_string(h))


def test_trajectory(ctx):
    """Its kernel keeps nothing beside the tables."""
    lib, make = ctx
    for dim in (1, 2, 3):
        n = LIMIT // (2 * dim * (dim + 1) * 8)
        for cells, want in ((n, OK), (n + 1, UNSUPPORTED)):
            h = make(dim, 2, [cells] + [1] * (dim - 1))
            assert lib.cpab_calc_trajectory(h, BASE, BASE, BASE, BASE, 0, 0.02, 50, 100, None) == want, (dim, cells)
