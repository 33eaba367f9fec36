"""Cell helpers of the FP32 integration (cpabdiffeo_b200/csrc/cpab_cell.cuh),
compiled as host code: the box of a cell, and the tetrahedra's lookup with a
margin that no displacement shorter than it (L1, box units) can use to change
the cell.  CPU only."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("margin") / "libmarginhost.so"
    cxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else "g++"
    subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-fno-fast-math",
                    "-I", str(ROOT / "cpabdiffeo_b200" / "csrc"), str(ROOT / "tests" / "cell_margin_host.cpp"),
                    "-o", str(out)], check=True, capture_output=True)
    return C.CDLL(str(out))


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("nCs,tess", [((1,), "II"), ((1 << 20,), "II"), ((512, 512), "I"), ((1000, 1048), "II"),
                                      ((1, 262144), "I"), ((7, 3), "I"), ((59, 59, 59), "I"), ((101, 101, 102), "II"),
                                      ((1, 2, 3), "I")])
def test_cell_box(lib, nCs, tess):
    """Every cell's box indices, up to the largest spaces (2^20 cells)."""
    dim = len(nCs)
    per = 1 if tess == "II" else (4 if dim == 2 else 5)
    n = int(np.prod(nCs)) * per
    kb = np.empty((n, dim), np.int32)
    assert lib.cell_boxes(dim, 1 if tess == "I" else 2, (C.c_int * 3)(*nCs), (C.c_double * 3)(*[1.0 / k for k in nCs]),
                          _ptr(kb)) == n
    want = np.stack(np.unravel_index(np.arange(n) // per, nCs[::-1])[::-1], 1)
    np.testing.assert_array_equal(kb, want)


@pytest.mark.parametrize("size", [1.0, 300.0])  # the unit domain, and one in voxels
@pytest.mark.parametrize("nCs", [(4, 4, 4), (1, 2, 1), (5, 3, 2), (1, 1, 1)])
def test_tet_margin(lib, nCs, size):
    rng = np.random.default_rng(5)
    n = 200000
    inc = np.full(3, size / nCs[0])  # cubes: the reference clamps z with the x box size
    top = inc * nCs

    def run(pts):
        pts = np.ascontiguousarray(pts, dtype=np.float32)
        plain, with_m, m = np.empty(n, np.int32), np.empty(n, np.int32), np.empty(n, np.float32)
        assert lib.tet_margins((C.c_int * 3)(*nCs), (C.c_double * 3)(*inc), _ptr(pts), _ptr(plain), _ptr(with_m),
                               _ptr(m), C.c_long(n)) == 1
        return plain, with_m, m

    x = rng.uniform(-0.2, 1.2, (n, 3)) * top
    grid = rng.integers(-1, np.asarray(nCs) + 2, (n // 2, 3)) * inc  # faces, edges and corners of boxes
    x[: n // 2] = np.where(rng.uniform(size=grid.shape) < 0.5, grid, x[: n // 2])
    x = x.astype(np.float32)
    plain, c, m = run(x)
    np.testing.assert_array_equal(c, plain)
    # float rounding of a box coordinate u <= 6: a few ulps, far below 1e-4
    step = rng.standard_normal((n, 3))
    step *= (np.maximum(np.minimum(m, 1.0) - 1e-4, 0) / np.abs(step).sum(1))[:, None]
    far = m > 1e-3
    assert far.mean() > 0.2
    np.testing.assert_array_equal(run((x + step * inc).astype(np.float32))[0][far], c[far])
