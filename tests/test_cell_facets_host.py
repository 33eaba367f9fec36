"""Facets (cpabdiffeo_b200/csrc/cpab_cell.cuh), compiled as host code, against the
bit-exact lookup: a point whose float margin to a cell's facets is above 1e-5
is in that cell, one below -1e-5 is not -- inside the domain, outside it, near
faces, edges and corners.  Both FP64 and FP32 integration decide by it.  CPU
only."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("facets") / "libfacetshost.so"
    cxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else "g++"
    subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-fno-fast-math",
                    "-I", str(ROOT / "cpabdiffeo_b200" / "csrc"), str(ROOT / "tests" / "cell_facets_host.cpp"),
                    "-o", str(out)], check=True, capture_output=True)
    return C.CDLL(str(out))


@pytest.mark.parametrize("size", [1.0, 300.0])
@pytest.mark.parametrize("nCs,tess", [((1,), "II"), ((100,), "II"), ((4, 4), "I"), ((5, 3), "I"), ((1, 1), "I"), ((1, 2), "I"),
                                      ((5, 3), "II"), ((4, 4, 4), "I"), ((1, 1, 1), "I"), ((2, 3, 2), "I"),
                                      ((3, 2, 4), "II")])
def test_sign_is_certain_beyond_1e5(lib, nCs, tess, size):
    rng = np.random.default_rng(6)
    dim, n = len(nCs), 400000
    inc = np.full(dim, size / nCs[0]) if (dim, tess) == (3, "I") else size / np.asarray(nCs)  # 3D type I: cubes
    top = inc * nCs

    def points():
        x = rng.uniform(-1.0, np.asarray(nCs) + 1.0, (n, dim))
        near = rng.integers(-2, 2 * np.asarray(nCs) + 3, (n, dim)) / 2 + rng.normal(0, 1, (n, dim)) * 10.0 ** rng.uniform(-7, -1, (n, 1))
        return np.where(rng.uniform(size=(n, dim)) < 0.3, near, x)  # faces, box centres, edges, corners

    p = points()
    # q: another point, or one a short step away
    q = np.where(rng.uniform(size=(n, 1)) < 0.3, points(), p + rng.normal(0, 1, (n, dim)) * 10.0 ** rng.uniform(-6, -0.3, (n, 1)))
    p, q = (np.ascontiguousarray(a * inc) for a in (p, q))
    cp, cq, m = np.empty(n, np.int32), np.empty(n, np.int32), np.empty(n, np.float32)
    assert lib.facet_margins(dim, 1 if tess == "I" else 2, (C.c_int * 3)(*nCs), (C.c_double * 3)(*inc),
                             *(a.ctypes.data_as(C.c_void_p) for a in (p, q, cp, cq, m)), C.c_long(n)) == 1
    near = np.abs(q / inc).max(1) < 8  # as the callers ask
    assert (m > 1e-5).any()
    np.testing.assert_array_equal(cq[near & (m > 1e-5)], cp[near & (m > 1e-5)])
    out = near & (m < -1e-5)
    assert not (cq[out] == cp[out]).any()
