"""Composed steps (cpabdiffeo_b200/csrc/cpab_jump.cuh), compiled as host code,
against single steps in the reference's arithmetic: the whole trajectory of
points in the domain, on its faces and corners and beyond them, fields that
keep the domain and fields that do not.  CPU only.

FP64: the two take the same steps unless rounding decides which side of a
facet a point is on, so they differ by rounding (1e-16 a step, up to 5100
steps, grown by a flow that expands by less than 1e3): 1e-9.
"""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from cpabdiffeo_b200.space import Prior, build_space

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("jump") / "libjumphost.so"
    cxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else "g++"
    subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-fno-fast-math", "-w",
                    "-I", "/usr/local/cuda/include", "-I", str(ROOT / "cpabdiffeo_b200" / "csrc"),
                    "-I", str(ROOT / "tests"), str(ROOT / "tests" / "jump_host.cpp"), "-o", str(out)], check=True)
    return C.CDLL(str(out))


def _expm_affine(M):
    """expm of [M; 0] (M [.., D, D+1]) by its Taylor sum of M / 2^8, squared back."""
    D = M.shape[-2]
    Z = np.zeros(M.shape[:-2] + (D + 1, D + 1))
    Z[..., :D, :] = M / 256
    E = term = np.broadcast_to(np.eye(D + 1), Z.shape)
    for k in range(1, 13):
        term = term @ Z / k
        E = E + term
    for _ in range(8):
        E = E @ E
    return E[..., :D, :]


def _walk(lib, nCs, tess, top, x, dt, nT, nODE, f32=False, r_least=1, seed=0, closed=True, wild=0.0, A=None):
    dim = len(nCs)
    geo = build_space(dim, nCs, tess, xmaxs=top, zero_v_across_bdry=(closed,) * dim)
    rng = np.random.default_rng(seed)
    if A is None:
        A = (geo.B @ Prior.create(geo, 0.15, 0.5).sample(1, rng)[0]).reshape(geo.nC, dim, dim + 1)
    if wild:  # any piecewise-affine field: it turns and jumps from cell to cell
        A = rng.normal(0, wild, A.shape)
    A, T = (np.ascontiguousarray(a) for a in (A, _expm_affine(dt * A)))
    x = np.ascontiguousarray(x, np.float64)
    got, want = np.empty_like(x), np.empty_like(x)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    inc = np.asarray(top) / np.asarray(nCs)
    assert lib.jump_walk(dim, 1 if tess == "I" else 2, (C.c_int * 3)(*nCs), (C.c_double * 3)(*inc), int(f32), p(A), p(T),
                         p(x), p(got), p(want), C.c_long(len(x)), nT, nODE, C.c_double(dt), r_least) == 1
    return np.abs(got - want).max(1)


def _points(rng, nCs, top, n, beyond):
    """Uniform up to `beyond` (of a box) outside the domain on every side, a third of them past a corner of it."""
    top = np.asarray(top, float)
    inc = top / np.asarray(nCs)
    x = rng.uniform(-beyond, 1 + beyond, (n, len(nCs))) * inc + rng.integers(0, np.asarray(nCs), (n, len(nCs))) * inc
    d = rng.uniform(0, beyond, (n // 3, len(nCs))) * inc
    x[: n // 3] = np.where(rng.uniform(size=d.shape) < 0.5, -d, top + d)
    return x


TETS = [((2, 2, 2), (1.0,) * 3), ((4, 4, 4), (1.0,) * 3), ((2, 3, 2), (1.0, 2.0, 1.0)), ((4, 2, 3), (1.0,) * 3),
        ((2, 2, 4), (1.0,) * 3)]


@pytest.mark.parametrize("seed", [0, 1])
@pytest.mark.parametrize("nCs,top,beyond,closed", [(*c, *b) for c in TETS for b in ((0.8, True), (0.0, False))] +
                         [((1, 1, 1), (1.0,) * 3, b, False) for b in (0.8, 0.0)])  # (closed: no such field)
def test_tet_keep_test_past_corners(lib, nCs, top, beyond, closed, seed):
    """3D type I, one step at a time: a step is kept exactly when its end is in the cell, also where the point is
    past the domain and the reference's lookup takes the coordinates of the nearest point inside.  FP32: a point
    within float rounding of a facet (1e-7 of a box; some 1e-5 to 1e-4 of the points meet one) may part."""
    rng = np.random.default_rng(40 + seed)
    x = _points(rng, nCs, top, 6000, beyond)
    err = _walk(lib, nCs, "I", top, x, 0.02, 50, 10, r_least=31, seed=seed, closed=closed)
    print(nCs, beyond, closed, f"max {err.max():.2e} share beyond 1e-9: {(err > 1e-9).mean():.2e}")
    assert err.max() < 1e-9
    x = x.astype(np.float32)
    err = _walk(lib, nCs, "I", top, x, 0.02, 50, 10, f32=True, r_least=31, seed=seed, closed=closed)
    print(f"FP32: max {err.max():.2e} share beyond 1e-5: {(err > 1e-5).mean():.2e}")
    assert (err > 1e-5).mean() <= 5e-4


@pytest.mark.parametrize("wild", [0.0, 0.6])  # a prior field, and one that turns and jumps from cell to cell
@pytest.mark.parametrize("nCs,tess,top,closed", [
    ((2, 2, 4), "I", (1.0,) * 3, True), ((2, 2, 4), "I", (1.0,) * 3, False), ((4, 2, 3), "I", (1.0,) * 3, True),
    ((4, 2, 3), "I", (1.0,) * 3, False), ((1, 1, 1), "I", (1.0,) * 3, False), ((2, 3, 2), "I", (1.0, 2.0, 1.0), True),
    ((2, 3, 2), "II", (1.0,) * 3, False), ((1, 1), "I", (1.0,) * 2, False), ((5, 3), "I", (1.0, 2.0), False),
    ((3, 2), "II", (1.0,) * 2, False), ((5,), "II", (1.0,), False)])
def test_jumps_equal_single_steps(lib, nCs, tess, top, closed, wild):
    """Jumps take the steps that the scheme would: points in the domain and past it, boxes of any shape (3D type I:
    also where the reference clamps z inside the domain or beyond its top)."""
    rng = np.random.default_rng(50)
    x = _points(rng, nCs, top, 20000, 0.5)
    err = _walk(lib, nCs, tess, top, x, 0.02, 50, 10, seed=2, closed=closed, wild=wild)
    print(nCs, tess, closed, wild, f"max {err.max():.2e} share beyond 1e-9: {(err > 1e-9).mean():.2e}")
    assert err.max() < 1e-9


@pytest.mark.parametrize("nCs", [(4, 2, 3), (2, 2, 4), (3, 3, 2), (1, 1, 5), (5, 1, 1)])
def test_tet_sign_with_any_boxes(lib, nCs):
    """3D type I with x and z boxes of different sizes, where the reference clamps z inside the domain or beyond its top:
    a point whose margin is beyond 1e-5 is in the cell or is not, as its sign says (with x boxes the larger ones, below
    the top).  The FP64 integration decides by it."""
    rng = np.random.default_rng(53)
    n, inc = 300000, 1.0 / np.asarray(nCs)
    x = _points(rng, nCs, (1.0,) * 3, n, 0.8)
    y = np.ascontiguousarray(x + rng.normal(0, 1, (n, 3)) * inc * 10.0 ** rng.uniform(-6, -0.3, (n, 1)))
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    c, d, m = np.empty(n, np.int32), np.empty(n, np.int32), np.empty(n, np.float32)
    assert lib.facet_margins(3, 1, (C.c_int * 3)(*nCs), (C.c_double * 3)(*inc), p(x), p(y), p(c), p(d), p(m), C.c_long(n)) == 1
    known = np.ones(n, bool) if inc[0] <= inc[2] else (x[:, 2] < 1) & (y[:, 2] < 1)
    np.testing.assert_array_equal(c[known & (m > 1e-5)], d[known & (m > 1e-5)])
    assert not (c == d)[known & (m < -1e-5)].any()
    assert (known & (m > 1e-5)).mean() > 0.2 and (known & (m < -1e-5)).mean() > 0.02


@pytest.mark.parametrize("nCs", [(1, 1), (1, 3), (2, 1), (4, 4)])
def test_triangle_margin_is_a_distance(lib, nCs):
    """2D type I: no displacement shorter than the margin (|.|_1, box units) leaves the cell, past a corner of the
    domain either, where a triangle keeps only the side towards the domain."""
    rng = np.random.default_rng(51)
    n, inc = 200000, 1.0 / np.asarray(nCs)
    x = _points(rng, nCs, (1.0, 1.0), n, 3.0)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    c, c2, m = np.empty(n, np.int32), np.empty(n, np.int32), np.empty(n, np.float32)
    args = 2, 1, (C.c_int * 3)(*nCs), (C.c_double * 3)(*inc)
    assert lib.facet_margins(*args, p(x), p(x), p(c), p(c2), p(m), C.c_long(n)) == 1
    step = rng.standard_normal((n, 2)) * np.where(rng.uniform(size=(n, 2)) < 0.4, 0.0, 1.0) + 1e-9
    step *= (np.maximum(np.minimum(m, 20.0) - 1e-4, 0) / np.abs(step).sum(1))[:, None]
    y = np.ascontiguousarray(x + step * inc)
    assert lib.facet_margins(*args, p(y), p(y), p(c2), p(c2.copy()), p(m.copy()), C.c_long(n)) == 1
    np.testing.assert_array_equal(c2[m > 1e-3], c[m > 1e-3])


@pytest.mark.parametrize("dt", [0.02, -0.02])
def test_arcs_over_a_face_in_either_direction_of_time(lib, dt):
    """Circles around a point near a face that reach over it by up to a fifth of their radius: a jump from before the
    arc to behind it would miss the cell beyond, where nothing moves.  A negative dt is a flow like any other."""
    rng = np.random.default_rng(52)
    ang, r = rng.uniform(0, 2 * np.pi, 4000), rng.uniform(0.04, 0.06, 4000)
    x = np.stack([0.45 + r * np.cos(ang), 0.5 + r * np.sin(ang)], 1)
    A = np.zeros((2, 2, 3))
    A[0] = [[0, -1, 0.5], [1, 0, -0.45]]
    err = _walk(lib, (2, 1), "II", (1.0, 1.0), x, dt, 64, 10, A=A)
    print(dt, f"max {err.max():.2e} share beyond 1e-9: {(err > 1e-9).mean():.2e}")
    assert err.max() < 1e-9


@pytest.mark.parametrize("wild", [0.0, 0.6])
@pytest.mark.parametrize("nCs,tess,top,closed", [
    ((7,), "II", (1.0,), True), ((4, 4), "I", (1.0, 1.0), True), ((5, 3), "I", (1.0, 1.0), False),
    ((3, 7), "II", (1.0, 1.0), True), ((3, 3, 3), "I", (1.0,) * 3, True), ((2, 2, 2), "I", (1.0,) * 3, False),
    ((2, 3, 5), "II", (1.0,) * 3, True)])
def test_adjoint_follows_calc_T(lib, nCs, tess, top, closed, wild):
    """The adjoint's FP64 moves are calc_T's steps: of every point, also on faces, edges, corners and diagonals of boxes
    (where only the reference's own arithmetic says which cell it is in) and past the domain, dT/dx along its branch.
    Rounding of up to 5000 steps, grown by the flow: 1e-8 of the largest entry.  Step by step go only those that come
    within rounding of a facet after the start, or past the domain in 3D type I."""
    dim, nT, nODE, dt = len(nCs), 50, 100, 0.02
    rng = np.random.default_rng(60)
    geo = build_space(dim, nCs, tess, xmaxs=top, zero_v_across_bdry=(closed,) * dim)
    A = (geo.B @ Prior.create(geo, 0.15, 0.5).sample(1, rng)[0]).reshape(geo.nC, dim, dim + 1)
    if wild:
        A = rng.normal(0, wild, A.shape)
    A, T = (np.ascontiguousarray(a) for a in (A, _expm_affine(dt * A)))
    inc, n = np.asarray(top) / np.asarray(nCs), 1500
    on = (rng.integers(0, np.asarray(nCs) + 1, (n, dim)) + rng.choice([0.0, 0.25, 0.5, 0.75], (n, dim))) * inc  # facets
    free = rng.uniform(-0.3, 1.3, (n, dim)) * top
    for name, x in (("inside", rng.uniform(0, 1, (n, dim)) * top), ("facets", np.where(on <= top, on, free * 0.7 + 0.15)),
                    ("around", free)):
        x = np.ascontiguousarray(x)
        g = rng.standard_normal((n, dim))
        got, want = np.empty_like(x), np.empty_like(x)
        p = lambda a: a.ctypes.data_as(C.c_void_p)
        lib.jump_adjoint.restype = C.c_long
        k = lib.jump_adjoint(dim, 1 if tess == "I" else 2, (C.c_int * 3)(*nCs), (C.c_double * 3)(*inc), p(A), p(T), p(x), p(g),
                             p(got), p(want), C.c_long(n), nT, nODE, C.c_double(dt))
        err = np.abs(got - want).max(1) / np.abs(want).max()
        print(nCs, tess, name, f"max {err.max():.1e} beyond 1e-8: {(err > 1e-8).mean():.1e} step by step: {k / n:.1e}")
        assert err.max() < 1e-8
        if name == "inside" and not wild and closed:
            assert k <= 2


@pytest.mark.parametrize("size", [0.01, 0.1, 0.3, 0.5])  # of h L, h the sub-step
def test_kappa_covers_the_flow_of_the_substeps(lib, size):
    """The margin a jump of sub-steps needs is that of the flow through their ends, whose field is log(S) / h, S the
    midpoint map: up to 9 % steeper than the cell's own where the sub-steps are coarse."""
    from scipy.linalg import logm
    rng = np.random.default_rng(54)
    nCs, nODE, h = (6, 5), 4, 0.125
    n, inc = 30, 1.0 / np.asarray(nCs)
    A = rng.normal(0, 1, (n, 2, 3))
    A[:, :, :2] *= (size / h / np.abs(A[:, :, :2] * inc[None, None] / inc[None, :, None]).sum(1).max(1))[:, None, None]
    T, kappa = np.ascontiguousarray(_expm_affine(nODE * h * A)), np.empty((2, n))
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    assert lib.jump_kappa((C.c_int * 2)(*nCs), (C.c_double * 2)(*inc), p(A), p(T), 8, nODE, C.c_double(nODE * h), p(kappa)) == 2
    for c in range(n):
        L = A[c, :, :2]
        S = np.eye(2) + h * L + h * h / 2 * L @ L
        Lf = logm(S).real / h * inc[None] / inc[:, None]
        for l in range(2):
            x = np.abs(Lf).sum(0).max() * h * 2 ** (l + 1)
            if kappa[l, c] < 1e29 and x < 1.4:
                assert kappa[l, c] >= 0.5 * x * np.exp(x) / (2 - np.expm1(x) / x)
