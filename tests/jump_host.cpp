// Host build of the composed steps (cpabdiffeo_b200/csrc/cpab_jump.cuh) for tests/test_jump_host.py.
#include "cuda_host.h"

#include <vector>

#include "cell_facets_host.cpp"
#include "cpab_jump.cuh"

using namespace cpab;

// End points of n points: `got` by composed steps in Real, `want` step by step in the reference's arithmetic.
template <int DIM, int TESS, typename Real>
static void walk(const Tess &t, const double *A, const double *T, const double *x, double *got, double *want, long n,
                 int nT, int nODE, double dt, int r_least)
{
    constexpr int NE = DIM * (DIM + 1);
    const JumpCfg jc = jump_cfg(DIM, t.nC, nT, nODE, SCHEME_REF, (size_t)227 * 1024, sizeof(Real), r_least);
    const double h = dt / nODE;
    // room around the tables: level 0 reads an entry of kappa that it ignores
    std::vector<double> smem(jump_bytes(jc, DIM, t.nC, sizeof(Real)) / 8 + 2);
    const JumpTables<Real> tab =
        stage_jump<DIM, TESS, Real>(A, T, t, jc, dt, h, false, reinterpret_cast<unsigned char *>(smem.data()));
    for (long i = 0; i < n; ++i) {
        Real p[DIM], r[DIM];
        for (int k = 0; k < DIM; ++k) p[k] = (Real)x[i * DIM + k];
        Path<DIM, TESS, Real> s;
        s.begin(t, jc, p, nT);
        for (int mi; !s.done();) s.unit(t, jc, tab, nODE, mi, r);
        Real y[DIM];
        s.w.position(t, y);
        double q[DIM];
        for (int k = 0; k < DIM; ++k) {
            got[i * DIM + k] = y[k];
            q[k] = p[k];
        }
        for (int step = 0; step < nT; ++step) {
            const int c = exact_cell<DIM, TESS>(t, q);
            double e[DIM];
            exact_affine<DIM>(e, T + c * NE, q);
            if (exact_cell<DIM, TESS>(t, e) == c) {
                for (int k = 0; k < DIM; ++k) q[k] = e[k];
            } else {
                for (int k = 0; k < nODE; ++k) exact_midpoint<DIM>(q, A + exact_cell<DIM, TESS>(t, q) * NE, h);
            }
        }
        for (int k = 0; k < DIM; ++k) want[i * DIM + k] = q[k];
    }
}

extern "C" int jump_walk(int dim, int tess, const int *nCs, const double *incs, int f32, const double *A, const double *T,
                         const double *x, double *got, double *want, long n, int nT, int nODE, double dt, int r_least)
{
    Tess t;
    if (!make_tess(dim, tess, nCs, incs, t)) return 0;
    auto go = [&](auto real) {
        using R = decltype(real);
        if (dim == 1) walk<1, 2, R>(t, A, T, x, got, want, n, nT, nODE, dt, r_least);
        else if (dim == 2 && tess == 1) walk<2, 1, R>(t, A, T, x, got, want, n, nT, nODE, dt, r_least);
        else if (dim == 2) walk<2, 2, R>(t, A, T, x, got, want, n, nT, nODE, dt, r_least);
        else if (tess == 1) walk<3, 1, R>(t, A, T, x, got, want, n, nT, nODE, dt, r_least);
        else walk<3, 2, R>(t, A, T, x, got, want, n, nT, nODE, dt, r_least);
    };
    if (f32) go(float());
    else go(double());
    return 1;
}
