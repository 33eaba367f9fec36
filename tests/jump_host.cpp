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
        ExactPath<DIM, TESS> e;
        e.c = -1;
        int mi;
        while (!s.done()) s.settled_unit(t, jc, tab, A, T, h, nT, nODE, p, e, mi, r);
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

// dLoss/dx of n points for dLoss/dT(x) = g: `got` down the list of the adjoint's moves, `want` down the steps of the
// reference's arithmetic; returns how many points the former took step by step.
template <int DIM, int TESS>
static long adjoint(const Tess &t, const double *A, const double *T, const double *x, const double *g, double *got,
                    double *want, long n, int nT, int nODE, double dt)
{
    constexpr int NE = DIM * (DIM + 1), NH = DIM + 1;
    const JumpCfg jc = jump_cfg(DIM, t.nC, nT, nODE, SCHEME_REF, (size_t)227 * 1024, 8);
    const double h = dt / nODE;
    std::vector<double> smem(jump_bytes(jc, DIM, t.nC, 8) / 8 + 2);
    const JumpTables<double> tab =
        stage_jump<DIM, TESS, double>(A, T, t, jc, dt, h, false, reinterpret_cast<unsigned char *>(smem.data()));
    long exact = 0;
    std::vector<int> rows;
    for (long i = 0; i < n; ++i) {
        double r[DIM], v[DIM], q[DIM];
        int mi;
        Path<DIM, TESS, double> s;
        ExactPath<DIM, TESS> e;
        e.c = -1;
        rows.clear();
        for (s.begin(t, jc, x + i * DIM, nT); !s.done();)
            if (s.settled_unit(t, jc, tab, A, T, h, nT, nODE, x + i * DIM, e, mi, r)) rows.push_back(mi);
        exact += e.c >= 0;
        auto back = [&](const double *M, bool columns, bool plus_one) {
            double o[DIM];
            for (int c = 0; c < DIM; ++c) {
                o[c] = plus_one ? v[c] : 0.0;
                for (int k = 0; k < DIM; ++k) o[c] += (columns ? M[c * DIM + k] : M[k * NH + c]) * v[k];
            }
            for (int c = 0; c < DIM; ++c) v[c] = o[c];
        };
        for (int k = 0; k < DIM; ++k) v[k] = g[i * DIM + k] * t.inc[k];
        for (size_t k = rows.size(); k-- > 0;) back(tab.map + (size_t)rows[k] * NE, true, true);
        for (int k = 0; k < DIM; ++k) got[i * DIM + k] = v[k] * t.inv_inc[k];

        rows.clear();  // cells; sub-steps as -1 - cell
        for (int k = 0; k < DIM; ++k) q[k] = x[i * DIM + k];
        for (int step = 0; step < nT; ++step) {
            const int c = exact_cell<DIM, TESS>(t, q);
            double e[DIM];
            exact_affine<DIM>(e, T + c * NE, q);
            if (exact_cell<DIM, TESS>(t, e) == c) {
                for (int k = 0; k < DIM; ++k) q[k] = e[k];
                rows.push_back(c);
                continue;
            }
            for (int k = 0; k < nODE; ++k) {
                const int cc = exact_cell<DIM, TESS>(t, q);
                exact_midpoint<DIM>(q, A + cc * NE, h);
                rows.push_back(-1 - cc);
            }
        }
        for (int k = 0; k < DIM; ++k) v[k] = g[i * DIM + k];
        for (size_t k = rows.size(); k-- > 0;) {
            if (rows[k] >= 0) {
                back(T + rows[k] * NE, false, false);
            } else {
                double D[NE];
                midpoint_increment<DIM>(A + (-1 - rows[k]) * NE, h, D);
                back(D, false, true);
            }
        }
        for (int k = 0; k < DIM; ++k) want[i * DIM + k] = v[k];
    }
    return exact;
}

extern "C" long jump_adjoint(int dim, int tess, const int *nCs, const double *incs, const double *A, const double *T,
                             const double *x, const double *g, double *got, double *want, long n, int nT, int nODE, double dt)
{
    Tess t;
    if (!make_tess(dim, tess, nCs, incs, t)) return -1;
    if (dim == 1) return adjoint<1, 2>(t, A, T, x, g, got, want, n, nT, nODE, dt);
    if (dim == 2 && tess == 1) return adjoint<2, 1>(t, A, T, x, g, got, want, n, nT, nODE, dt);
    if (dim == 2) return adjoint<2, 2>(t, A, T, x, g, got, want, n, nT, nODE, dt);
    if (tess == 1) return adjoint<3, 1>(t, A, T, x, g, got, want, n, nT, nODE, dt);
    return adjoint<3, 2>(t, A, T, x, g, got, want, n, nT, nODE, dt);
}

// kappa of every level above 0 of the sub-step's map, per cell: the tables' value; returns how many levels (2D type II).
extern "C" int jump_kappa(const int *nCs, const double *incs, const double *A, const double *T, int nT, int nODE, double dt,
                          double *kappa)
{
    Tess t;
    if (!make_tess(2, 2, nCs, incs, t)) return -1;
    const JumpCfg jc = jump_cfg(2, t.nC, nT, nODE, SCHEME_REF, (size_t)227 * 1024, 8);
    std::vector<double> smem(jump_bytes(jc, 2, t.nC, 8) / 8 + 2);
    const JumpTables<double> tab =
        stage_jump<2, 2, double>(A, T, t, jc, dt, dt / nODE, false, reinterpret_cast<unsigned char *>(smem.data()));
    for (int l = 0; l < (jc.nS - 1) * t.nC; ++l) kappa[l] = tab.kap[(jc.nT - 1) * t.nC + l];
    return jc.nS - 1;
}
