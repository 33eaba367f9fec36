// cpab_integrate.cuh -- the integration arithmetic (exact double / fast
// float overloads) and the lane-scheduled warp loop shared by k_integrate
// (calc_T) and the fused registration likelihood.
#pragma once

#include <math_constants.h>

#include "cpab_device.cuh"

namespace cpab {

// ------------------------------------------------------------ arithmetic
//
// Two per-point states:
//  * double (bit-exact family): one double per coordinate, the reference's
//    arithmetic (cpab_cell.cuh).
//  * float (FP32 mode): an unnormalised compensated pair hi + lo per
//    coordinate plus x = fl(hi + lo), the float nearest the point, which the
//    cell lookup reads.  Each update adds its increment d to hi and the
//    rounding error of that addition (Fast2Sum; where |hi| < |d| the error
//    term is below ulp(d)) to lo, so the increments of the integration are
//    not lost to float rounding.  Every step is an increment from a small
//    matrix (cpab_jump.cuh): the closed-form step adds (T - I)[x; 1]; an
//    explicit midpoint sub-step of length h with the cell's velocity
//    v(x) = A[x; 1] (both evaluations in the cell of x, calc_2Dto2D.cu:177-196)
//    is, inside one cell, the affine map x + h v(x + h/2 v(x)) = x + (S - I)[x; 1]
//    with S - I = [h L + h^2/2 L^2 | h b + h^2/2 L b]      (A = [L | b]),
//    evaluated in double when the tables are staged.  Table roundings are
//    relative to the increments, not to the position.
// Shared-memory tables per cell (ne = DIM * (DIM + 1)) of the double states:
// A[ne] (EXACT: S[ne]) and T[ne], row-major as in global memory.  Float
// matrices are column-major (the DIM columns of the linear part, then the
// offset) so that one is read with 8-byte (1D/2D) or 16-byte (3D) loads.

template <int DIM, typename Real>
struct PState;

template <int DIM>
struct PState<DIM, double> {
    double p[DIM];
};

template <int DIM>
__device__ void stage_exact_substeps(const double *gA, const double *gT, int nC, double h, double *sS, double *sT);

// Stage one instance's double tables in shared memory (layout above).  EXACT
// scheme (2D/3D): the sub-step map is the exact flow S = expm(h A), h the
// sub-step length, instead of the signed A.
template <int DIM>
__device__ __forceinline__ void stage_tables(const double *gA, const double *gT, int nC, bool with_T, double h,
                                             double *sA, double *sT, bool exact_sub = false)
{
    if (exact_sub) {
        stage_exact_substeps<DIM>(gA, gT, nC, h, sA, sT);
        return;
    }
    // not unrolled: the staging loop's loads in flight would otherwise set
    // the register count of the integration loop that follows
#pragma unroll 1
    for (int i = threadIdx.x; i < nC * DIM * (DIM + 1); i += blockDim.x) {
        sA[i] = gA[i];
        if (with_T) sT[i] = gT[i];
    }
}

// A cell's column-major float matrix into registers (8-byte loads in 1D/2D,
// 16-byte loads in 3D; the tables' offsets keep those aligned).
template <int DIM>
__device__ __forceinline__ void load_cell(const float *p, float *m)
{
    constexpr int NE = DIM * (DIM + 1);
    if (DIM == 3) {
#pragma unroll
        for (int i = 0; i < NE / 4; ++i) {
            const float4 v = reinterpret_cast<const float4 *>(p)[i];
            m[4 * i] = v.x;
            m[4 * i + 1] = v.y;
            m[4 * i + 2] = v.z;
            m[4 * i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < NE / 2; ++i) {
            const float2 v = reinterpret_cast<const float2 *>(p)[i];
            m[2 * i] = v.x;
            m[2 * i + 1] = v.y;
        }
    }
}

template <int DIM, int TESS>
__device__ __forceinline__ int cell_of(const Tess &t, const PState<DIM, double> &s)
{
    return exact_cell<DIM, TESS>(t, s.p);
}

// One unit of work on a point in cell c: the candidate end point q of a
// closed-form step (fast: q = T_c [p; 1]) or of one explicit-midpoint
// sub-step with A_c, in the reference's arithmetic.  The caller looks up the
// cell of q; a closed-form step is kept when that is still c
// (calc_2Dto2D.cu:380-400), a sub-step always is, and its end cell is the cell
// of the next sub-step's start point.
template <int DIM>
__device__ __forceinline__ void advance(bool fast, const PState<DIM, double> &s, const double *A, const double *T,
                                        double h, PState<DIM, double> &q)
{
    if (fast) {
        exact_affine<DIM>(q.p, T, s.p);
    } else {
        q = s;
        exact_midpoint<DIM>(q.p, A, h);
    }
}
// Paired FP32 arithmetic (sm_100's FFMA2 / FADD2: two lanes of float math per
// instruction, each rounded as its scalar twin) for the (x, y) coordinates:
// the column-major cell matrix gives column k as the pair (M[0][k], M[1][k]).
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

// ------------------------------------------------------------ exact scheme (2D/3D)
//
// Sub-step map of the exact flow: column j of S - I is
// sum_{k>=1} h^k/k! L^{k-1} A[:, j]  (A = [L | b], homogeneous bottom row 0),
// summed per column until the terms fall below the sum's rounding.
// Tables: S row-major (the layout exact_affine-style code reads).
template <int DIM>
__device__ void stage_exact_substeps(const double *gA, const double *gT, int nC, double h, double *sS, double *sT)
{
    constexpr int NE = DIM * (DIM + 1);
#pragma unroll 1
    for (int c = threadIdx.x; c < nC; c += blockDim.x) {
        const double *a = gA + (size_t)c * NE;
        double L[DIM * DIM];
#pragma unroll
        for (int r = 0; r < DIM; ++r)
#pragma unroll
            for (int k = 0; k < DIM; ++k) L[r * DIM + k] = a[r * (DIM + 1) + k];
#pragma unroll 1
        for (int col = 0; col <= DIM; ++col) {
            double w[DIM], acc[DIM];
#pragma unroll
            for (int r = 0; r < DIM; ++r) {
                w[r] = h * a[r * (DIM + 1) + col];
                acc[r] = w[r];
            }
#pragma unroll 1
            for (int k = 2; k <= 40; ++k) {
                double nw[DIM], big = 0.0, am = 0.0;
#pragma unroll
                for (int r = 0; r < DIM; ++r) {
                    double v = 0.0;
#pragma unroll
                    for (int m = 0; m < DIM; ++m) v = fma(L[r * DIM + m], w[m], v);
                    nw[r] = v * (h / k);
                }
#pragma unroll
                for (int r = 0; r < DIM; ++r) {
                    w[r] = nw[r];
                    acc[r] += w[r];
                    big = fmax(big, fabs(w[r]));
                    am = fmax(am, fabs(acc[r]));
                }
                if (!(big > 1e-18 * am)) break;
            }
#pragma unroll
            for (int r = 0; r < DIM; ++r) sS[c * NE + r * (DIM + 1) + col] = acc[r] + (r == col ? 1.0 : 0.0);
        }
    }
#pragma unroll 1
    for (int i = threadIdx.x; i < nC * NE; i += blockDim.x) sT[i] = gT[i];
}

// What a lane needs to resolve an exit: the instance's signed A (global,
// row-major [nC, DIM*(DIM+1)]), the facet tables, the sub-step length and
// the lane's counters.
// Parked exits a warp resolves together, and the votes the oldest may wait
// (integrate_range, integrate_jump).  Resolving costs a few hundred FP64
// instructions however many lanes take part; in a batch of 512 instances of
// 8192 points (2D, 64 cells, FP32) 16 exits at a time took 1100 us, 24 995, 28
// or 31 960, 32 978 (FP64, 64 such instances: 28 815, 31 848, 32 889).
#ifndef CPAB_EXACT_CROSS_BATCH
#define CPAB_EXACT_CROSS_BATCH 28
#endif
#ifndef CPAB_EXACT_CROSS_WAIT
#define CPAB_EXACT_CROSS_WAIT 400
#endif

struct ExactCross {
    const double *A;
    const double *F;
    const int *nbr;
    int nF;
    double h;
    int cap;
    unsigned long long crossings, unresolved;
};

template <int DIM, int TESS>
__device__ __forceinline__ int lookup_d(const Tess &t, const double *p, double)
{
    return exact_cell<DIM, TESS>(t, p);
}
template <int DIM, int TESS>
__device__ __forceinline__ int lookup_d(const Tess &t, const double *p, float)
{
    float x[DIM];
#pragma unroll
    for (int i = 0; i < DIM; ++i) x[i] = (float)p[i];
    return fast_cell<DIM, TESS>(t, x);
}

// The flow inside a cell over a time t <= h (one sub-step) as a Taylor
// polynomial: x(t) = p + sum_{k>=1} w_k, w_k = t^k/k! u_k, u_1 = L p + b,
// u_k = L u_{k-1} (A = [L | b], read through the read-only cache at each use:
// held in registers it raised the kernel's spills, 37.3 against 36.1 ms).  The
// series stops at the first degree K whose omitted terms are provably below
// FP64 rounding of the first: with r = t |L| / (K+1) < 1 (|L| the max row
// sum), |w_{K+j}| <= |w_K| r^j, so the rest sums to at most |w_K| r/(1-r).
// At sub-step lengths (t |L| ~ 1e-3) that is K = 6 or 7; kExactDeg caps it,
// and a flow the cap does not resolve (t |L| above ~0.1) is reported so that
// exact_substep_cross keeps the reference scheme's sub-step end.
constexpr int kExactDeg = 10;
constexpr double kTaylorTol = 1e-17;
// 1/k for the Taylor recurrences (a product instead of an FP64 division per term)
static __constant__ double kInvInt[kExactDeg + 2] = {0.0,       1.0,       1.0 / 2,  1.0 / 3,
                                                     1.0 / 4,   1.0 / 5,   1.0 / 6,  1.0 / 7,
                                                     1.0 / 8,   1.0 / 9,   1.0 / 10, 1.0 / 11};

template <int DIM>
__device__ __forceinline__ double affine_norm(const double *__restrict__ A)
{
    double lnorm = 0.0;
#pragma unroll
    for (int r = 0; r < DIM; ++r) {
        double rs = 0.0;
#pragma unroll
        for (int m = 0; m < DIM; ++m) rs += fabs(__ldg(A + r * (DIM + 1) + m));
        lnorm = fmax(lnorm, rs);
    }
    return lnorm;
}

template <int DIM>
__device__ __forceinline__ void affine_lin(const double *__restrict__ A, const double *u, double *out)
{
#pragma unroll
    for (int r = 0; r < DIM; ++r) {
        double v = 0.0;
#pragma unroll
        for (int m = 0; m < DIM; ++m) v = fma(__ldg(A + r * (DIM + 1) + m), u[m], v);
        out[r] = v;
    }
}

template <int DIM>
__device__ __forceinline__ void velocity(const double *__restrict__ A, const double *p, double *v)
{
#pragma unroll
    for (int r = 0; r < DIM; ++r) {
        double s = __ldg(A + r * (DIM + 1) + DIM);
#pragma unroll
        for (int m = 0; m < DIM; ++m) s = fma(__ldg(A + r * (DIM + 1) + m), p[m], s);
        v[r] = s;
    }
}

// out = expm(t A)[p; 1] (out may alias p); false when kExactDeg terms do
// not bring the omitted rest below FP64 rounding of the first term
template <int DIM>
__device__ __noinline__ bool flow_taylor_any(const double *__restrict__ A, const double *p, double t, double *out)
{
    const double *Ar = A;  // global, read through __ldg
    const double lnorm = affine_norm<DIM>(A);
    double u[DIM], x[DIM];
    velocity<DIM>(Ar, p, u);
    double coef = t, first = 0.0;
#pragma unroll
    for (int r = 0; r < DIM; ++r) {
        x[r] = fma(coef, u[r], p[r]);
        first = fmax(first, fabs(coef * u[r]));
    }
    const double tl = fabs(t) * lnorm;
    bool ok = false;
#pragma unroll 1
    for (int k = 2; k <= kExactDeg; ++k) {
        double nu[DIM];
        affine_lin<DIM>(Ar, u, nu);
        coef *= t * kInvInt[k];
        double wk = 0.0;
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
            u[r] = nu[r];
            x[r] = fma(coef, u[r], x[r]);
            wk = fmax(wk, fabs(coef * u[r]));
        }
        const double rr = tl * kInvInt[k + 1];
        if (rr < 0.5 && wk * rr <= kTaylorTol * (1.0 - rr) * first) {
            ok = true;
            break;
        }
    }
#pragma unroll
    for (int r = 0; r < DIM; ++r) out[r] = x[r];
    return ok || first == 0.0;
}

// First root in [0, s] of g(t) = F . x(t) + F[DIM] along the flow of A from
// p, given g(0) = g0 < 0 < g(s): the Taylor coefficients of g,
// c_k = F . u_k / k!, up to the degree whose omitted rest is below FP64
// rounding of g over [0, s] (the bound of flow_taylor times |F|_1), and a
// safeguarded Newton iteration on that polynomial.  Returns NaN when
// kExactDeg terms do not resolve g to that rounding.
template <int DIM>
__device__ __noinline__ double facet_hit_time_any(const double *__restrict__ A, const double *__restrict__ F,
                                                 const double *p, double s, double g0)
{
    const double *Ar = A;  // global, read through __ldg
    const double lnorm = affine_norm<DIM>(A);
    double c[kExactDeg + 1];
    c[0] = g0;
    double u[DIM], Fn[DIM], f1 = 0.0;
#pragma unroll
    for (int r = 0; r < DIM; ++r) {
        Fn[r] = __ldg(F + r);
        f1 += fabs(Fn[r]);
    }
    velocity<DIM>(Ar, p, u);
    const double sl = s * lnorm;
    double inv_fact = 1.0, sk = 1.0, scale = 0.0;
    int K = 0;
#pragma unroll 1
    for (int k = 1; k <= kExactDeg; ++k) {
        if (k > 1) {
            double nu[DIM];
            affine_lin<DIM>(Ar, u, nu);
#pragma unroll
            for (int r = 0; r < DIM; ++r) u[r] = nu[r];
        }
        inv_fact *= kInvInt[k];
        sk *= s;
        double d = 0.0, un = 0.0;
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
            d = fma(Fn[r], u[r], d);
            un = fmax(un, fabs(u[r]));
        }
        c[k] = d * inv_fact;
        if (k == 1) {
            scale = fabs(g0) + fabs(c[1]) * s;
        } else {
            const double rr = sl * kInvInt[k + 1];
            if (rr < 0.5 && f1 * un * inv_fact * sk * rr <= kTaylorTol * (1.0 - rr) * scale) {
                K = k;
                break;
            }
        }
    }
    if (K == 0) return CUDART_NAN;
    auto P = [&](double t, double &dP) {
        double v = c[K], dv = 0.0;
#pragma unroll 1
        for (int k = K - 1; k >= 0; --k) {
            dv = fma(dv, t, v);
            v = fma(v, t, c[k]);
        }
        dP = dv;
        return v;
    };
    double lo = 0.0, hi = s, dP;
    const double ps = P(s, dP);
    if (!(ps > 0)) return s;
    double t = s * (-g0) / (ps - g0);
    if (!(t > lo && t < hi)) t = 0.5 * (lo + hi);
#pragma unroll 1
    for (int it = 0; it < 60; ++it) {
        const double g = P(t, dP);
        if (g > 0) hi = t; else lo = t;
        if (g == 0) return t;
        double tn = t - g / dP;
        if (!(tn > lo && tn < hi)) tn = 0.5 * (lo + hi);
        // converged within about two ulps (4.5e-16 relative is at least two
        // ulps in every binade: a tolerance under one ulp never ends an
        // iteration that alternates between neighbouring doubles)
        if (fabs(tn - t) <= 4.5e-16 * fabs(t) || hi - lo <= 4.5e-16 * hi) return tn;
        t = tn;
    }
    return 0.5 * (lo + hi);
}

// Both again, for the slow flows of ordinary sub-steps: with x = t |L| so small
// that the rest after kShortDeg terms, at most x^8 / 9! (1 + x) of the first
// one, is below kTaylorTol, the degree is fixed, the loops unroll and A stays
// in registers.  (x <= 0.03 makes that rest 2e-18.)  With the exits' facets
// picked before their times are computed (lanes used to enter the search at
// whichever of the facets was theirs, one facet after the other) the batch of
// 512 x 8192 points in 2D took 1100 us instead of 2015.
constexpr int kShortDeg = 8;
constexpr double kShortMax = 0.03;

template <int DIM>
struct AffineMap {
    double a[DIM * (DIM + 1)], norm;
    __device__ __forceinline__ void load(const double *__restrict__ A)
    {
        norm = 0.0;
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
            double rs = 0.0;
#pragma unroll
            for (int m = 0; m <= DIM; ++m) {
                a[r * (DIM + 1) + m] = __ldg(A + r * (DIM + 1) + m);
                if (m < DIM) rs += fabs(a[r * (DIM + 1) + m]);
            }
            norm = fmax(norm, rs);
        }
    }
    __device__ __forceinline__ void vel(const double *p, double *v) const
    {
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
            double s = a[r * (DIM + 1) + DIM];
#pragma unroll
            for (int m = 0; m < DIM; ++m) s = fma(a[r * (DIM + 1) + m], p[m], s);
            v[r] = s;
        }
    }
    __device__ __forceinline__ void lin(const double *u, double *v) const
    {
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
            double s = a[r * (DIM + 1)] * u[0];
#pragma unroll
            for (int m = 1; m < DIM; ++m) s = fma(a[r * (DIM + 1) + m], u[m], s);
            v[r] = s;
        }
    }
};

template <int DIM>
__device__ __forceinline__ bool flow_taylor(const AffineMap<DIM> &M, const double *__restrict__ A, const double *p,
                                            double t, double *out)
{
    if (!(fabs(t) * M.norm <= kShortMax)) return flow_taylor_any<DIM>(A, p, t, out);
    // p + t (v + t/2 L (v + t/3 L (v + ...)))
    double v[DIM], w[DIM];
    M.vel(p, v);
#pragma unroll
    for (int r = 0; r < DIM; ++r) w[r] = v[r];
#pragma unroll
    for (int k = kShortDeg; k > 1; --k) {
        double lw[DIM];
        M.lin(w, lw);
        const double tk = t * (1.0 / k);
#pragma unroll
        for (int r = 0; r < DIM; ++r) w[r] = fma(tk, lw[r], v[r]);
    }
#pragma unroll
    for (int r = 0; r < DIM; ++r) out[r] = fma(t, w[r], p[r]);
    return true;
}

template <int DIM>
__device__ __forceinline__ double facet_hit_time(const AffineMap<DIM> &M, const double *__restrict__ A,
                                                 const double *__restrict__ F, const double *p, double s, double g0)
{
    double c[kShortDeg + 1], u[DIM], Fn[DIM], f1 = 0.0, un = 0.0;
    M.vel(p, u);
#pragma unroll
    for (int r = 0; r < DIM; ++r) {
        Fn[r] = __ldg(F + r);
        f1 += fabs(Fn[r]);
        un = fmax(un, fabs(u[r]));
    }
    c[0] = g0;
    c[1] = 0.0;
#pragma unroll
    for (int r = 0; r < DIM; ++r) c[1] = fma(Fn[r], u[r], c[1]);
    // the rest: f1 |u| s x^8 / 9! (1 + x) of g, to be below rounding of g over [0, s]; x^8 <= 0.03^4 x^4
    const double x = s * M.norm, x2 = x * x;
    if (!(x <= kShortMax && f1 * un * s * (x2 * x2) * (kShortMax * kShortMax * kShortMax * kShortMax * 1.03 / 362880) <=
                                kTaylorTol * (fabs(g0) + fabs(c[1]) * s)))
        return facet_hit_time_any<DIM>(A, F, p, s, g0);
    double inv_fact = 1.0;
#pragma unroll
    for (int k = 2; k <= kShortDeg; ++k) {
        double nu[DIM], d = 0.0;
        M.lin(u, nu);
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
            u[r] = nu[r];
            d = fma(Fn[r], u[r], d);
        }
        inv_fact *= 1.0 / k;
        c[k] = d * inv_fact;
    }
    auto P = [&](double t, double &dP) {
        double v = c[kShortDeg], dv = 0.0;
#pragma unroll
        for (int k = kShortDeg - 1; k >= 0; --k) {
            dv = fma(dv, t, v);
            v = fma(v, t, c[k]);
        }
        dP = dv;
        return v;
    };
    // Newton with the slope's reciprocal in float (the polynomial is close to
    // linear: the secant is off by x at most, the second iterate by 1e-7 of
    // that), to the same end as facet_hit_time_any
    auto over = [](double g, double d) { return g * (double)__frcp_rn((float)d); };
    double lo = 0.0, hi = s, dP;
    const double ps = P(s, dP);
    if (!(ps > 0)) return s;
    double t = s * over(-g0, ps - g0);
    if (!(t > lo && t < hi)) t = 0.5 * (lo + hi);
#pragma unroll 1
    for (int it = 0; it < 60; ++it) {
        const double g = P(t, dP);
        if (g > 0) hi = t; else lo = t;
        if (g == 0) return t;
        double tn = t - over(g, dP);
        if (!(tn > lo && tn < hi)) tn = 0.5 * (lo + hi);
        if (fabs(tn - t) <= 4.5e-16 * fabs(t) || hi - lo <= 4.5e-16 * hi) return tn;
        t = tn;
    }
    return 0.5 * (lo + hi);
}

// A sub-step of length h from p in cell c ended at q outside c: the exact
// flow from p, exit times through interior facets, the neighbour across the
// exited facet, the rest of the sub-step there (and so on).  q becomes the
// point at the sub-step's end; returns its cell.  FP64 throughout (the
// hitting times; Real is the precision whose cell lookup decides).  When no interior facet
// explains the exit (a point on the domain boundary) or the crossings exceed
// the cap, q is the end point of the flow in the current cell (as in the
// reference scheme, which keeps its sub-step's end wherever it lands).
template <int DIM, int TESS, typename Real>
__device__ __forceinline__ int exact_substep_cross(const Tess &t, ExactCross &ex, int c,
                                                   const double *from, double *q)
{
    constexpr int NH = DIM + 1, NE = DIM * NH;
    double p[DIM], y[DIM];
#pragma unroll
    for (int r = 0; r < DIM; ++r) {
        p[r] = from[r];
        y[r] = q[r];
    }
    auto end_at = [&](const double *x) {
#pragma unroll
        for (int r = 0; r < DIM; ++r) q[r] = x[r];
    };
    double s = ex.h;
#pragma unroll 1
    for (int crossings = 0;;) {
        // (the caller found q outside c; later ends are looked up here)
        if (crossings > 0 && lookup_d<DIM, TESS>(t, y, Real(0)) == c) {
            end_at(y);
            return c;
        }
        const double *A = ex.A + (size_t)c * NE;
        const double *Fc = ex.F + (size_t)c * ex.nF * NH;
        AffineMap<DIM> M;
        M.load(A);
        double tau = s;
        int kbest = -1;
        // the facets with y beyond them first: lanes then resolve their hits together, whichever facet it is
        unsigned beyond = 0;
#pragma unroll 1
        for (int k = 0; k < ex.nF; ++k) {
            const double *F = Fc + k * NH;
            double ge = __ldg(F + DIM);
#pragma unroll
            for (int r = 0; r < DIM; ++r) ge = fma(__ldg(F + r), y[r], ge);
            if (ge > 0 && __ldg(ex.nbr + c * ex.nF + k) >= 0) beyond |= 1u << k;
        }
#pragma unroll 1
        for (; beyond; beyond &= beyond - 1) {
            const int k = __ffs(beyond) - 1;
            const double *F = Fc + k * NH;
            double g0 = __ldg(F + DIM);
#pragma unroll
            for (int r = 0; r < DIM; ++r) g0 = fma(__ldg(F + r), p[r], g0);
            const double r = (g0 >= 0) ? 0.0 : facet_hit_time<DIM>(M, A, F, p, s, g0);
            if (kbest < 0 || r < tau) {
                tau = r;
                kbest = k;
            }
        }
        if (kbest < 0 || !(tau == tau) || ++crossings > ex.cap) {
            ++ex.unresolved;
            end_at(y);
            return lookup_d<DIM, TESS>(t, y, Real(0));
        }
        flow_taylor<DIM>(M, A, p, tau, p);
        s -= tau;
        c = __ldg(ex.nbr + c * ex.nF + kbest);
        ++ex.crossings;
        if (!(s > 0)) {
            end_at(p);
            return c;
        }
        M.load(ex.A + (size_t)c * NE);
        if (!flow_taylor<DIM>(M, ex.A + (size_t)c * NE, p, s, y)) {
            // the neighbour's flow is too fast for the polynomial over the
            // rest of the sub-step: the reference scheme's sub-step end
            ++ex.unresolved;
            return lookup_d<DIM, TESS>(t, q, Real(0));
        }
    }
}

// EXACT unit: the closed-form step with T (the reference's arithmetic) or one sub-step of the exact flow with S.
template <int DIM>
__device__ __forceinline__ void advance_exact(bool fast, const PState<DIM, double> &s, const double *S,
                                              const double *T, PState<DIM, double> &q)
{
    if (fast) {
        exact_affine<DIM>(q.p, T, s.p);
    } else {
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
            double v = S[r * (DIM + 1) + DIM];
#pragma unroll
            for (int m = 0; m < DIM; ++m) v = fma(S[r * (DIM + 1) + m], s.p[m], v);
            q.p[r] = v;
        }
    }
}

// ------------------------------------------------------------ integration

// One warp integrates the points [ws, we).  Every lane owns one point and
// advances it by one unit per iteration -- a closed-form Trel step or one
// midpoint sub-step, which cost about the same and share most of their
// instructions (advance) -- and claims the next unprocessed point of the
// range as soon as its own is finished.  A point that falls back to
// nStepsODE sub-steps therefore keeps one lane busy, not the whole warp.
// Results do not depend on the schedule: each point follows exactly the
// reference's sequence of operations.
//   Src::load(idx, p)      gives the start position of point idx
//   Snk::put(idx, p)       receives its end position
//   perm (optional, shared memory): the k-th point of the range is
//   ws_base + perm[k - ws_base] (a cell-sorted order inside the tile).
//   start_cells (optional, with perm): cell of point perm_base + i at [i],
//   as computed by the caller's sort pass (same lookup, same point).
//   claim (optional, shared memory, zero on entry): all warps of the CTA
//   share one queue over [ws, we) -- a warp whose lanes finish claims the next
//   points of the whole tile, so no warp idles at the end-of-tile barrier
//   while another still works through a fixed slice.
// Every iteration ends with the question whether the candidate end point is
// still in the cell c of its start: for a closed-form step it is the
// reference's keep test, for a sub-step it decides the cell the next one
// starts in, which the reference would look up from the same point.  Almost
// always the answer needs no lookup: the margin of the point to the facets of
// c, in float, is off by less than kSure, so beyond that its sign is certain
// (InCell); only within it, and where a sub-step moved to another cell, is the
// reference's lookup evaluated.  And
// since the next steps' ends don't wait for the answer, kBurst of them are
// in flight at a time.  Measured on 512 x 512 points, 2D, 64 cells, 50 steps:
// 318 us against 512 with a lookup per step.
constexpr float kSure = 1e-5f;
constexpr int kBurst = 4;

template <int DIM, int TESS>
struct InCell {
    Facets<DIM, TESS> f;
    double ctr[DIM];  // the box's centre in box units

    __device__ __forceinline__ void enter(const Tess &t, int c)
    {
        int kb[DIM];
        cell_box<DIM, TESS>(t, c, kb);
        f.enter(t, c, kb);
#pragma unroll
        for (int i = 0; i < DIM; ++i) ctr[i] = (double)kb[i] + 0.5;
    }
    // 1: p is in the cell, -1: it is not, 0: too close to a facet (or far away, or NaN) for float to tell
    __device__ __forceinline__ int holds(const Tess &t, const double *p) const
    {
        // past the top of boxes flatter in z than in x the facets say nothing (Facets<3, 1>)
        if (DIM == 3 && TESS == 1 && t.inc[0] > t.inc[2] && !(p[2] < t.span[2])) return 0;
        float r[DIM], far = 0.0f;
#pragma unroll
        for (int i = 0; i < DIM; ++i) {
            r[i] = (float)fma(p[i], t.inv_inc[i], -ctr[i]);
            far = fmaxf(far, fabsf(r[i]));
        }
        const float m = f.margin(r);
        return !(far < 8.0f) ? 0 : m > kSure ? 1 : m < -kSure ? -1 : 0;
    }
};

// A burst: up to G steps of one kind (fast: closed-form, else sub-steps) from
// st with the cell's matrix, each from the end of the one before, their ends'
// answers independent of one another; then the steps up to the first end that
// is not for certain in the cell are taken.  Returns how many of the first n;
// `end` is the first end not taken and `verdict` what is known of it.
template <int DIM, int TESS, int SCHEME, int G>
__device__ __forceinline__ int burst(const Tess &t, const InCell<DIM, TESS> &here, bool fast, int n, const double *table,
                                     double h, PState<DIM, double> &st, PState<DIM, double> &end, int &verdict)
{
    constexpr int NE = DIM * (DIM + 1);
    double M[NE];
#pragma unroll
    for (int e = 0; e < NE; ++e) M[e] = table[e];
    PState<DIM, double> q[G + 1];
    int in[G];
    q[0] = st;
#pragma unroll
    for (int g = 0; g < G; ++g) {
        if (SCHEME == SCHEME_EXACT) advance_exact<DIM>(fast, q[g], M, M, q[g + 1]);
        else advance<DIM>(fast, q[g], M, M, h, q[g + 1]);
        in[g] = here.holds(t, q[g + 1].p);
    }
    int took = 0;
    verdict = in[0];
    end = q[1];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        if (took == g && g < n && in[g] > 0) {
            took = g + 1;
            st = q[g + 1];
            if (g + 1 < G) {
                end = q[g + 2 <= G ? g + 2 : G];
                verdict = in[g + 1 < G ? g + 1 : g];
            }
        }
    }
    return took;
}

// Bursts of one (ONE, kernels of their own) where z is clamped inside the domain (3D type I, boxes flatter in x than
// in z): above the clamp the reference's field jumps, points slide along its facets and most bursts end after a step.
// 16 x 20000 points, 4x2x3 boxes: 11.9 ms in bursts, 8.2 one at a time; 2x2x4, flatter in z: 0.56 in bursts.
inline bool one_at_a_time(const Tess &t) { return t.dim == 3 && t.tess == 1 && t.inc[0] < t.inc[2]; }

template <int DIM, int TESS, int SCHEME, bool ONE, class Src, class Snk>
__device__ __forceinline__ void integrate_range(const Tess &t, int nT, int nODE, const double *sA, const double *sT,
                                                int64_t ws, int64_t we, double h, const Src &src, Snk &snk,
                                                unsigned long long &c_fast, unsigned long long &c_fb,
                                                unsigned long long &c_sub, unsigned long long &c_pts,
                                                const int *perm = nullptr, int64_t perm_base = 0,
                                                unsigned long long *claim = nullptr,
                                                const int *start_cells = nullptr, ExactCross *ex = nullptr)
{
    constexpr int NE = DIM * (DIM + 1);
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    int64_t next = ws + 32;
    int64_t k;
    if (claim) {
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(claim, 32ull);
        k = ws + (int64_t)__shfl_sync(FULL, b, 0) + lane;
    } else {
        k = ws + lane;
    }
    bool active = k < we;
    int64_t idx = (active && perm) ? perm_base + perm[k - perm_base] : k;
    PState<DIM, double> st;
    InCell<DIM, TESS> here;
    int steps_left = 0, sub_left = 0, c = 0;
    if (active) {
        src.load(idx, st.p);
        c = start_cells ? start_cells[idx - perm_base] : cell_of<DIM, TESS>(t, st);
        here.enter(t, c);
        steps_left = nT;
        sub_left = (SCHEME == SCHEME_SIMPLE) ? nT * nODE : 0;
    }
    // EXACT: a sub-step that ends outside its cell parks the lane (pend)
    // instead of resolving the exit at once: resolving takes about as long as
    // a hundred units, and done alone it leaves the other 31 lanes idle.  The
    // warp resolves all parked lanes together once kCrossBatch of them wait,
    // every active lane waits, or the oldest has waited kCrossWait votes; a
    // parked lane keeps only the sub-step's start and recomputes its end then
    // (same arithmetic, fewer registers held).  Each point's arithmetic is
    // unchanged.
    constexpr int kCrossBatch = CPAB_EXACT_CROSS_BATCH, kCrossWait = CPAB_EXACT_CROSS_WAIT;
    bool pend = false;
    int pend_votes = 0;
    unsigned n_fb = 0, n_pts = 0;
    while (__any_sync(FULL, active)) {
        bool fin = false;
        if (active && !pend) {
            const bool fast = (SCHEME == SCHEME_REF || SCHEME == SCHEME_EXACT) && sub_left == 0;
            constexpr int G = ONE ? 1 : kBurst;
            const int n = min(G, fast ? steps_left : sub_left);
            PState<DIM, double> end;
            int verdict;
            int took = burst<DIM, TESS, SCHEME, G>(t, here, fast, n, (fast ? sT : sA) + c * NE, h, st, end, verdict);
            bool moved = false;  // `end` taken too
            if (took < n) {
                // which cell matters only where a sub-step ends (EXACT resolves its exits itself)
                int cq = -1;
                if (verdict == 0 || (!fast && SCHEME != SCHEME_EXACT)) cq = cell_of<DIM, TESS>(t, end);
                if (cq != c && fast) {
                    // the end point left the cell: redo the step with nStepsODE sub-steps from its start
                    steps_left -= took;
                    took = 0;
                    sub_left = nODE;
                    ++n_fb;
                } else if (cq != c && SCHEME == SCHEME_EXACT) {
                    pend = true;
                } else {
                    moved = true;
                    st = end;
                    if (cq != c) here.enter(t, cq);
                    c = cq;
                }
            }
            if (fast) {
                steps_left -= took + (moved ? 1 : 0);
            } else {
                sub_left -= took + (moved ? 1 : 0);
                if (SCHEME != SCHEME_SIMPLE && sub_left == 0) --steps_left;
            }
            fin = (SCHEME == SCHEME_SIMPLE) ? (sub_left == 0) : (steps_left == 0);
            if (fin) {
                snk.put(idx, st.p);
                ++n_pts;
            }
        }
        if (SCHEME == SCHEME_EXACT) {
            const unsigned pm = __ballot_sync(FULL, pend);
            if (pm) {
                const unsigned am = __ballot_sync(FULL, active);
                if (__popc(pm) >= kCrossBatch || pm == am || ++pend_votes > kCrossWait) {
                    pend_votes = 0;
                    if (pend) {
                        // the parked sub-step's end, recomputed with the same arithmetic
                        PState<DIM, double> qp;
                        advance_exact<DIM>(false, st, sA + c * NE, sT + c * NE, qp);
                        c = exact_substep_cross<DIM, TESS, double>(t, *ex, c, st.p, qp.p);
                        here.enter(t, c);
                        st = qp;
                        pend = false;
                        --sub_left;
                        if (sub_left == 0) --steps_left;
                        fin = steps_left == 0;
                        if (fin) {
                            snk.put(idx, st.p);
                            ++n_pts;
                        }
                    }
                }
            }
        }
        unsigned done = __ballot_sync(FULL, fin);
        if (done) {
            int64_t base;
            if (claim) {
                unsigned long long b = 0;
                if (lane == 0) b = atomicAdd(claim, (unsigned long long)__popc(done));
                base = ws + (int64_t)__shfl_sync(FULL, b, 0);
            } else {
                base = next;
            }
            if (fin) {
                k = base + __popc(done & lt);
                active = k < we;
                if (active) {
                    idx = perm ? perm_base + perm[k - perm_base] : k;
                    src.load(idx, st.p);
                    c = start_cells ? start_cells[idx - perm_base] : cell_of<DIM, TESS>(t, st);
                    here.enter(t, c);
                    steps_left = nT;
                    sub_left = (SCHEME == SCHEME_SIMPLE) ? nT * nODE : 0;
                }
            }
            next += __popc(done);
        }
    }
    // every closed-form step of a time step is kept or replaced by nStepsODE sub-steps
    c_pts += n_pts;
    if (SCHEME == SCHEME_SIMPLE) {
        c_sub += (unsigned long long)n_pts * nT * nODE;
    } else {
        c_fb += n_fb;
        c_sub += (unsigned long long)n_fb * nODE;
        c_fast += (unsigned long long)n_pts * nT - n_fb;
    }
}

// The reference scheme over [ws, ws + n_range) by one CTA, phase by phase: all
// points take closed-form steps until they are done or leave their cell, then
// the ones that left take their nStepsODE sub-steps, and so on.  In a warp
// whose lanes choose for themselves (integrate_range), a few points with
// sub-steps to take keep the others' lanes idle and the two kinds of step run
// one after the other; here every warp runs one kind, the sub-steps all of the
// same number.  Same steps per point, in the same order.  Positions wait in
// shared memory between phases, kChunk points at a time.  Measured on 512 x 512
// points, 2D, 64 cells, one direction: 240 us against 318, 3D, 320
// cells, 131072 points: 527 against 695.  A launch of a few
// thousand points, whose time is the longest point's chain of steps, is faster
// in integrate_range (1000 points
// there and back: 109 us against 112; 16 x 1000: 135 against 137; 40 x 1000:
// 230 against 218).
constexpr int kChunk = 1024;

__host__ __device__ inline size_t phase_scratch_bytes(int dim, int tile_pts)
{
    const size_t n = tile_pts < kChunk ? tile_pts : kChunk;
    return (n * ((size_t)dim * sizeof(double) + 2 * sizeof(int) + 2 * sizeof(unsigned short)) + 15) & ~(size_t)15;
}

template <int DIM, int TESS, bool ONE, class Src, class Snk>
__device__ __forceinline__ void integrate_phases(const Tess &t, int nT, int nODE, const double *sA, const double *sT,
                                                 int64_t ws, int n_range, double h, const Src &src, Snk &snk,
                                                 unsigned long long &c_fast, unsigned long long &c_fb,
                                                 unsigned long long &c_sub, unsigned long long &c_pts, const int *perm,
                                                 int tile_pts, unsigned char *scratch)
{
    constexpr int NE = DIM * (DIM + 1), kT = ONE ? 1 : 2, kS = ONE ? 1 : 4;  // burst lengths
    __shared__ int s_claim, s_nT, s_nS;
    const int cap = min(tile_pts, kChunk), lane = threadIdx.x & 31;
    const int chunks = (n_range + cap - 1) / cap, each = chunks ? (n_range + chunks - 1) / chunks : 1;
    const unsigned lt = (1u << lane) - 1u;
    double *s_p = reinterpret_cast<double *>(scratch);       // [cap][DIM]
    int *s_c = reinterpret_cast<int *>(s_p + cap * DIM);     // cell
    int *s_left = s_c + cap;                                 // time steps to go
    unsigned short *l_T = reinterpret_cast<unsigned short *>(s_left + cap), *l_S = l_T + cap;
    unsigned n_fb = 0, n_pts = 0;
    for (int b0 = 0; b0 < n_range; b0 += each) {
        const int m = min(each, n_range - b0);
        auto point = [&](int i) { return perm ? perm[b0 + i] : b0 + i; };
        auto finish = [&](int i, const double *p) {
            snk.put(ws + point(i), p);
            ++n_pts;
        };
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            PState<DIM, double> st;
            src.load(ws + point(i), st.p);
#pragma unroll
            for (int k = 0; k < DIM; ++k) s_p[i * DIM + k] = st.p[k];
            s_c[i] = cell_of<DIM, TESS>(t, st);
            s_left[i] = nT;
            l_T[i] = (unsigned short)i;
        }
        if (threadIdx.x == 0) {
            s_nT = m;
            s_claim = s_nS = 0;
        }
        __syncthreads();
        for (;;) {
            const int todo = s_nT;
            // closed-form steps: lanes take points of the list as they get free
            {
                PState<DIM, double> st;
                InCell<DIM, TESS> here;
                int i = 0, c = 0, left = 0;
                bool active = false, more = true;
                for (;;) {
                    const unsigned idle = __ballot_sync(FULL, !active);
                    if (more && idle) {
                        int b = 0;
                        if (lane == 0) b = atomicAdd(&s_claim, __popc(idle));
                        b = __shfl_sync(FULL, b, 0);
                        more = b + __popc(idle) < todo;
                        const int k = b + __popc(idle & lt);
                        if (!active && k < todo) {
                            active = true;
                            i = l_T[k];
                            c = s_c[i];
                            left = s_left[i];
#pragma unroll
                            for (int d = 0; d < DIM; ++d) st.p[d] = s_p[i * DIM + d];
                            here.enter(t, c);
                        }
                    }
                    if (!__any_sync(FULL, active)) break;
                    if (active) {
                        PState<DIM, double> end;
                        int verdict;
                        const int n = min(kT, left);
                        const int took = burst<DIM, TESS, SCHEME_REF, kT>(t, here, true, n, sT + c * NE, h, st, end,
                                                                          verdict);
                        left -= took;
                        if (took < n) {
                            if (verdict == 0 && cell_of<DIM, TESS>(t, end) == c) {
                                st = end;
                                --left;
                            } else {
                                // the end point left the cell: redo the step with nStepsODE sub-steps
#pragma unroll
                                for (int d = 0; d < DIM; ++d) s_p[i * DIM + d] = st.p[d];
                                s_left[i] = left;
                                l_S[atomicAdd(&s_nS, 1)] = (unsigned short)i;
                                active = false;
                                ++n_fb;
                            }
                        }
                        if (active && left == 0) {
                            finish(i, st.p);
                            active = false;
                        }
                    }
                }
            }
            __syncthreads();
            const int leaving = s_nS;
            if (threadIdx.x == 0) s_nT = s_claim = 0;
            if (leaving == 0) break;
            __syncthreads();
            for (int k = threadIdx.x; k < leaving; k += blockDim.x) {
                const int i = l_S[k];
                PState<DIM, double> st;
                InCell<DIM, TESS> here;
                int c = s_c[i], sub = nODE;
#pragma unroll
                for (int d = 0; d < DIM; ++d) st.p[d] = s_p[i * DIM + d];
                here.enter(t, c);
                while (sub > 0) {
                    PState<DIM, double> end;
                    int verdict;
                    const int n = min(kS, sub);
                    const int took = burst<DIM, TESS, SCHEME_REF, kS>(t, here, false, n, sA + c * NE, h, st, end, verdict);
                    sub -= took;
                    if (took < n) {
                        const int cq = cell_of<DIM, TESS>(t, end);
                        st = end;
                        --sub;
                        if (cq != c) here.enter(t, cq);
                        c = cq;
                    }
                }
                const int left = s_left[i] - 1;
                if (left == 0) {
                    finish(i, st.p);
                } else {
                    s_left[i] = left;
                    s_c[i] = c;
#pragma unroll
                    for (int d = 0; d < DIM; ++d) s_p[i * DIM + d] = st.p[d];
                    l_T[atomicAdd(&s_nT, 1)] = (unsigned short)i;
                }
            }
            __syncthreads();
            if (threadIdx.x == 0) s_nS = 0;
            __syncthreads();
        }
        __syncthreads();
    }
    c_pts += n_pts;
    c_fb += n_fb;
    c_sub += (unsigned long long)n_fb * nODE;
    c_fast += (unsigned long long)n_pts * nT - n_fb;
}

}  // namespace cpab
