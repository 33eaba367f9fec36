// cpab_jump.cuh -- the FP32 integration: many steps of a scheme at once
// through the powers of a cell's step maps.
//
// While a point stays in one cell, each closed-form step applies the same
// affine map T_c = expm(dt A_c), and each sub-step the same map S_c (the
// explicit-midpoint map, or expm(h A_c) for the exact scheme): 2^k steps are
// one application of the map's 2^k-th power.  A CTA stages these powers per
// instance (level l of a map: its 2^(l r)-th power), and a unit of work is
// one of them.  The scheme's sequence of steps is unchanged: every step
// skipped over is one that the scheme would have taken from inside the cell
// to inside the cell.  That is certain when the path cannot leave the cell in
// between, which the two end points show:
//   * both lie in the cell c (the scheme's own lookup), and
//   * the larger of their margins m (least distance to a facet shared with
//     another cell, box units) is at least tau^2 B / 2, where B
//     bounds the second derivative of every facet functional along the path
//     over the jump's time tau: a functional g with g(0), g(tau) <= 0, one of
//     them <= -tau^2 B / 2 and |g''| <= B stays <= 0 in between.
// With L the cell's linear part in box units, rho = |L|_1, x = rho |tau|: the
// path's velocity is e^{L t} v0, so B <= rho e^x |v0|_1 (facet functionals
// have coefficients 0, +-1), and its displacement d = tau phi(L tau) v0,
// phi(z) = (e^z - 1)/z, gives |v0|_1 <= |d|_1 / (tau (2 - phi(x))).  So the
// margin needed is |d|_1 kappa with
//     kappa = 1/2 x e^x / (2 - phi(x))        (x < 1.2, else no jump),
// tabulated per cell and level with 2 % to spare for the float arithmetic.  (The
// midpoint sub-steps' flow is that of log(S) / h, for which rho is raised.)
//
// The argument takes facets that are planes.  The tetrahedra's are bent where
// the domain ends (or z is clamped): beyond, the lookup takes the nearest
// coordinate inside.  A jump therefore starts and ends inside, and in a box
// that touches an end its margin is twice the above: between its ends the path
// may pass the end by e_i(s) <= B_i s (tau - s) / 2 in coordinate i, B_i
// bounding that coordinate's second derivative, sum B_i <= B; the facet's
// functional of the clamped coordinates differs from g by sum e_i at most, and
// g(s) + sum e_i(s) <= (tau - s) / tau (-m + 2 B tau s / 2) <= 0 for
// m >= tau^2 B.  With x boxes larger than z boxes the cells past the top are
// others altogether (the lookup folds z back into the box): no jumps in a box
// below it whose field crosses it.
//
// A jump that is not certain is dropped, and the exit estimated from the rate
// at which the dropped candidate lost its margin (`per_m`); the next jumps aim
// short of it (8.7 units per point; 11.4 by bisection down the levels).  Level
// 0 is the scheme itself: a closed-form step is kept or replaced by
// nStepsODE sub-steps, a sub-step always taken.
//
// A lane keeps its point's position r in its box (from the box's centre, in
// box units, |r| <= 1/2 inside) as a compensated pair, and the maps act on r:
// rounding is then relative to a box, not to the domain, and the margin of a
// candidate end point needs no cell lookup -- it is the smallest of the facet
// functionals of the lane's current cell (Facets), negative when the
// candidate left it.  The cell is looked up again only where a sub-step leaves
// it.
//
// Measured on 2D prior fields (64 cells, dt 0.02, 50 steps, 100 sub-steps
// per leaving step): 8.7 units per point instead of 95.  8.4 M points in 1024
// instances: 3.17 ms with one step per unit, 0.73 ms.
// FP32 error against 64 bits of the registration likelihood (256 fields x
// 256^2 pixels): 5.1e-8 before, 2.8e-8.
#pragma once

#include "cpab_integrate.cuh"

namespace cpab {

// Units of work a lane runs between changes of phase (kUnits), changes of
// phase between the warp's votes (kRounds), and units of a first pass.
// Measured on 8.4 M points (2D, 64 cells): 3 x 2 0.70 ms, 2 x 3 0.71, 2 x 2
// and 4 x 1 0.72, 1 x 4 0.73, 2 x 1 0.80.
constexpr int kUnits = 3, kRounds = 2, kFirstUnits = 5;
// Resident CTAs of 256 threads the register allocation must allow per SM:
// 4 (64 registers) in 1D and 2D -- 3 and 5 measured 0.72 and 0.77 ms on the
// same points -- and 2 in 3D, whose tables leave room for no more (0.25 ms
// against 0.27 ms for 3 on 0.5 M points of 320 cells).
template <int DIM>
constexpr int kJumpCtas = DIM == 3 ? 2 : 4;

// Shared memory of the tables: the maps (increments M - I, column-major),
// then kappa of every level above 0.  (Level 0 reads kappa too and ignores it:
// an entry before its own table's, in the maps where there is none.)
__host__ __device__ inline size_t jump_bytes(const JumpCfg &j, int dim, int nC, size_t el = sizeof(float))
{
    const size_t kap = (size_t)(j.nT > 0 ? j.nT - 1 : 0) + j.nS - 1;
    const size_t b = ((size_t)(j.nT + j.nS) * dim * (dim + 1) + kap) * nC * el;
    return (b + 15) & ~(size_t)15;
}

// log2 of the ratio between levels: every power of two while the tables stay
// within 40 KB, every fourth power up to 64 KB, every eighth or sixteenth up to
// 112 KB (two CTAs per SM), else level 0 alone; fewer levels when `avail`
// bytes (what shared memory the kernel's other needs leave) do not hold the
// choice.  The choice depends on the space and the step counts, not on the
// batch, so results do not either.
inline JumpCfg jump_cfg(int dim, int nC, int nTimeSteps, int nStepsODE, int scheme, size_t avail,
                        size_t el = sizeof(float), int r_least = 1)
{
    auto log2i = [](long long v) {
        int k = 0;
        while (v > 1) {
            v >>= 1;
            ++k;
        }
        return k;
    };
    const int lt = log2i(nTimeSteps);
    int ls = log2i(scheme == SCHEME_SIMPLE ? (long long)nTimeSteps * nStepsODE : nStepsODE);
    if (ls > 8) ls = 8;
    JumpCfg j{0, 0, 0, 0, 0};
    for (int r : {1, 2, 3, 4, 5, 6, 31}) {
        if (r < r_least) continue;
        j.r = r;
        j.mul = (32 + r - 1) / r;
        j.nT = scheme == SCHEME_SIMPLE ? 0 : (lt > 8 ? 8 : lt) / r + 1;
        j.nS = ls / r + 1;
        const size_t b = jump_bytes(j, dim, nC, el), budget = (size_t)(r == 1 ? 40 : r == 2 ? 64 : 112) * 1024;
        if (r == 31 || (b <= budget && b <= avail)) break;
    }
    return j;
}

template <typename Real>
struct JumpTables {
    const Real *map;  // [nT + nS][nC][DIM * (DIM + 1)]
    const Real *kap;  // [nT - 1 + nS - 1][nC]
};

// 2 D + D_lin D: the increment of a map applied twice.
template <int DIM>
__device__ __forceinline__ void twice(double *D)
{
    constexpr int NH = DIM + 1, NE = DIM * NH;
    double D2[NE];
#pragma unroll
    for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int col = 0; col < NH; ++col) {
            double s = 2.0 * D[r * NH + col];
#pragma unroll
            for (int k = 0; k < DIM; ++k) s = fma(D[r * NH + k], D[k * NH + col], s);
            D2[r * NH + col] = s;
        }
#pragma unroll
    for (int e = 0; e < NE; ++e) D[e] = D2[e];
}

// The midpoint map's increment h A + h^2/2 L A  (A = [L | b]).
template <int DIM>
__device__ __forceinline__ void midpoint_increment(const double *a, double h, double *D)
{
    constexpr int NH = DIM + 1;
#pragma unroll
    for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int col = 0; col < NH; ++col) {
            double l2 = 0.0;
#pragma unroll
            for (int k = 0; k < DIM; ++k) l2 += a[r * NH + k] * a[k * NH + col];
            D[r * NH + col] = h * (a[r * NH + col] + 0.5 * h * l2);
        }
}

// Stage one instance's tables from its signed A and Trel: one thread per
// (map, cell) squares the increment D = M - I upwards in FP64,
// (I + D)^2 - I = 2 D + D_lin D.
template <int DIM, int TESS, typename Real = float>
__device__ __forceinline__ JumpTables<Real> stage_jump(const double *gA, const double *gT, const Tess &t,
                                                       const JumpCfg &jc, double dt, double h, bool exact_sub,
                                                       unsigned char *smem)
{
    constexpr int NH = DIM + 1, NE = DIM * NH;
    const int nC = t.nC;
    Real *map = reinterpret_cast<Real *>(smem);
    Real *kap = map + (size_t)(jc.nT + jc.nS) * nC * NE;
    const int kinds = jc.nT > 0 ? 2 : 1;
#pragma unroll 1
    for (int i = threadIdx.x; i < kinds * nC; i += blockDim.x) {
        const bool sub = i >= nC || jc.nT == 0;
        const int c = i < nC ? i : i - nC;
        const double *a = gA + (size_t)c * NE;
        double D[NE];
        double tau = sub ? h : dt;
        if (!sub) {
#pragma unroll
            for (int e = 0; e < NE; ++e) D[e] = gT[(size_t)c * NE + e] - (e % NH == e / NH ? 1.0 : 0.0);
        } else if (!exact_sub) {
            midpoint_increment<DIM>(a, h, D);
        } else {
            // expm(h A) - I by its Taylor sum, to the sum's rounding
            double w[NE];
#pragma unroll
            for (int e = 0; e < NE; ++e) D[e] = w[e] = h * a[e];
#pragma unroll 1
            for (int k = 2; k <= 40; ++k) {
                double nw[NE], big = 0.0, am = 0.0;
#pragma unroll
                for (int r = 0; r < DIM; ++r)
#pragma unroll
                    for (int col = 0; col < NH; ++col) {
                        double v = 0.0;
#pragma unroll
                        for (int m = 0; m < DIM; ++m) v = fma(a[r * NH + m], w[m * NH + col], v);
                        nw[r * NH + col] = v * (h / k);
                    }
#pragma unroll
                for (int e = 0; e < NE; ++e) {
                    w[e] = nw[e];
                    D[e] += w[e];
                    big = fmax(big, fabs(w[e]));
                    am = fmax(am, fabs(D[e]));
                }
                if (!(big > 1e-18 * am)) break;
            }
        }
        // the box's centre
        double ctr[DIM];
        {
            int kb[DIM];
            cell_box<DIM, TESS>(t, c, kb);
#pragma unroll
            for (int r = 0; r < DIM; ++r) ctr[r] = ((double)kb[r] + 0.5) * t.inc[r];
        }
        // rho = |L|_1 in box units
        double rho = 0.0;
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
            double s = 0.0;
#pragma unroll
            for (int r = 0; r < DIM; ++r) s += fabs(a[r * NH + k]) * t.inv_inc[r];
            rho = fmax(rho, s * t.inc[k]);
        }
        // the midpoint map's flow is that of log(S) / h = L - h^2 L^3 / 6 + ...: at most this much steeper
        if (sub && !exact_sub) rho *= 1.0 + h * h * rho * rho / 3.0;
        // twice the margin where a facet is bent in the box
        float bent = 1.0f;
        if constexpr (DIM == 3 && TESS == 1) {
            int kb[DIM];
            cell_box<DIM, TESS>(t, c, kb);
            const int n[3] = {t.nC0, t.nC1, t.nC2};
#pragma unroll
            for (int r = 0; r < DIM; ++r)
                if (kb[r] == 0 || kb[r] == n[r] - 1 || (r == 2 && (double)(kb[r] + 1) * t.inc[r] >= t.hi[2])) bent = 2.0f;
            if (t.inc[0] > t.inc[2] && kb[DIM - 1] == n[2] - 1) {
                // the velocity across the top, at its middle and the most it differs from that
                const double *az = a + 2 * NH;
                const double ax = az[0] * t.inc[0], ay = az[1] * t.inc[1], top = az[2] * t.span[2] + az[3];
                const double mid = ax * (kb[0] + 0.5) + ay * (kb[1] + 0.5) + top;
                const double size = fabs(ax) * (kb[0] + 1) + fabs(ay) * (kb[1] + 1) + fabs(az[2] * t.span[2]) + fabs(az[3]);
                if (!(fabs(mid) + 0.5 * (fabs(ax) + fabs(ay)) <= 1e-12 * size)) bent = CUDART_INF_F;
            }
        }
        const int levels = sub ? jc.nS : jc.nT, row0 = sub ? jc.nT : 0;
        const int kap0 = sub ? (jc.nT > 0 ? jc.nT - 1 : 0) : 0;
#pragma unroll 1
        for (int l = 0; l < levels; ++l) {
            Real *m = map + ((size_t)(row0 + l) * nC + c) * NE;
#pragma unroll
            for (int r = 0; r < DIM; ++r) {
                double off = D[r * NH + DIM];  // the displacement of the box's centre
#pragma unroll
                for (int col = 0; col < DIM; ++col) {
                    m[col * DIM + r] = (Real)(D[r * NH + col] * t.inc[col] * t.inv_inc[r]);
                    off = fma(D[r * NH + col], ctr[col], off);
                }
                m[DIM * DIM + r] = (Real)(off * t.inv_inc[r]);
            }
            if (l > 0) {
                const float x = (float)(rho * fabs(tau)), em = expm1f(x), room = 2.0f - em / x;
                kap[(size_t)(kap0 + l - 1) * nC + c] =
                    x < 1e-6f && bent < 3.0f ? 1e-6f : (x < 1.2f ? bent * 0.51f * x * (1.0f + em) / room : CUDART_INF_F);
            }
            if (l + 1 < levels) {
#pragma unroll 1
                for (int q = 0; q < jc.r; ++q) {
                    twice<DIM>(D);
                    tau *= 2.0;
                }
            }
        }
    }
    return JumpTables<Real>{map, kap};
}

// ------------------------------------------------------------ walkers
//
// One lane's point: its cell c, margin m, and position.
//   place(t, x)          at the absolute position x (looks the cell up)
//   place_in(t, x, c)    the same, in the given cell (margin unknown: 0)
//   position(t, x)       the absolute position
//   step(t, map, q)      q: the candidate end of one composed step with the
//                        column-major map; returns |d|_1 in box units; q.m is
//                        its margin, negative when it left the cell
//   keeps(t, q)          after a single step with q.m < 0: whether it is in the
//                        cell all the same (kept out of the units' way)
//   take(q, yes)         moves to q, in the same cell, when yes
//   leave(t, q)          moves to q, looking its cell up
//   where(t, q, x)       absolute position of a candidate

// Position in a box, box units from the centre: float as a compensated pair
// hi + lo, double as it is.
template <int DIM, typename Real>
struct BoxPos;
template <int DIM>
struct BoxPos<DIM, float> {
    float hi[DIM], lo[DIM];
    __device__ __forceinline__ float x(int i) const { return hi[i] + lo[i]; }
};
template <int DIM>
struct BoxPos<DIM, double> {
    double hi[DIM];
    __device__ __forceinline__ double x(int i) const { return hi[i]; }
};

template <int DIM, typename Real>
struct BoxCand {
    BoxPos<DIM, Real> p;
    Real x[DIM];
    Real m;
};

template <int DIM, int TESS, typename Real>
struct FacetsOf {
    using type = Facets<DIM, TESS>;
};
template <typename Real>
struct FacetsOf<3, 1, Real> {
    using type = InnerTet<Real>;
};

template <int DIM, int TESS, typename Real>
struct WalkLocal {
    BoxPos<DIM, Real> p;
    int c;
    Real m;
    typename FacetsOf<DIM, TESS, Real>::type f;

    __device__ __forceinline__ void set_local(const Tess &t, const double *x, const int *kb)
    {
#pragma unroll
        for (int i = 0; i < DIM; ++i) {
            const double r = fma(x[i], t.inv_inc[i], -((double)kb[i] + 0.5));
            p.hi[i] = (Real)r;
            if constexpr (sizeof(Real) == 4) p.lo[i] = (float)(r - (double)p.hi[i]);
        }
    }
    // float coordinates in float arithmetic: x / inc with the low part of
    // 1/inc, rounded once relative to the position in the box
    __device__ __forceinline__ void set_local(const Tess &t, const float *x, const int *kb)
    {
#pragma unroll
        for (int i = 0; i < DIM; ++i) {
            p.hi[i] = fmaf(x[i], t.finv_inc[i], -((float)kb[i] + 0.5f));
            p.lo[i] = x[i] * t.finv_inc_lo[i];
        }
    }
    template <typename Elem>
    __device__ __forceinline__ void box_of(const Tess &t, const Elem *x, int *kb) const
    {
        const int n[3] = {t.nC0, t.nC1, t.nC2};
#pragma unroll
        for (int i = 0; i < DIM; ++i) {  // NaN -> 0
            const Real u = floor((Real)x[i] * (Real)(sizeof(Real) == 4 ? (double)t.finv_inc[i] : t.inv_inc[i]));
            kb[i] = (int)least(most(u, Real(0)), Real(n[i] - 1));
        }
    }
    static __device__ __forceinline__ double exact_x(const BoxPos<DIM, float> &q, int i)
    {
        return (double)q.hi[i] + (double)q.lo[i];
    }
    static __device__ __forceinline__ double exact_x(const BoxPos<DIM, double> &q, int i) { return q.hi[i]; }
    __device__ __forceinline__ void to_absolute(const Tess &t, const BoxPos<DIM, Real> &q, double *x) const
    {
        int kb[DIM];
        cell_box<DIM, TESS>(t, c, kb);
#pragma unroll
        for (int i = 0; i < DIM; ++i)
            x[i] = (((double)kb[i] + 0.5) + exact_x(q, i)) * t.inc[i];
    }
    // the same rounded to float: the centre (k + 1/2) inc as a float and its
    // rest, and one rounding of the sum
    __device__ __forceinline__ void to_absolute(const Tess &t, const BoxPos<DIM, Real> &q, float *x) const
    {
        int kb[DIM];
        cell_box<DIM, TESS>(t, c, kb);
#pragma unroll
        for (int i = 0; i < DIM; ++i) {
            const float k = (float)kb[i] + 0.5f, ctr = k * t.finc[i];
            const float rest = fmaf(k, t.finc[i], -ctr) + k * t.finc_lo[i];
            x[i] = ctr + (rest + fmaf(q.hi[i], t.finc[i], q.lo[i] * t.finc[i]));
        }
    }
    template <typename Elem>
    __device__ __forceinline__ void position(const Tess &t, Elem *x) const
    {
        to_absolute(t, p, x);
    }
    __device__ __forceinline__ void where(const Tess &t, const BoxCand<DIM, Real> &q, double *x) const
    {
        to_absolute(t, q.p, x);
    }
    __device__ __forceinline__ void move(const BoxCand<DIM, Real> &q, bool yes)
    {
#pragma unroll
        for (int i = 0; i < DIM; ++i) {
            p.hi[i] = yes ? q.p.hi[i] : p.hi[i];
            if constexpr (sizeof(Real) == 4) p.lo[i] = yes ? q.p.lo[i] : p.lo[i];
        }
        m = yes ? q.m : m;
    }
    // the box of a candidate, with its position relative to that box
    __device__ __forceinline__ void shift_box(const Tess &t, BoxCand<DIM, Real> &q, int *kb) const
    {
        const int n[3] = {t.nC0, t.nC1, t.nC2};
        cell_box<DIM, TESS>(t, c, kb);
#pragma unroll
        for (int i = 0; i < DIM; ++i) {
            const Real s = least(most(floor(q.x[i] + Real(0.5)), Real(-kb[i])), Real(n[i] - 1 - kb[i]));
            kb[i] += (int)s;
            q.p.hi[i] -= s;
            q.x[i] = q.p.x(i);
        }
    }
    __device__ __forceinline__ Real advance(const Real *map, BoxCand<DIM, Real> &q) const
    {
        if constexpr (sizeof(Real) == 8) {
            double len = 0.0;
#pragma unroll
            for (int r = 0; r < DIM; ++r) {
                double d = map[DIM * DIM + r];
#pragma unroll
                for (int k = 0; k < DIM; ++k) d = fma(map[k * DIM + r], p.hi[k], d);
                q.x[r] = q.p.hi[r] = p.hi[r] + d;
                len += fabs(d);
            }
            return len;
        } else {
            return advance_f(map, q);
        }
    }
    __device__ __forceinline__ float advance_f(const float *map, BoxCand<DIM, float> &q) const
    {
        float mm[DIM * (DIM + 1)];
        load_cell<DIM>(map, mm);
        if constexpr (DIM == 1) {
            const float d = fmaf(mm[0], p.hi[0] + p.lo[0], mm[1]);
            const float s = p.hi[0] + d;
            q.p.lo[0] = p.lo[0] + (d - (s - p.hi[0]));
            q.p.hi[0] = s;
            q.x[0] = s + q.p.lo[0];
            return fabsf(d);
        } else {
            // coordinates 0 and 1 as one pair (FFMA2 / FADD2)
            const float2 h = make_float2(p.hi[0], p.hi[1]), l = make_float2(p.lo[0], p.lo[1]);
            const float2 r = __fadd2_rn(h, l);
            float2 d = __ffma2_rn(make_float2(mm[0], mm[1]), make_float2(r.x, r.x),
                                  make_float2(mm[DIM * DIM], mm[DIM * DIM + 1]));
            d = __ffma2_rn(make_float2(mm[DIM], mm[DIM + 1]), make_float2(r.y, r.y), d);
            float len = 0.0f;
            if constexpr (DIM == 3) {
                const float z = p.hi[2] + p.lo[2];
                d = __ffma2_rn(make_float2(mm[6], mm[7]), make_float2(z, z), d);
                const float dz = fmaf(mm[8], z, fmaf(mm[5], r.y, fmaf(mm[2], r.x, mm[11])));
                const float s = p.hi[2] + dz;
                q.p.lo[2] = p.lo[2] + (dz - (s - p.hi[2]));
                q.p.hi[2] = s;
                q.x[2] = s + q.p.lo[2];
                len = fabsf(dz);
            }
            const float2 s = __fadd2_rn(h, d);
            const float2 l2 = __fadd2_rn(l, __fadd2_rn(d, neg2(__fadd2_rn(s, neg2(h)))));
            const float2 x = __fadd2_rn(s, l2);
            q.p.hi[0] = s.x;
            q.p.hi[1] = s.y;
            q.p.lo[0] = l2.x;
            q.p.lo[1] = l2.y;
            q.x[0] = x.x;
            q.x[1] = x.y;
            return len + (fabsf(d.x) + fabsf(d.y));
        }
    }
};

// Box cells (1D and type II).
template <int DIM, typename Real>
struct WalkBox : WalkLocal<DIM, 2, Real> {
    using B = WalkLocal<DIM, 2, Real>;
    using Cand = BoxCand<DIM, Real>;
    using B::c;
    using B::f;
    using B::m;
    using B::p;

    __device__ __forceinline__ void enter(const Tess &t, const int *kb)
    {
        const int n[3] = {t.nC0, t.nC1, t.nC2};
        int stride = 1;
        c = 0;
#pragma unroll
        for (int i = 0; i < DIM; ++i) {
            c += kb[i] * stride;
            stride *= n[i];
        }
        f.enter(t, c, kb);
    }
    template <typename Elem>
    __device__ __forceinline__ void place(const Tess &t, const Elem *x)
    {
        int kb[DIM];
        Real r[DIM];
        B::box_of(t, x, kb);
        B::set_local(t, x, kb);
        enter(t, kb);
#pragma unroll
        for (int i = 0; i < DIM; ++i) r[i] = p.x(i);
        m = f.margin(r);
    }
    template <typename Elem>
    __device__ __forceinline__ void place_in(const Tess &t, const Elem *x, int cell)
    {
        int kb[DIM];
        cell_box<DIM, 2>(t, cell, kb);
        B::set_local(t, x, kb);
        enter(t, kb);
        m = 0;
    }
    __device__ __forceinline__ Real step(const Tess &, const Real *map, Cand &q) const
    {
        const Real len = B::advance(map, q);
        q.m = f.margin(q.x);
        return len;
    }
    __device__ __forceinline__ bool keeps(const Tess &, const Cand &) const { return false; }
    __device__ __forceinline__ void take(const Cand &q, bool yes) { B::move(q, yes); }
    __device__ __forceinline__ void leave(const Tess &t, Cand &q)
    {
        int kb[DIM];
        B::shift_box(t, q, kb);
        enter(t, kb);
        p = q.p;
        m = f.margin(q.x);
    }
};

// 2D type I: the triangle by the signs of x - y and x + y, in the domain and
// outside (Facets<2, 1>).
template <typename Real>
struct WalkTri : WalkLocal<2, 1, Real> {
    using B = WalkLocal<2, 1, Real>;
    using Cand = BoxCand<2, Real>;
    using B::c;
    using B::f;
    using B::m;
    using B::p;

    __device__ __forceinline__ void enter(const Tess &t, const int *kb, bool up, bool right)
    {
        c = (kb[0] + kb[1] * t.nC0) * 4 + (up ? (right ? 2 : 3) : (right ? 1 : 0));
        f.enter(t, c, kb);
    }
    template <typename Elem>
    __device__ __forceinline__ void place(const Tess &t, const Elem *x)
    {
        int kb[2];
        B::box_of(t, x, kb);
        B::set_local(t, x, kb);
        const Real r[2] = {p.x(0), p.x(1)};
        enter(t, kb, r[0] < r[1], r[0] + r[1] > Real(0));
        m = f.margin(r);
    }
    template <typename Elem>
    __device__ __forceinline__ void place_in(const Tess &t, const Elem *x, int cell)
    {
        int kb[2];
        c = cell;
        cell_box<2, 1>(t, cell, kb);
        B::set_local(t, x, kb);
        f.enter(t, cell, kb);
        m = 0;
    }
    __device__ __forceinline__ Real step(const Tess &, const Real *map, Cand &q) const
    {
        const Real len = B::advance(map, q);
        q.m = f.margin(q.x);
        return len;
    }
    __device__ __forceinline__ bool keeps(const Tess &, const Cand &) const { return false; }
    __device__ __forceinline__ void take(const Cand &q, bool yes) { B::move(q, yes); }
    __device__ __forceinline__ void leave(const Tess &t, Cand &q)
    {
        int kb[2];
        B::shift_box(t, q, kb);
        enter(t, kb, q.x[0] < q.x[1], q.x[0] + q.x[1] > Real(0));
        p = q.p;
        m = f.margin(q.x);
    }
};

// 3D type I: a new cell is looked up at the absolute position.  A candidate past
// the domain, where the lookup takes the nearest point inside and no margin is
// a distance, is outside to a step (InnerTet: q.m < kPast); of a single step
// `keeps` then asks the lookup.  Jumps never end there, nor (m = 0) start.
// Points on the domain's boundary, which stay there up to rounding, count as
// inside.
template <typename Real>
struct WalkTet : WalkLocal<3, 1, Real> {
    using B = WalkLocal<3, 1, Real>;
    using Cand = BoxCand<3, Real>;
    using B::c;
    using B::f;
    using B::m;
    using B::p;

    static __device__ __forceinline__ int cell_at(const Tess &t, const float *a) { return fast_cell<3, 1>(t, a); }
    static __device__ __forceinline__ int cell_at(const Tess &t, const double *a) { return exact_cell<3, 1>(t, a); }
    // the cell of a position relative to the box of c
    __device__ __forceinline__ int lookup(const Tess &t, const Real *x) const
    {
        Real a[3];
        int kb[3];
        cell_box<3, 1>(t, c, kb);
#pragma unroll
        for (int i = 0; i < 3; ++i) a[i] = ((Real)kb[i] + Real(0.5) + x[i]) * (Real)t.inc[i];
        return cell_at(t, a);
    }
    template <typename Elem>
    __device__ __forceinline__ void place(const Tess &t, const Elem *x)
    {
        Real a[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) a[i] = (Real)x[i];
        place_in(t, x, cell_at(t, a));
        set_margin();
    }
    __device__ __forceinline__ void set_margin()
    {
        const Real r[3] = {p.x(0), p.x(1), p.x(2)};
        m = most(f.margin(r), Real(0));
    }
    template <typename Elem>
    __device__ __forceinline__ void place_in(const Tess &t, const Elem *x, int cell)
    {
        int kb[3];
        c = cell;
        cell_box<3, 1>(t, cell, kb);
        f.enter(t, cell, kb);
        B::set_local(t, x, kb);
        m = 0;
    }
    __device__ __forceinline__ Real step(const Tess &, const Real *map, Cand &q) const
    {
        const Real len = B::advance(map, q);
        q.m = f.margin(q.x);
        return len;
    }
    __device__ __forceinline__ bool keeps(const Tess &t, const Cand &q) const
    {
        return q.m < InnerTet<Real>::kPast && lookup(t, q.x) == c;
    }
    // the margin of x past the domain, by the clamped coordinates (0: not known)
    __device__ __forceinline__ Real margin_past(const Tess &t, const Real *x) const
    {
        if (t.inc[0] > t.inc[2]) return 0;
        int kb[3];
        Facets<3, 1> clamped;
        cell_box<3, 1>(t, c, kb);
        clamped.enter(t, c, kb);
        return clamped.margin(x);
    }
    __device__ __forceinline__ void take(const Cand &q, bool yes) { B::move(q, yes); }
    __device__ __forceinline__ void leave(const Tess &t, Cand &q)
    {
        double x[3];
        const int cell = lookup(t, q.x);
        B::where(t, q, x);
        place_in(t, x, cell);
        set_margin();
    }
};

template <int DIM, int TESS, typename Real>
struct WalkerOf {
    using type = WalkBox<DIM, Real>;
};
template <typename Real>
struct WalkerOf<2, 1, Real> {
    using type = WalkTri<Real>;
};
template <typename Real>
struct WalkerOf<3, 1, Real> {
    using type = WalkTet<Real>;
};

// One point on its way through calc_T, for the adjoint: the moves that calc_T
// makes, so that the gradient is that of its branch at every step.
//
// FP32: the decisions of integrate_jump for one lane on its own (whose first
// pass makes the same moves where it gets through).
//
// FP64: calc_T goes step by step in the reference's arithmetic, this in jumps,
// so positions differ by rounding: `err` (|.|_1, box units) gains kRound reach a
// step, `reach` bounding the position in boxes, and grows or shrinks with a
// move's linear part.  A decision that a margin within 2 err makes (a jump's
// ends beyond that leave 3/4 of it in between) is in doubt, and ExactPath, which
// goes step by step from the start of the point or from where it was last
// asked, catches up, makes it, and hands over its position (settled_unit): some 1e-7
// of the points, and those of grids that move along a facet, on each of their
// steps.

// calc_T in its FP64 arithmetic: at x in cell c (`here`, entered by the caller), `left` closed-form steps to go, or
// sub-steps of the first of `steps`.
template <int DIM, int TESS>
struct ExactPath {
    double x[DIM];
    int c, left, steps;
    bool sub;

    __device__ __forceinline__ void begin(const Tess &t, const double *from, int nT)
    {
#pragma unroll
        for (int i = 0; i < DIM; ++i) x[i] = from[i];
        c = exact_cell<DIM, TESS>(t, x);
        left = nT;
        steps = 0;
        sub = false;
    }
    __device__ __forceinline__ bool done() const { return left == 0; }
    // One step, as a move from r in the box of its cell by row mi of level 0 (s_row: the first of the sub-steps'); false:
    // none, but the finding that sub-steps follow.
    __device__ __forceinline__ bool step(const Tess &t, const double *A, const double *T, double h, int nODE, int s_row,
                                         InCell<DIM, TESS> &here, int &mi, double *r)
    {
        constexpr int NE = DIM * (DIM + 1);
        double y[DIM];
        if (sub) {
#pragma unroll
            for (int i = 0; i < DIM; ++i) y[i] = x[i];
            exact_midpoint<DIM>(y, A + (size_t)c * NE, h);
        } else {
            exact_affine<DIM>(y, T + (size_t)c * NE, x);
        }
        const int in = here.holds(t, y), cy = in > 0 ? c : in < 0 && !sub ? -1 : exact_cell<DIM, TESS>(t, y);
        if (!sub && cy != c) {
            steps = left;
            left = nODE;
            sub = true;
            return false;
        }
        mi = (sub ? s_row : 0) + c;
#pragma unroll
        for (int i = 0; i < DIM; ++i) {
            r[i] = fma(x[i], t.inv_inc[i], -here.ctr[i]);
            x[i] = y[i];
        }
        if (cy != c) here.enter(t, cy);
        c = cy;
        --left;
        if (sub && left == 0) {
            sub = false;
            left = --steps;
        }
        return true;
    }
    // how far a path has come that has `n` closed-form steps to go, or as many sub-steps of the first of k: < 0: not as
    // far as this one, 0: as far
    __device__ __forceinline__ int behind(bool s, int n, int k) const
    {
        const int mine = sub ? steps : left, its = s ? k : n;
        if (mine != its) return mine - its;
        if (sub != s) return sub ? -1 : 1;
        return sub ? left - n : 0;
    }
};

// Take e to where a path (see `behind`) of the point at x0 stands, from its last place or, where that is ahead, from the
// start, and, `one` more step on; what step() returned.  Out of line: rare, and its lookups would take the registers of
// the jumps around it.
template <int DIM, int TESS>
__device__ __noinline__ bool catch_up(const Tess &t, const double *A, const double *T, double h, int nT, int nODE, int s_row,
                                      const double *x0, bool sub, int left, int steps, bool one, ExactPath<DIM, TESS> &e,
                                      int &mi, double *r)
{
    if (e.c < 0 || e.behind(sub, left, steps) < 0) {
        double x[DIM];
#pragma unroll
        for (int i = 0; i < DIM; ++i) x[i] = x0[i];
        e.begin(t, x, nT);
    }
    InCell<DIM, TESS> here;
    here.enter(t, e.c);
    int row;
    double from[DIM];
    while (!e.done() && e.behind(sub, left, steps) > 0) e.step(t, A, T, h, nODE, s_row, here, row, from);
    return one && !e.done() && e.step(t, A, T, h, nODE, s_row, here, mi, r);
}

// What an FP64 Path keeps beside its walker to follow calc_T.
template <typename Real>
struct PathExtra {
};
template <>
struct PathExtra<double> {
    bool doubt_step, doubt_cell;  // of the last unit: its decision; the cell its sub-step ended in
    double err, reach;
};

template <int DIM, int TESS, typename Real>
struct Path : PathExtra<Real> {
    using Walker = typename WalkerOf<DIM, TESS, Real>::type;
    static constexpr int NE = DIM * (DIM + 1);
    static constexpr bool kTet = DIM == 3 && TESS == 1, kF64 = sizeof(Real) == 8;
    // A step's roundings in calc_T's arithmetic, relative to the position: 2 D + 1 of u = 1.1e-16 in a closed-form
    // step, 1 in a sub-step and h|A| (3 D + 1) in its velocities.  (Those here are relative to the box, and fewer.)
    static constexpr double kRound = (3 * DIM + 2) * 1.1102230246251565e-16;
    Walker w;
    Real per_m;
    int left, steps, row, kshift, top;
    bool sub;

    __device__ __forceinline__ void to_steps(const JumpCfg &jc, int nC, int n)
    {
        left = n;
        sub = false;
        row = w.c;
        kshift = nC;
        top = jc.nT - 1;
        per_m = Real(1e30);
    }
    __device__ __forceinline__ void to_substeps(const JumpCfg &jc, int nC, int n)
    {
        left = n;
        sub = true;
        row = jc.nT * nC + w.c;
        kshift = 2 * nC;
        top = jc.nS - 1;
    }
    __device__ __forceinline__ void begin(const Tess &t, const JumpCfg &jc, const Real *x, int nT)
    {
        steps = 0;
        if constexpr (kF64) {
            w.place_in(t, x, exact_cell<DIM, TESS>(t, x));
            Real r[DIM];
            this->doubt_step = this->doubt_cell = false;
            this->reach = t.nC0 + t.nC1 + t.nC2;
#pragma unroll
            for (int i = 0; i < DIM; ++i) {
                r[i] = w.p.x(i);
                this->reach += fabs(r[i]);
            }
            this->err = kRound * this->reach;
            w.m = most(w.f.margin(r), Real(0));
        } else {
            w.place(t, x);
        }
        to_steps(jc, t.nC, nT);
    }
    __device__ __forceinline__ bool done() const { return left == 0; }
    // (of a candidate past the domain only that it is outside is known)
    static __device__ __forceinline__ Real lost(Real m) { return kTet ? most(m, Real(-1)) : m; }
    static __device__ __forceinline__ float rate(float a, float b) { return __fdividef(a, b); }
    static __device__ __forceinline__ double rate(double a, double b) { return a / b; }
    // One unit; true when it moved, by the table row mi from r.
    __device__ __forceinline__ bool unit(const Tess &t, const JumpCfg &jc, const JumpTables<Real> &tab, int nODE, int &mi,
                                         Real *r)
    {
        const int nC = t.nC, lg = 31 - __clz(max(min(left, whole(w.m * per_m)), 1));
        const int l = min((lg * jc.mul) >> 5, top), n = 1 << (l * jc.r);
        typename Walker::Cand q;
        mi = l * nC + row;
        const Real *m = tab.map + (size_t)mi * NE;
        const Real len = w.step(t, m, q), need = len * (l > 0 ? tab.kap[mi - kshift] : Real(0));
        bool stays = !(q.m < Real(0)), take = stays && (l == 0 || most(w.m, q.m) >= need);
        if constexpr (kF64) {
            if (take || l == 0) {
                double norm = 0.0, known = l == 0 ? size_of(q.m) : q.m;
#pragma unroll
                for (int k = 0; k < DIM; ++k) {
                    double col = 0.0;
#pragma unroll
                    for (int i = 0; i < DIM; ++i) col += fabs(m[k * DIM + i] + (i == k ? 1.0 : 0.0));
                    norm = fmax(norm, col);
                }
                const double reach = this->reach + len;
                // (within a jump a rounding grows by e^x <= 1 + 2 kappa at most)
                const double steps_err = n * (kRound * reach) * (l > 0 ? 1.0 + 2.0 * tab.kap[mi - kshift] : 1.0);
                const double err = fma(this->err, norm, steps_err);
                if constexpr (kTet) {
                    if (q.m < InnerTet<Real>::kPast) known = size_of(w.margin_past(t, q.x));
                }
                // (3D type I: within the domain's tolerance a margin holds to three times that)
                this->doubt_step = !(known > 2 * err + (kTet ? 4 * InnerTet<Real>::kOver : 0.0));
                if (take || sub) {
                    this->err = err;
                    this->reach = reach;
                }
            }
        }
        if (!stays && l == 0 && w.keeps(t, q)) {
            take = true;
            q.m = 0;
            per_m = Real(1e30);
        }
        if (take || (l == 0 && sub)) {
#pragma unroll
            for (int i = 0; i < DIM; ++i) r[i] = w.p.x(i);
            left -= n;
            if (take) {
                w.take(q, true);
            } else {
                w.leave(t, q);
                if constexpr (kF64) {
                    double known = w.m;
                    if constexpr (kTet) {
                        if (w.m == 0) known = w.margin_past(t, w.p.hi);
                    }
                    this->doubt_cell = !(known > 2 * this->err);
                }
                per_m = Real(1e30);
                row = jc.nT * nC + w.c;
            }
            if (left == 0 && sub) to_steps(jc, nC, --steps);
            return true;
        }
        // dropped: see integrate_jump
        per_m = rate((stays ? Real(0.5) : Real(0.999)) * Real(l == 0 && !sub ? nODE : n),
                     stays ? most(w.m, Real(1e-12)) : w.m - lost(q.m));
        if (l == 0) {
            steps = left;
            to_substeps(jc, nC, nODE);
        }
        return false;
    }
    __device__ __forceinline__ bool doubtful() const
    {
        if constexpr (kF64) return this->doubt_step || this->doubt_cell;
        return false;
    }
    // A unit (true when it moved), its doubts settled.  A, T: the tables' signed A and Trel, x0 the point's start.
    __device__ __forceinline__ bool settled_unit(const Tess &t, const JumpCfg &jc, const JumpTables<Real> &tab,
                                                 const double *A, const double *T, double h, int nT, int nODE,
                                                 const Real *x0, ExactPath<DIM, TESS> &e, int &mi, Real *r)
    {
        const bool sub_before = sub;
        const int left_before = left, steps_before = steps;
        bool moved = unit(t, jc, tab, nODE, mi, r);
        if constexpr (kF64) {
            if (!doubtful()) return moved;
            const bool one = this->doubt_step;
            const bool did = catch_up<DIM, TESS>(t, A, T, h, nT, nODE, jc.nT * t.nC, x0, one ? sub_before : sub,
                                                 one ? left_before : left, one ? steps_before : steps, one, e, mi, r);
            if (one) moved = did;
            this->doubt_step = this->doubt_cell = false;
            w.place_in(t, e.x, e.c);
            Real p[DIM];
#pragma unroll
            for (int i = 0; i < DIM; ++i) p[i] = w.p.x(i);
            w.m = most(w.f.margin(p), Real(0));
            this->err = kRound * this->reach;
            if (e.sub) to_substeps(jc, t.nC, e.left);
            else to_steps(jc, t.nC, e.left);
            steps = e.steps;
            per_m = Real(1e30);
        }
        return moved;
    }
};

// Per-warp queue of points that the first pass left over (entries, shared memory).
constexpr int kQueue = 64;
__host__ __device__ inline size_t queue_bytes(int block) { return (size_t)(block / 32) * kQueue * sizeof(unsigned short); }

// The FP32 twin of integrate_range.  Warps claim 32 points of the range at a
// time and try to carry them through all their closed-form steps at once
// (first pass: lanes in step, loads and stores coalesced; on the prior's
// fields half of the points or more stay in their cell).  Points that may
// leave their cell go to the warp's queue and from there one to a lane, the
// lane advancing its point by one composed step per unit and taking the next
// from the queue when done; another first pass runs whenever the queue does
// not hold enough for the idle lanes.  Every closed-form step of a time step
// is either kept or replaced by nStepsODE sub-steps, so the counts of both
// follow from the number of replaced ones (c_fb).
template <int DIM, int TESS, int SCHEME, class Src, class Snk>
__device__ __forceinline__ void integrate_jump(const Tess &t, int nT, int nODE, const JumpCfg &jc,
                                               const JumpTables<float> &tab, int64_t ws, int n_range, const Src &src,
                                               Snk &snk, unsigned long long &c_fast, unsigned long long &c_fb,
                                               unsigned long long &c_sub, unsigned long long &c_pts, int *claim,
                                               unsigned short *queues, ExactCross *ex)
{
    using Walker = typename WalkerOf<DIM, TESS, float>::type;
    using Cand = typename Walker::Cand;
    constexpr int NE = DIM * (DIM + 1);
    constexpr bool kTet = DIM == 3 && TESS == 1;
    constexpr float kHuge = 1e30f;
    const int lane = threadIdx.x & 31, nC = t.nC;
    const unsigned lt = (1u << lane) - 1u;
    // A lane's phase: closed-form steps of the remaining time steps (`left`
    // of them), or sub-steps of the current one (`left` of them, `steps` time
    // steps to go).  `row`: the phase's level 0 row of w.c in the maps; kappa of
    // level l >= 1 sits at l nC + row - kshift (level 0 reads an entry before
    // it, inside the tables, and ignores it).
    const int s_row = jc.nT * nC;
    Walker w;
    w.c = 0;
    w.m = 0.0f;
    int left = 0, steps = 0, row = 0, kshift = nC, top = 0, idx = 0;
    float per_m = kHuge;  // estimated steps per unit of margin until the exit
    bool sub = false, active = false;
    unsigned n_fb = 0, n_pts = 0;
    auto to_steps = [&](int n) {  // n time steps to go
        left = n;
        sub = SCHEME == SCHEME_SIMPLE;
        row = w.c;
        kshift = nC;
        top = (SCHEME == SCHEME_SIMPLE ? jc.nS : jc.nT) - 1;
        per_m = kHuge;
    };
    auto to_substeps = [&](int n) {
        left = n;
        sub = true;
        row = s_row + w.c;
        kshift = jc.nT > 0 ? 2 * nC : nC;
        top = jc.nS - 1;
    };
    auto start = [&](int k) {
        active = true;
        typename Src::Elem x[DIM];
        idx = k;
        src.load(ws + k, x);
        w.place(t, x);
        steps = 1;
        to_steps(SCHEME == SCHEME_SIMPLE ? nT * nODE : nT);
    };
    auto finish = [&]() {
        typename Src::Elem x[DIM];
        w.position(t, x);
        snk.put(ws + idx, x);
        ++n_pts;
        active = false;
    };
    // level and step count of the largest composed step within n >= 1 steps
    auto level = [&](int n, int l_top, int &count) {
        const int l = min(((31 - __clz(n)) * jc.mul) >> 5, l_top);
        count = 1 << (l * jc.r);
        return l * nC;
    };
    unsigned short *queue = queues + (threadIdx.x >> 5) * kQueue;
    int queued = 0;
    bool more = true;  // the range may hold unclaimed points
    // Idle lanes take points: from the queue, after as many first passes as
    // it takes to fill it (a pass adds at most 32, so kQueue holds).
    auto refill = [&]() {
        const unsigned idle = __ballot_sync(FULL, !active);
        const int want = __popc(idle);
        if (!queues) {
            int b = 0;
            if (lane == 0) b = atomicAdd(claim, want);
            b = __shfl_sync(FULL, b, 0);
            more = b + want < n_range;
            const int k = b + __popc(idle & lt);
            if (!active && k < n_range) start(k);
            __syncwarp();
            return;
        }
        while (more && queued < want) {
            int b = 0;
            if (lane == 0) b = atomicAdd(claim, 32);
            b = __shfl_sync(FULL, b, 0);
            if (b + 32 >= n_range) more = false;
            if (b >= n_range) break;
            const bool have = b + lane < n_range;
            bool left_over = have;
            if (SCHEME != SCHEME_SIMPLE) {
                Walker v;
                typename Src::Elem x[DIM];
                v.c = 0;
                if (have) {
                    src.load(ws + b + lane, x);
                    v.place(t, x);
                }
                int togo = have ? nT : 0;
                bool go = have;
#pragma unroll 1
                for (int u = 0; u < kFirstUnits && __any_sync(FULL, go); ++u) {
                    int n;
                    const int l = level(max(togo, 1), jc.nT - 1, n);
                    Cand q;
                    const float need = v.step(t, tab.map + (l + v.c) * NE, q) * tab.kap[l + v.c - nC];
                    // (from a margin of 0 single steps: as below, and a tetrahedron's may mean past the domain)
                    const bool sure = fmaxf(v.m, q.m) >= need && v.m > 0.0f;
                    go = go && !(q.m < 0.0f) && (l == 0 || sure);
                    v.take(q, go);
                    togo -= go ? n : 0;
                    go = go && togo > 0;
                }
                left_over = have && togo > 0;
                if (have && togo == 0) {
                    v.position(t, x);
                    snk.put(ws + b + lane, x);
                    ++n_pts;
                }
            }
            const unsigned lo = __ballot_sync(FULL, left_over);
            if (left_over) queue[queued + __popc(lo & lt)] = (unsigned short)(b + lane);
            queued += __popc(lo);
            __syncwarp();
        }
        if (!active) {
            const int k = queued - 1 - __popc(idle & lt);
            if (k >= 0) start(queue[k]);
        }
        queued = max(queued - want, 0);
        __syncwarp();
    };
    refill();
    // A lane whose sub-step leaves its cell parks (`park`): the warp moves its
    // parked lanes into their new cells together -- done at once, each such
    // lane would hold up the other 31 (about one lane of a warp leaves its
    // cell per unit).  A parked lane keeps only the sub-step's start and
    // recomputes its end.  EXACT resolves the exits, which takes far longer,
    // once kCrossBatch lanes wait (as integrate_range).
    constexpr int kCrossBatch = CPAB_EXACT_CROSS_BATCH, kCrossWait = CPAB_EXACT_CROSS_WAIT;
    bool park = false;
    int park_votes = 0;
    while (__any_sync(FULL, active)) {
        // units without branches: lanes that wait run along without effect
#pragma unroll 1
        for (int h = 0; h < kRounds; ++h) {
            bool go = active && !park && left > 0, out = false, past = false;
#pragma unroll
            for (int u = 0; u < kUnits; ++u) {
                int n;
                const int l = level(max(min(left, whole(w.m * per_m)), 1), top, n);
                Cand q;
                const float need = w.step(t, tab.map + (l + row) * NE, q) * tab.kap[l + row - kshift];
                const bool stays = !(q.m < 0.0f);  // NaN stays
                const bool take = go && stays && (l == 0 || fmaxf(w.m, q.m) >= need);
                // Dropped: the exit is estimated where the margin is used up at
                // the rate it was lost (a candidate inside, but not certain:
                // at half its steps).  The estimate stays below n steps, so the
                // next jump from here is a shorter one.
                if (go && !take) {
                    per_m = __fdividef((stays ? 0.5f : 0.999f) * (float)(l == 0 && !sub ? nODE : n),
                                       stays ? fmaxf(w.m, 1e-12f) : w.m - (kTet ? fmaxf(q.m, -1.0f) : q.m));
                    if (kTet) past = q.m < InnerTet<float>::kPast;
                }
                out = out || (go && !take && l == 0);
                w.take(q, take);
                left -= take ? n : 0;
                go = go && !out && left > 0;
            }
            if (kTet && out && past) {
                // past the domain: the lookup says whether the step left the cell
                Cand q;
                w.step(t, tab.map + row * NE, q);
                if (w.keeps(t, q)) {
                    q.m = 0.0f;
                    w.take(q, true);
                    --left;
                    out = false;
                    per_m = kHuge;
                }
            }
            if (SCHEME == SCHEME_SIMPLE) {
                park = park || out;
            } else {
                park = park || (out && sub);
                if (out && !sub) {
                    // the closed-form step leaves the cell: redo it with nStepsODE sub-steps
                    steps = left;
                    to_substeps(nODE);
                    ++n_fb;
                } else if (left == 0 && sub && !park) {
                    to_steps(--steps);
                }
            }
        }
        const unsigned pm = __ballot_sync(FULL, park);
        bool resolve = pm != 0;
        if (SCHEME == SCHEME_EXACT && pm) {
            const unsigned am = __ballot_sync(FULL, active && left > 0);
            resolve = __popc(pm) >= kCrossBatch || pm == am || ++park_votes > kCrossWait;
            if (resolve) park_votes = 0;
        }
        if (resolve && park) {
            // the parked sub-step's end, recomputed with the same arithmetic
            Cand q;
            w.step(t, tab.map + row * NE, q);
            if (SCHEME == SCHEME_EXACT) {
                double from[DIM], to[DIM];
                w.position(t, from);
                w.where(t, q, to);
                const int c = exact_substep_cross<DIM, TESS, float>(t, *ex, w.c, from, to);
                w.place_in(t, to, c);
            } else {
                w.leave(t, q);
            }
            park = false;
            // of the new cell's exit nothing is known
            if (SCHEME == SCHEME_SIMPLE) {
                to_steps(left - 1);
            } else if (left > 1) {
                to_substeps(left - 1);
                per_m = kHuge;
            } else {
                to_steps(--steps);
            }
        }
        if (active && !park && left == 0) finish();
        if (__any_sync(FULL, !active) && (more || queued > 0)) refill();
    }
    c_pts += n_pts;
    if (SCHEME == SCHEME_SIMPLE) {
        c_sub += (unsigned long long)n_pts * nT * nODE;
    } else {
        c_fb += n_fb;
        c_sub += (unsigned long long)n_fb * nODE;
        c_fast += (unsigned long long)n_pts * nT - n_fb;
    }
}

}  // namespace cpab
