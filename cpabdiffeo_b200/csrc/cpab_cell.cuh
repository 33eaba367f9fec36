// cpab_cell.cuh -- cell lookup and affine evaluation shared by every kernel.
//
// Two arithmetic families:
//
//  * exact (double): reproduces the reference's double-precision cell lookup
//    bit for bit (cpab/gpu/calc_1Dto1D.cu:56-259, calc_2Dto2D.cu:38-153,
//    calc_3Dto3D.cu:43-137) and its left-to-right affine sums with every
//    product and sum rounded on its own (no fused multiply-add).  The
//    reference evaluates  (p - fmod(p, inc)) / inc  and rounds it; this file
//    computes the same integer k and the same remainder r = fmod(p, inc)
//    without fmod or a division:
//        k = floor(p * (1/inc))            (estimate, off by at most one)
//        r = fma(-k, inc, p)               (exact: p - k*inc is representable
//                                           whenever k is the true quotient)
//        fix k by one if r < 0 or r >= inc, recompute r.
//    Because fmod is exact in IEEE arithmetic, r equals fmod(p, inc) bit for
//    bit, and round((p - r)/inc) equals k for every k < 2^50.  Quotients
//    that feed a comparison (xmod/inc) still use a correctly rounded
//    division, or an exact product when inc is a power of two.
//
//  * fast (float): the same tessellation geometry in single precision with
//    fused multiply-adds, for the FP32 mode, whose results are held to a
//    tolerance against the double-precision oracle.
//
// Everything is __host__ __device__ so the exact family can be checked
// against the oracle on the CPU (tests/test_cell_lookup_host.py).
#pragma once

#include <stdint.h>
#include <math.h>

#ifdef __CUDACC__
#define CPAB_HD __host__ __device__ __forceinline__
#else
#define CPAB_HD inline
#endif

// Non-contracted double arithmetic.  nvcc never fuses the __d*_rn
// intrinsics; the host build uses -ffp-contract=off.
#if defined(__CUDA_ARCH__)
#define XMUL(a, b) __dmul_rn((a), (b))
#define XADD(a, b) __dadd_rn((a), (b))
#define XSUB(a, b) __dsub_rn((a), (b))
#define XDIV(a, b) __ddiv_rn((a), (b))
#define XFMA(a, b, c) __fma_rn((a), (b), (c))
#else
#define XMUL(a, b) ((a) * (b))
#define XADD(a, b) ((a) + (b))
#define XSUB(a, b) ((a) - (b))
#define XDIV(a, b) ((a) / (b))
#define XFMA(a, b, c) fma((a), (b), (c))
#endif

namespace cpab {

// Geometry of one tessellation, precomputed on the host once per space.
// All derived doubles are formed exactly as the reference forms them
// (e.g. hi = (double)nC * inc - 1e-10, calc_2Dto2D.cu:55).
struct Tess {
    int dim;           // 1, 2, 3
    int tess;          // 1 = type I (simplices), 2 = type II (boxes)
    int nC0, nC1, nC2; // boxes per axis
    int nC;            // number of cells
    double inc[3];     // box size per axis (reference "incs")
    double inv_inc[3]; // 1/inc, used only as a quotient estimate
    double span[3];    // (double)nCk * inc_k
    double hi[3];      // clamp for type I: (double)nCk*inc_k - 1e-10 (axis 2 uses inc_x)
    int pow2[3];       // inc_k is a power of two: xmod/inc == xmod*(1/inc) exactly
    float finc[3], finv_inc[3], fspan[3], fhi[3];
    float finc_lo[3], finv_inc_lo[3];  // inc - finc, 1/inc - finv_inc
    float finv_n[3];                   // 1 / nCk
};

// Geometry of a tessellation from box counts and box sizes, derived
// exactly as the reference derives its constants.  Returns false if the
// arguments are invalid.
inline bool make_tess(int dim, int tess, const int *nCs, const double *incs, Tess &t)
{
    t = Tess();
    if (dim < 1 || dim > 3 || (tess != 1 && tess != 2)) return false;
    t.dim = dim;
    t.tess = tess;
    int n[3] = {1, 1, 1};
    for (int k = 0; k < dim; ++k) {
        if (nCs[k] < 1 || !(incs[k] > 0) || !(incs[k] < INFINITY)) return false;
        n[k] = nCs[k];
    }
    t.nC0 = n[0];
    t.nC1 = dim > 1 ? n[1] : 0;
    t.nC2 = dim > 2 ? n[2] : 0;
    long long nC = (long long)n[0] * n[1] * n[2];
    if (tess == 1) nC *= (dim == 2 ? 4 : 5);
    if (nC > (1 << 20)) return false;
    t.nC = (int)nC;
    for (int k = 0; k < 3; ++k) {
        double inc = k < dim ? incs[k] : 1.0;
        t.inc[k] = inc;
        t.inv_inc[k] = 1.0 / inc;
        int e = 0;
        t.pow2[k] = (frexp(inc, &e) == 0.5) ? 1 : 0;
        t.span[k] = (double)n[k] * inc;
        t.hi[k] = (double)n[k] * inc - 0.0000000001;
    }
    // calc_3Dto3D.cu:59 clamps z with nC2*inc_x
    if (dim == 3 && tess == 1) t.hi[2] = (double)n[2] * t.inc[0] - 0.0000000001;
    for (int k = 0; k < 3; ++k) {
        t.finc[k] = (float)t.inc[k];
        t.finv_inc[k] = (float)(1.0 / t.inc[k]);
        t.finc_lo[k] = (float)(t.inc[k] - (double)t.finc[k]);
        t.finv_inc_lo[k] = (float)(1.0 / t.inc[k] - (double)t.finv_inc[k]);
        t.finv_n[k] = 1.0f / (float)n[k];
        t.fspan[k] = (float)t.span[k];
        double top = (dim == 3 && tess == 1 && k == 2) ? (double)n[2] * t.inc[0] : t.span[k];
        // float clamp strictly below the span so floor() stays in the last box,
        // also where the product with 1/inc rounds up
        t.fhi[k] = nextafterf((float)top, 0.0f);
        if (top == t.span[k])
            while (t.fhi[k] > 0.0f && t.fhi[k] * t.finv_inc[k] >= (float)n[k]) t.fhi[k] = nextafterf(t.fhi[k], 0.0f);
    }
    return true;
}

// ---------------------------------------------------------------- exact

// k = trunc-toward-floor(p/inc) and r = fmod(p, inc) for finite p >= 0.
CPAB_HD void exact_floor_rem(double p, double inc, double inv, double &k, double &r)
{
    k = floor(p * inv);
    r = XFMA(-k, inc, p);
    if (r < 0.0) {
        k -= 1.0;
        r = XFMA(-k, inc, p);
    } else if (r >= inc) {
        k += 1.0;
        r = XFMA(-k, inc, p);
    }
}

// round(min(n-1, max(0, (p - fmod(p,inc))/inc)))  (type II / 1D axis).
// NaN and +-inf give 0 as in the reference (fmod(inf) is NaN, max(0,NaN)=0).
CPAB_HD int exact_box_coord(double p, int n, double inc, double inv)
{
    if (!(p >= 0.0) || !(p < INFINITY)) return 0;
    double k, r;
    exact_floor_rem(p, inc, inv, k, r);
    double lim = (double)(n - 1);
    return (int)(k < lim ? k : lim);
}

CPAB_HD double exact_frac(double xmod, double inc, double inv, int pow2)
{
    return pow2 ? XMUL(xmod, inv) : XDIV(xmod, inc);
}

// 2D type I (calc_2Dto2D.cu:53-148): 4 triangles per box, 0 top, 1 right,
// 2 bottom, 3 left; separate rules for points outside the domain.
CPAB_HD int exact_cell_2d_tri(const Tess &t, const double *p)
{
    const double ix = t.inc[0], iy = t.inc[1];
    double p0 = fmin(t.hi[0], fmax(0.0, p[0]));
    double p1 = fmin(t.hi[1], fmax(0.0, p[1]));
    double kx, xmod, ky, ymod;
    exact_floor_rem(p0, ix, t.inv_inc[0], kx, xmod);
    exact_floor_rem(p1, iy, t.inv_inc[1], ky, ymod);
    const double limx = (double)(t.nC0 - 1), limy = (double)(t.nC1 - 1);
    int c = ((int)(kx < limx ? kx : limx) + (int)(ky < limy ? ky : limy) * t.nC0) * 4;
    if (p[0] <= 0) {
        if (p[1] <= 0 && XDIV(p[1], iy) < XDIV(p[0], ix)) return c;
        if (p[1] >= t.span[1] && XSUB(XDIV(p[1], iy), (double)t.nC1) > XDIV(-p[0], ix)) return c + 2;
        return c + 3;
    }
    if (p[0] >= t.span[0]) {
        if (p[1] <= 0 && XDIV(-p[1], iy) > XSUB(XDIV(p[0], ix), (double)t.nC0)) return c;
        if (p[1] >= t.span[1] &&
            XSUB(XDIV(p[1], iy), (double)t.nC1) > XSUB(XDIV(p[0], ix), (double)t.nC0)) return c + 2;
        return c + 1;
    }
    if (p[1] <= 0) return c;
    if (p[1] >= t.span[1]) return c + 2;
    double x = exact_frac(xmod, ix, t.inv_inc[0], t.pow2[0]);
    double y = exact_frac(ymod, iy, t.inv_inc[1], t.pow2[1]);
    double omx = XSUB(1.0, x);
    if (x < y) return c + ((omx < y) ? 2 : 3);
    return c + ((omx < y) ? 1 : 0);
}

// 3D type I (calc_3Dto3D.cu:55-133): 5 tetrahedra per box with a
// checkerboard flip; the z clamp uses nC2*inc_x (hi[2] carries it).
CPAB_HD int exact_cell_3d_tet(const Tess &t, const double *p)
{
    double p0 = fmin(t.hi[0], fmax(0.0, p[0]));
    double p1 = fmin(t.hi[1], fmax(0.0, p[1]));
    double p2 = fmin(t.hi[2], fmax(0.0, p[2]));
    double ki, xmod, kj, ymod, kk, zmod;
    exact_floor_rem(p0, t.inc[0], t.inv_inc[0], ki, xmod);
    exact_floor_rem(p1, t.inc[1], t.inv_inc[1], kj, ymod);
    exact_floor_rem(p2, t.inc[2], t.inv_inc[2], kk, zmod);
    const double li = (double)(t.nC0 - 1), lj = (double)(t.nC1 - 1), lk = (double)(t.nC2 - 1);
    int i = (int)(ki < li ? ki : li), j = (int)(kj < lj ? kj : lj), k = (int)(kk < lk ? kk : lk);
    int c = (i + j * t.nC0 + k * t.nC1 * t.nC0) * 5;
    double x = exact_frac(xmod, t.inc[0], t.inv_inc[0], t.pow2[0]);
    double y = exact_frac(ymod, t.inc[1], t.inv_inc[1], t.pow2[1]);
    double z = exact_frac(zmod, t.inc[2], t.inv_inc[2], t.pow2[2]);
    bool flip = ((i ^ j ^ k) & 1) != 0;  // k even: i,j of different parity; k odd: same parity
    if (flip) {
        double tmp = x;
        x = y;
        y = XSUB(1.0, tmp);
    }
    if (XADD(XSUB(-x, y), z) >= 0) return c + 1;
    if (XSUB(XADD(XADD(x, y), z), 2.0) >= 0) return c + 2;
    if (XSUB(XADD(-x, y), z) >= 0) return c + 3;
    if (XSUB(XSUB(x, y), z) >= 0) return c + 4;
    return c;
}

template <int DIM, int TESS>
CPAB_HD int exact_cell(const Tess &t, const double *p)
{
    if (DIM == 1) return exact_box_coord(p[0], t.nC0, t.inc[0], t.inv_inc[0]);
    if (DIM == 2) {
        if (TESS == 2)
            return exact_box_coord(p[0], t.nC0, t.inc[0], t.inv_inc[0]) +
                   exact_box_coord(p[1], t.nC1, t.inc[1], t.inv_inc[1]) * t.nC0;
        return exact_cell_2d_tri(t, p);
    }
    if (TESS == 2)
        return exact_box_coord(p[0], t.nC0, t.inc[0], t.inv_inc[0]) +
               exact_box_coord(p[1], t.nC1, t.inc[1], t.inv_inc[1]) * t.nC0 +
               exact_box_coord(p[2], t.nC2, t.inc[2], t.inv_inc[2]) * t.nC1 * t.nC0;
    return exact_cell_3d_tet(t, p);
}

// x = A [b; 1], sums left to right, every operation rounded on its own
// (A_times_b_affine, calc_1Dto1D.cu:18-34).
template <int DIM>
CPAB_HD void exact_affine(double *x, const double *A, const double *b)
{
    if (DIM == 1) {
        x[0] = XADD(XMUL(A[0], b[0]), A[1]);
    } else if (DIM == 2) {
        x[0] = XADD(XADD(XMUL(A[0], b[0]), XMUL(A[1], b[1])), A[2]);
        x[1] = XADD(XADD(XMUL(A[3], b[0]), XMUL(A[4], b[1])), A[5]);
    } else {
        x[0] = XADD(XADD(XADD(XMUL(A[0], b[0]), XMUL(A[1], b[1])), XMUL(A[2], b[2])), A[3]);
        x[1] = XADD(XADD(XADD(XMUL(A[4], b[0]), XMUL(A[5], b[1])), XMUL(A[6], b[2])), A[7]);
        x[2] = XADD(XADD(XADD(XMUL(A[8], b[0]), XMUL(A[9], b[1])), XMUL(A[10], b[2])), A[11]);
    }
}

// One explicit-midpoint sub-step of solveODE (calc_2Dto2D.cu:177-196):
// pMid = p + h*v/2 ; p += vMid*h, with the cell of p for both evaluations.
template <int DIM>
CPAB_HD void exact_midpoint(double *p, const double *A, double h)
{
    double v[DIM], pm[DIM];
    exact_affine<DIM>(v, A, p);
#pragma unroll
    for (int i = 0; i < DIM; ++i) pm[i] = XADD(p[i], XMUL(XMUL(h, v[i]), 0.5));  // / 2: the same double
    exact_affine<DIM>(v, A, pm);
#pragma unroll
    for (int i = 0; i < DIM; ++i) p[i] = XADD(p[i], XMUL(v[i], h));
}

// ---------------------------------------------------------------- fast (float)

CPAB_HD int fast_box_coord(float p, int n, float inv)
{
#ifdef __CUDA_ARCH__
    // one float->int conversion rounding down; NaN converts to 0, +-inf saturate
    int k = __float2int_rd(p * inv);
    return min(max(k, 0), n - 1);
#else
    float k = floorf(p * inv);
    k = fminf(fmaxf(k, 0.0f), (float)(n - 1));  // NaN -> 0
    return (int)k;
#endif
}

CPAB_HD int fast_cell_2d_tri(const Tess &t, const float *p)
{
    if (p[0] > 0.0f && p[0] < t.fhi[0] && p[1] > 0.0f && p[1] < t.fhi[1]) {
        // strictly inside the domain (the common case): the clamps below are
        // no-ops and none of the boundary rules applies -- same result
#ifdef __CUDA_ARCH__
        // both axes as one pair (FMUL2 / FADD2, each lane rounded as its scalar twin)
        const float2 uw = __fmul2_rn(make_float2(p[0], p[1]), make_float2(t.finv_inc[0], t.finv_inc[1]));
        const float kx = floorf(uw.x), ky = floorf(uw.y);
        const float2 xy = __fadd2_rn(uw, make_float2(-kx, -ky));
        const float x = xy.x, y = xy.y;
#else
        const float u = p[0] * t.finv_inc[0], w = p[1] * t.finv_inc[1];
        const float kx = floorf(u), ky = floorf(w);
        const float x = u - kx, y = w - ky;
#endif
        const int c = ((int)fminf(kx, (float)(t.nC0 - 1)) + (int)fminf(ky, (float)(t.nC1 - 1)) * t.nC0) * 4;
        const float omx = 1.0f - x;
        return c + ((x < y) ? ((omx < y) ? 2 : 3) : ((omx < y) ? 1 : 0));
    }
    float p0 = fminf(t.fhi[0], fmaxf(0.0f, p[0]));
    float p1 = fminf(t.fhi[1], fmaxf(0.0f, p[1]));
    float u = p0 * t.finv_inc[0], w = p1 * t.finv_inc[1];
    float kx = floorf(u), ky = floorf(w);
    float x = u - kx, y = w - ky;
    int c = ((int)fminf(kx, (float)(t.nC0 - 1)) + (int)fminf(ky, (float)(t.nC1 - 1)) * t.nC0) * 4;
    if (p[0] <= 0) {
        float a = p[0] * t.finv_inc[0], b = p[1] * t.finv_inc[1];
        if (p[1] <= 0 && b < a) return c;
        if (p[1] >= t.fspan[1] && b - (float)t.nC1 > -a) return c + 2;
        return c + 3;
    }
    if (p[0] >= t.fspan[0]) {
        float a = p[0] * t.finv_inc[0], b = p[1] * t.finv_inc[1];
        if (p[1] <= 0 && -b > a - (float)t.nC0) return c;
        if (p[1] >= t.fspan[1] && b - (float)t.nC1 > a - (float)t.nC0) return c + 2;
        return c + 1;
    }
    if (p[1] <= 0) return c;
    if (p[1] >= t.fspan[1]) return c + 2;
    float omx = 1.0f - x;
    if (x < y) return c + ((omx < y) ? 2 : 3);
    return c + ((omx < y) ? 1 : 0);
}

CPAB_HD int fast_cell_3d_tet(const Tess &t, const float *p)
{
    float u0 = fminf(t.fhi[0], fmaxf(0.0f, p[0])) * t.finv_inc[0];
    float u1 = fminf(t.fhi[1], fmaxf(0.0f, p[1])) * t.finv_inc[1];
    float u2 = fminf(t.fhi[2], fmaxf(0.0f, p[2])) * t.finv_inc[2];
    float fi = floorf(u0), fj = floorf(u1), fk = floorf(u2);
    float x = u0 - fi, y = u1 - fj, z = u2 - fk;
    int i = (int)fminf(fi, (float)(t.nC0 - 1));
    int j = (int)fminf(fj, (float)(t.nC1 - 1));
    int k = (int)fminf(fk, (float)(t.nC2 - 1));
    int c = (i + j * t.nC0 + k * t.nC1 * t.nC0) * 5;
    if ((i ^ j ^ k) & 1) {
        float tmp = x;
        x = y;
        y = 1.0f - tmp;
    }
    if (-x - y + z >= 0) return c + 1;
    if (x + y + z - 2.0f >= 0) return c + 2;
    if (-x + y - z >= 0) return c + 3;
    if (x - y - z >= 0) return c + 4;
    return c;
}

template <int DIM, int TESS>
CPAB_HD int fast_cell(const Tess &t, const float *p)
{
    if (DIM == 1) return fast_box_coord(p[0], t.nC0, t.finv_inc[0]);
    if (DIM == 2) {
        if (TESS == 2)
            return fast_box_coord(p[0], t.nC0, t.finv_inc[0]) +
                   fast_box_coord(p[1], t.nC1, t.finv_inc[1]) * t.nC0;
        return fast_cell_2d_tri(t, p);
    }
    if (TESS == 2)
        return fast_box_coord(p[0], t.nC0, t.finv_inc[0]) +
               fast_box_coord(p[1], t.nC1, t.finv_inc[1]) * t.nC0 +
               fast_box_coord(p[2], t.nC2, t.finv_inc[2]) * t.nC1 * t.nC0;
    return fast_cell_3d_tet(t, p);
}

// fast_cell_3d_tet with m: a lower bound of the distances from the point to the
// facets its cell shares with another cell, in box units (coordinates divided
// by the box sizes; a cut plane's distance is its functional -x - y + z, ...
// with coefficients +-1).  Facets on the domain boundary do not count: the
// cell continues outside.  Points outside take the margins of the nearest
// point inside.  m exceeds a distance only by float rounding; for NaN
// coordinates it means nothing.
CPAB_HD int fast_cell_3d_tet_m(const Tess &t, const float *p, float &m)
{
    const int n[3] = {t.nC0, t.nC1, t.nC2};
    int kb[3];
    float f[3], face = 2.0f;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int i = 0; i < 3; ++i) {
        const float u = fminf(t.fhi[i], fmaxf(0.0f, p[i])) * t.finv_inc[i], fl = floorf(u);
        kb[i] = (int)fminf(fl, (float)(n[i] - 1));
        f[i] = u - fl;
        // the nearest of the box's faces inside the domain, a lower bound of a corner tetrahedron's three
        if (kb[i] > 0) face = fminf(face, f[i]);
        if (kb[i] < n[i] - 1) face = fminf(face, 1.0f - f[i]);
    }
    float x = f[0], y = f[1];
    const float z = f[2];
    if ((kb[0] ^ kb[1] ^ kb[2]) & 1) {
        const float tmp = x;
        x = y;
        y = 1.0f - tmp;
    }
    // the four cut planes, in fast_cell_3d_tet's order and arithmetic
    const float e1 = -x - y + z, e2 = x + y + z - 2.0f, e3 = -x + y - z, e4 = x - y - z;
    const int tet = e1 >= 0 ? 1 : e2 >= 0 ? 2 : e3 >= 0 ? 3 : e4 >= 0 ? 4 : 0;
    m = fminf(fminf(fabsf(e1), fabsf(e2)), fminf(fabsf(e3), fabsf(e4)));
    if (tet) m = fminf(m, face);
    return (kb[0] + kb[1] * t.nC0 + kb[2] * t.nC1 * t.nC0) * 5 + tet;
}

// The box indices of cell c.  Quotients of integers below 2^20 by a float
// product: the quotient's error stays below 2^-23 2^20 / n = 1/(8 n), its
// distance from the next integer is at least 1/(2 n).
template <int DIM, int TESS>
CPAB_HD void cell_box(const Tess &t, int c, int *kb)
{
    const int n[3] = {t.nC0, t.nC1, t.nC2};
    int b = TESS == 1 ? (DIM == 2 ? c >> 2 : c / 5) : c;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int i = 0; i + 1 < DIM; ++i) {
        const int q = (int)(((float)b + 0.5f) * t.finv_n[i]);
        kb[i] = b - q * n[i];
        b = q;
    }
    kb[DIM - 1] = b;
}

// ---------------------------------------------------------------- facets of a cell
//
// Positions relative to a box: box units from its centre.  margin(x) is the
// smallest of the functionals that bound the cell (coefficients 0, +-1 in the
// coordinates): >= 0 in the cell, < 0 outside, up to rounding.  Facets on the
// domain boundary do not count, the cells continue outside as in the
// reference's lookup.  Either precision.

constexpr float kFar = 1e30f;  // distance to a facet on the domain boundary

CPAB_HD float flip(float v, bool neg) { return neg ? -v : v; }
CPAB_HD double flip(double v, bool neg) { return neg ? -v : v; }
CPAB_HD float least(float a, float b) { return fminf(a, b); }
CPAB_HD double least(double a, double b) { return fmin(a, b); }
CPAB_HD float most(float a, float b) { return fmaxf(a, b); }
CPAB_HD double most(double a, double b) { return fmax(a, b); }
CPAB_HD float size_of(float a) { return fabsf(a); }
CPAB_HD double size_of(double a) { return fabs(a); }
// towards zero, saturating; NaN -> 0 (a conversion on the device)
template <typename Real>
CPAB_HD int whole(Real v)
{
#ifdef __CUDA_ARCH__
    return (int)v;
#else
    return v >= Real(2147483647) ? 2147483647 : v > Real(-2147483648.0) ? (int)v : v == v ? -2147483647 - 1 : 0;
#endif
}
CPAB_HD float fused(float a, float b, float c) { return fmaf(a, b, c); }
CPAB_HD double fused(double a, double b, double c) { return fma(a, b, c); }

// Box cells (1D and type II): the box's faces.
template <int DIM, int TESS>
struct Facets {
    float flo[DIM], fhi[DIM];  // 1/2, or kFar where the domain ends

    CPAB_HD void enter(const Tess &t, int, const int *kb)
    {
        const int n[3] = {t.nC0, t.nC1, t.nC2};
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int i = 0; i < DIM; ++i) {
            flo[i] = kb[i] > 0 ? 0.5f : kFar;
            fhi[i] = kb[i] < n[i] - 1 ? 0.5f : kFar;
        }
    }
    template <typename Real>
    CPAB_HD Real margin(const Real *x) const
    {
        Real v = least(flo[0] + x[0], fhi[0] - x[0]);
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int i = 1; i < DIM; ++i) v = least(v, least(flo[i] + x[i], fhi[i] - x[i]));
        return v;
    }
};

// 2D type I: four triangles per box between its diagonals, 0 at low y, then
// counterclockwise.  With v the box coordinate towards a triangle's side and u
// the one along it, the triangle is |u| <= v <= 1/2.  Outside the domain the
// reference's rules (calc_2Dto2D.cu:53-148) continue it: beyond its side over
// the side's width (|u| <= 1/2), and beyond a corner of the domain up to the
// box's diagonal continued (|u| <= v).
template <>
struct Facets<2, 1> {
    bool along_x;    // v is the y coordinate
    bool neg;        // v points down it
    float side;      // 1/2, or kFar where the side ends the domain
    float ulo, uhi;  // beyond such a side: 1/2 at the box's faces in u inside the domain, else kFar

    CPAB_HD void enter(const Tess &t, int c, const int *kb)
    {
        const int tri = c & 3;
        const bool up = tri >= 2, right = tri == 1 || tri == 2;
        along_x = up == right;
        neg = !right;
        const int k = along_x ? kb[1] : kb[0], n = along_x ? t.nC1 : t.nC0;
        const int ku = along_x ? kb[0] : kb[1], nu = along_x ? t.nC0 : t.nC1;
        const bool end = k == (right ? n - 1 : 0);
        side = end ? kFar : 0.5f;
        ulo = end && ku > 0 ? 0.5f : kFar;
        uhi = end && ku < nu - 1 ? 0.5f : kFar;
    }
    template <typename Real>
    CPAB_HD Real margin(const Real *x) const
    {
        const Real v = flip(along_x ? x[1] : x[0], neg), u = along_x ? x[0] : x[1];
        return least(least(v - size_of(u), side - v), least(ulo + u, uhi - u));
    }
};

// 3D type I: five tetrahedra per box, four at corners and the centre one.  In
// box coordinates R a corner tetrahedron belongs to a corner sigma (signs of
// product + in even boxes, - in odd ones): with y_a = sigma_a R_a it is
// y0 + y1 + y2 >= 1/2 inside the box's three faces y_a <= 1/2 there; the centre
// is where no corner's sum reaches 1/2.  Coordinates beyond the domain count
// as on its boundary (the reference clamps them, calc_3Dto3D.cu:55-60), hence
// the clamped y in the sums: there the margin does not tell a cell from its
// neighbours for certain (past a corner of the domain every coordinate is
// clamped, and the sums of a corner and of the centre are both 0 over all of
// it).  The reference clamps z with the x box size.  Where that is the smaller one,
// the clamp lies inside the domain and takes the place of its top here; where
// it is the larger one, these facets do not describe the cells past the top.
template <>
struct Facets<3, 1> {
    bool neg[3];    // signs of sigma
    float face[3];  // 1/2, or kFar where the face ends the domain (and for the centre)
    float low[3];   // -1/2 where the opposite face ends the domain, else -kFar
    float cap[3];   // 1/2 where the face ends the domain (z: where it is clamped), else kFar
    bool centre;

    CPAB_HD void enter(const Tess &t, int c, const int *kb)
    {
        const int n[3] = {t.nC0, t.nC1, t.nC2};
        const int tet = c - c / 5 * 5;
        const bool odd = ((kb[0] ^ kb[1] ^ kb[2]) & 1) != 0;
        centre = tet == 0;
        // signs in exact_cell_3d_tet's turned coordinates (odd boxes: (x, y) -> (y, -x))
        const bool n0 = tet == 1 || tet == 3, n1 = tet == 1 || tet == 4;
        neg[0] = odd ? !n1 : n0;
        neg[1] = odd ? n0 : n1;
        neg[2] = tet == 3 || tet == 4;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int i = 0; i < 3; ++i) {
            const float lo = kb[i] == 0 ? 0.5f : kFar;
            float hi = kb[i] == n[i] - 1 ? 0.5f : kFar;
            if (i == 2 && t.inc[0] < t.inc[2]) {
                const float z = (float)(t.hi[2] * t.inv_inc[2] - ((double)kb[2] + 0.5));
                if (z < 0.5f) hi = z;
            }
            cap[i] = neg[i] ? lo : hi;
            low[i] = neg[i] ? -hi : -lo;
            face[i] = centre || cap[i] < kFar ? kFar : 0.5f;
        }
    }
    template <typename Real>
    CPAB_HD Real margin(const Real *x) const
    {
        Real y[3], sum = Real(-0.5), far = kFar;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int i = 0; i < 3; ++i) {
            const Real f = flip(x[i], neg[i]);
            far = least(far, face[i] - f);
            y[i] = most(least(f, Real(cap[i])), Real(low[i]));
            sum += y[i];
        }
        // the four corners' sums: sigma with an even number of signs flipped
        const Real a = y[0] + y[1], d = y[0] - y[1];
        const Real all = most(size_of(a) + y[2], size_of(d) - y[2]);
        return centre ? Real(0.5) - all : least(sum, far);
    }
};

// The same cells up to the domain's ends only: margin is that of Facets inside
// the domain, or within kOver (box units) of it, and below kPast beyond, where
// the clamped coordinates would say nothing certain.  One multiply-add per end
// takes the place of Facets' clamps: kSteep (end + kOver - y), the steepness
// keeping it out of the minimum inside.
template <typename Real>
struct InnerTet {
    static constexpr Real kOver = sizeof(Real) == 4 ? Real(1e-6) : Real(1e-12);
    static constexpr Real kSteep = sizeof(Real) == 4 ? Real(1e36f) : Real(1e200);
    static constexpr Real kPast = Real(-1e20);
    bool neg[3], centre;
    Real steep[3], hi[3], lo[3];  // towards sigma: face (steep 1) or end (kSteep); away from it: end

    CPAB_HD void enter(const Tess &t, int c, const int *kb)
    {
        Facets<3, 1> f;
        f.enter(t, c, kb);
        centre = f.centre;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int i = 0; i < 3; ++i) {
            neg[i] = f.neg[i];
            const bool face = f.face[i] < kFar;
            steep[i] = face ? Real(1) : kSteep;
            hi[i] = face ? Real(0.5) : f.cap[i] < kFar ? kSteep * (Real(f.cap[i]) + kOver) : Real(INFINITY);
            lo[i] = f.low[i] > -kFar ? kSteep * (kOver - Real(f.low[i])) : Real(INFINITY);
        }
    }
    CPAB_HD Real margin(const Real *x) const
    {
        Real y[3], sum = Real(-0.5), far = kFar;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int i = 0; i < 3; ++i) {
            y[i] = flip(x[i], neg[i]);
            far = least(far, least(fused(-steep[i], y[i], hi[i]), fused(kSteep, y[i], lo[i])));
            sum += y[i];
        }
        const Real a = y[0] + y[1], d = y[0] - y[1];
        const Real all = most(size_of(a) + y[2], size_of(d) - y[2]);
        return least(centre ? Real(0.5) - all : sum, far);
    }
};

}  // namespace cpab
