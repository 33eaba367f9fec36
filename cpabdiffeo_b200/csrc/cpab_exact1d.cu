// cpab_exact1d.cu -- closed-form 1D integration across cell boundaries.
//
// Restates cpab/cpa1d/calcs/ClosedFormInt.py (calc_phi :64-165,
// find_crossing_time :193-256, calc_affine_phi :171-192) for a batch of
// instances on the unit interval with nC equal cells and zero-velocity
// boundary.  Inside cell c the velocity is v(x) = a x + b, so
//     x(t) = e^{a t} x + b (e^{a t} - 1) / a        (x + t b if a == 0)
// and the time to reach the cell's exit endpoint xe is
//     t = log((xe + b/a) / (x + b/a)) / a           ((xe - x)/b if a ~ 0).
// A point walks from cell to cell, consuming the remaining time, until it
// stops inside a cell or the velocity cannot carry it over the next
// endpoint (sign change / zero velocity), with the reference's 1e-16 and
// 1e-12 nudges at endpoints and its np.allclose(., 0) tests (|.| <= 1e-8).
//
// FP64 walks, with double hitting times throughout.  FP32 (float points) takes
// intervals of the flow map where an instance has the points for it: their ends
// and anchors come from double hitting times, and a point is one formula in
// float from its anchor on (k_exact1d_intervals); the error stays that of the
// walk, 2.2e-8 of the norm.  Other points and instances walk in double; in
// spaces of too many cells for the intervals' tables FP32 walks with the first
// exit time as a difference of logarithms and the last exponential in float
// (cf_crossing_f32, cf_phi_f32).
#include <math_constants.h>

#include "cpab_device.cuh"
#include "cpab_launch.h"

namespace cpab {

struct Exact1D {
    const double *A;  // [nC, 2] signed (a, b) of the current instance, shared memory
    const double *ba; // [nC] b / a
    const double *ia; // [nC] 1.0 / a
    const double *lx; // [2 nC] log|xn + b/a| of the cell's exit points (xn: right, then left), FP32 mode
    int nC;
    double step;      // 1/nC: vertices x_k = k*step, x_nC = 1 (np.linspace(0,1,nC+1))
};

__device__ __forceinline__ double vert(const Exact1D &e, int k) { return k == e.nC ? 1.0 : (double)k * e.step; }

__device__ __forceinline__ int cf_cell(const Exact1D &e, double x)
{
    double f = floor(x * (double)e.nC);
    f = fmin(fmax(f, 0.0), (double)(e.nC - 1));
    return (int)f;
}

__device__ __forceinline__ double cf_v(const Exact1D &e, double x, int c)
{
    if (!(0 <= x && x <= 1)) return 0.0;
    return e.A[2 * c] * x + e.A[2 * c + 1];
}

__device__ __forceinline__ bool near0(double v) { return fabs(v) <= 1e-8; }

// find_crossing_time; next = -1 for "never".
__device__ double cf_crossing(const Exact1D &e, double x, int c, int &next)
{
    const double a = e.A[2 * c], b = e.A[2 * c + 1];
    const double v = cf_v(e, x, c);
    next = -1;
    if (near0(v)) return CUDART_INF;
    const int cn = c + (v > 0 ? 1 : -1);
    if (!(0 <= cn && cn < e.nC)) return CUDART_INF;
    double xn = (v > 0) ? vert(e, cn) + 1e-16 : vert(e, c) - 1e-16;
    const double vn = cf_v(e, xn, cn);
    if (near0(vn)) return CUDART_INF;
    if ((v > 0) != (vn > 0)) return CUDART_INF;
    double t;
    if (xn == 0 || xn == 1) t = CUDART_INF;
    else if (near0(a)) t = (xn - x) / b;
    else t = e.ia[c] * log((xn + e.ba[c]) / (x + e.ba[c]));   // 1.0/a * log((xn + b/a) / (x + b/a))
    next = cn;
    return t;
}

// FP32 mode (float points; hitting times stay FP64): the time to the exit
// of the first cell as a difference of logarithms, log|xn + b/a| taken from
// the per-cell table, so that a point costs one log and no division; within
// a few ulps of the reference's log of the ratio, i.e. a time error of order
// 1e-16 |log(...)| / |a| -- far below the float result's rounding.
__device__ double cf_crossing_f32(const Exact1D &e, double x, int c, int &next)
{
    const double a = e.A[2 * c], b = e.A[2 * c + 1];
    const double v = cf_v(e, x, c);
    next = -1;
    if (near0(v)) return CUDART_INF;
    const int cn = c + (v > 0 ? 1 : -1);
    if (!(0 <= cn && cn < e.nC)) return CUDART_INF;
    const double xn = (v > 0) ? vert(e, cn) + 1e-16 : vert(e, c) - 1e-16;
    const double vn = cf_v(e, xn, cn);
    if (near0(vn)) return CUDART_INF;
    if ((v > 0) != (vn > 0)) return CUDART_INF;
    double t;
    if (xn == 0 || xn == 1) t = CUDART_INF;
    else if (near0(a)) t = (xn - x) / b;
    else t = e.ia[c] * (e.lx[2 * c + (v > 0 ? 0 : 1)] - log(fabs(x + e.ba[c])));
    next = cn;
    return t;
}

// FP32 mode: the final position x + t v(x) phi(a t), phi(z) = (e^z - 1)/z,
// with v in FP64 (it multiplies the flow's expansion e^{a t}) and phi in
// FP32 (relative error ~2e-7 of a displacement within one cell).  Equal in
// exact arithmetic to the reference's e^{at} x + b (e^{at} - 1)/a.
__device__ __forceinline__ double cf_phi_f32(const Exact1D &e, int c, double x, double t)
{
    const double a = e.A[2 * c], b = e.A[2 * c + 1];
    if (!(0 <= x && x <= 1)) return x;
    if (a == 0) return x + t * b;
    const double v = fma(a, x, b);
    const float z = (float)(a * t);
    const float phi = fabsf(z) < 1e-3f ? fmaf(z, fmaf(z, fmaf(z, 1.f / 24.f, 1.f / 6.f), 0.5f), 1.f)
                                       : expm1f(z) / z;
    return fma(t * v, (double)phi, x);
}

__device__ __forceinline__ double cf_phi(const Exact1D &e, int c, double x, double t)
{
    double a = e.A[2 * c], b = e.A[2 * c + 1];
    if (!(0 <= x && x <= 1)) { a = 0; b = 0; }
    if (a == 0) return x + t * b;
    const double ea = exp(t * a);
    return ea * x + b * (ea - 1) * e.ia[c];  // b (e^{at} - 1) / a with the cell's precomputed 1/a
}

// Every visit after the first starts at a nudged vertex (x_k + 1e-12 when
// entering cell k from the left, x_{k+1} - 1e-12 from the right), so its
// hitting time depends on (cell, direction) only.  Those are evaluated once
// per instance with the same function (cf_crossing) into shared memory, one
// record per (cell k, direction dir) at index 2 k + dir:
//   te[.] = {hitting time, entry point},
//   cn[.] = {cell of the entry point, index of the next record or -1}
// (dir 0: entered from the left, 1: from the right), so a step of the walk
// is one 16-byte and one 8-byte load.  The results are those of evaluating
// cf_crossing at every visit.
// All points of a cell that leave it in one direction cross at least `hops`
// more cells: the ones the slowest of them -- the point that enters at the far
// vertex -- crosses.  A point's walk therefore starts at record rec, `hops`
// records after the cell's neighbour, cum of its time gone.  Two per cell
// (c, to the right) at 2 c and (c, to the left) at 2 c + 1.
struct Skip {
    double cum;
    int rec, hops;
};

struct Transit {
    double2 *te;
    int2 *cn;
    Skip *skip;  // [2 nC] or nullptr
};

// Transit record entered when moving from cell c into cell n (from the left
// when moving right): 2 n + dir, or -1 when there is no next cell.
__device__ __forceinline__ int record_of(int n, int c) { return n < 0 ? -1 : 2 * n + (n > c ? 0 : 1); }

__device__ void build_transit(const Exact1D &e, Transit tr)
{
    for (int r = threadIdx.x; r < 2 * e.nC; r += blockDim.x) {
        const int k = r >> 1;
        const double x = fmin(1.0, fmax(0.0, (r & 1) ? vert(e, k + 1) - 1e-12 : vert(e, k) + 1e-12));
        const int c = cf_cell(e, x);
        int n;
        const double t = cf_crossing(e, x, c, n);
        tr.te[r] = make_double2(t, x);
        tr.cn[r] = make_int2(c, record_of(n, c));
    }
}

// After build_transit and a barrier.  The slowest point's time through its own
// cell is the record of entering that cell (when that record leads on in the
// same direction; else points near a zero of the velocity take any time and
// nothing is skipped).  The margin keeps every skipped comparison true for
// all points of the cell: that record enters 1e-12 inside the vertex, and a
// point on it takes up to 1e-12 / v longer (v at least 1e-8, or it never
// leaves: 1e-4); times are logarithms over a, each rounded to some 1e-15 / a (a
// at least 1e-8: 1e-7).
__device__ void build_skip(const Exact1D &e, const Transit &tr, double t_total)
{
    for (int i = threadIdx.x; i < 2 * e.nC; i += blockDim.x) {
        const int c = i >> 1, cn = c + ((i & 1) ? -1 : 1);
        Skip s{0.0, -1, 0};
        if (0 <= cn && cn < e.nC) {
            s.rec = record_of(cn, c);
            if (tr.cn[i].x == c && tr.cn[i].y == s.rec) {
                const double t_min = t_total - tr.te[i].x - (3e-4 + 1e-9 * fabs(t_total));
                // one direction has at most nC - 1 crossings
                while (s.hops < e.nC && s.cum + tr.te[s.rec].x < t_min) {
                    const int next = tr.cn[s.rec].y;
                    if ((unsigned)next >= (unsigned)(2 * e.nC)) break;
                    s.cum += tr.te[s.rec].x;
                    s.rec = next;
                    ++s.hops;
                }
            }
        }
        tr.skip[i] = s;
    }
}

// calc_phi for one point; returns false when the crossing cap is hit
// (the reference raises ValueError, ClosedFormInt.py:155-160).  F32: the
// first hitting time and the final position of the FP32 mode (above).
template <bool F32>
__device__ bool cf_point(const Exact1D &e, const Transit &tr, double x, double t, int cap, double &out,
                         unsigned &visits)
{
    double x_old = x, t_rem = t;
    if (0 < x_old && x_old < 1) {
        // on a vertex with non-positive velocity: start just left of it
        double u = x_old * (double)e.nC;
        int k = (int)rint(u);
        if (k >= 0 && k <= e.nC && vert(e, k) == x_old) {
            int c = k < e.nC ? k : e.nC - 1;
            double vk = e.A[2 * c] * x_old + e.A[2 * c + 1];
            if (!(vk > 0)) x_old = x_old - 1e-16;
        }
    }
    // first visit: general position
    int c = cf_cell(e, x_old), cn;
    double tc = F32 ? cf_crossing_f32(e, x_old, c, cn) : cf_crossing(e, x_old, c, cn);
    // the record of the next cell (entered at its nudged vertex, from the left when moving right)
    int idx = record_of(cn, c);
    bool ok = true;
    // walk the transit table (cheap, divergent); the final exponential runs
    // after the loop so that all lanes of a warp evaluate it together
    for (int counter = 0;;) {
        ++visits;
        // stop when the remaining time ends inside this cell, when no further
        // crossing exists (idx -1, or any index outside the table), and on NaN
        // (comparisons with NaN are false)
        if (!(tc < t_rem) || (unsigned)idx >= (unsigned)(2 * e.nC)) break;
        t_rem -= tc;
        if (tr.skip && counter == 0) {
            const Skip s = tr.skip[2 * c + (idx & 1)];
            t_rem -= s.cum;
            idx = s.rec;
            counter = s.hops;
            visits += s.hops;
        }
        const double2 te = tr.te[idx];
        if (++counter >= cap) {
            // the point would have been left at the crossing it just made
            x_old = te.y;
            ok = false;
            break;
        }
        const int2 nn = tr.cn[idx];
        x_old = te.y;
        tc = te.x;
        c = nn.x;
        idx = nn.y;
    }
    out = ok ? fmin(1.0, fmax(0.0, F32 ? cf_phi_f32(e, c, x_old, t_rem) : cf_phi(e, c, x_old, t_rem))) : x_old;
    return ok;
}

// Cell-sort key of a start point: only groups points (any key in [0, nC)
// keeps the results; the walk itself uses cf_cell), so float points take a
// float product and a conversion (NaN converts to 0).
__device__ __forceinline__ int sort_key(const Exact1D &e, double x) { return cf_cell(e, x); }
__device__ __forceinline__ int sort_key(const Exact1D &e, float x)
{
    return min(max((int)(x * (float)e.nC), 0), e.nC - 1);
}

// Shared memory of k_exact1d: per cell A (2 doubles), b/a and 1/a (2), the
// two exit logarithms (2), and two transit records (2 x (16 + 8) bytes) --
// 96 bytes, so what follows is 16-byte aligned -- and, when cell-sorting,
// sorted start points and results in input order [tile_pts] (Real), the
// permutation [tile_pts] (16-bit) and the histogram [nC] (int).
// Instances of fewer points than this walk without the table, whose making takes longer than it saves (FP64, 4096
// instances of 128 points 47.9 us with it, 43.9 without, of 256 points 55.8 and 59.4, of 512 75.8 and 97.5).
constexpr int kSkipFew = 256;
size_t exact1d_skip_bytes(int nC) { return (size_t)nC * 2 * sizeof(Skip); }

size_t exact1d_smem_bytes(int nC, int tile_pts, int sort, int prec)
{
    size_t b = (size_t)nC * (6 * sizeof(double) + 2 * (sizeof(double2) + sizeof(int2)));
    if (sort)
        b += 2 * (size_t)tile_pts * (prec == PREC_F64 ? sizeof(double) : sizeof(float)) +
             (size_t)tile_pts * sizeof(unsigned short) + ((size_t)nC + 2) * sizeof(int);
    return b;
}

// Resident CTAs of 256 threads the register allocation must allow per SM,
// and the tiles a CTA takes in a row.  Measured on the batched 1D workload
// (88 M points, 4096 instances), same box: 6 CTAs (40 registers) in groups
// of 2 tiles 1.98 ms; 6 CTAs, single tiles 2.02 ms; 5 CTAs (48 registers)
// 2.05 ms in groups of 2, 2.09 ms in groups of 4, 2.17 ms single; the
// compiler's own register choice (96) 2.51 ms.  A contiguous range of tiles
// per CTA (one table build per instance and CTA) was slower (3.10 ms):
// instances differ in cost, and strided groups spread them over the CTAs.
#ifndef CPAB_EXACT1D_MIN_BLOCKS
#define CPAB_EXACT1D_MIN_BLOCKS 6
#endif
#ifndef CPAB_EXACT1D_TILE_GROUP
#define CPAB_EXACT1D_TILE_GROUP 2
#endif

template <typename Real>
__global__ void __launch_bounds__(256, CPAB_EXACT1D_MIN_BLOCKS) k_exact1d(IntegrateArgs a, bool skip)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int nC = a.t.nC;
    double *sA = reinterpret_cast<double *>(smem_raw);
    double *s_ba = sA + 2 * nC, *s_ia = s_ba + nC, *s_lx = s_ia + nC;
    Transit tr;
    tr.te = reinterpret_cast<double2 *>(s_lx + 2 * nC);
    tr.cn = reinterpret_cast<int2 *>(tr.te + 2 * nC);
    Skip *const skips = skip ? reinterpret_cast<Skip *>(tr.cn + 2 * nC) : nullptr;
    tr.skip = nullptr;
    // cell-sort scratch (see exact1d_smem_bytes)
    const int tp = a.batch.tile_pts;
    Real *s_xs = reinterpret_cast<Real *>(skip ? (void *)(skips + 2 * nC) : (void *)(tr.cn + 2 * nC));
    Real *s_y = s_xs + tp;
    unsigned short *s_perm = reinterpret_cast<unsigned short *>(s_y + tp);
    // the histogram after the 16-bit permutation, rounded up to a 4-byte boundary
    int *s_hist = reinterpret_cast<int *>(s_perm + ((tp + 1) & ~1));
    __shared__ TileInfo s_tile;
    __shared__ int s_claim;
    const double T_total = a.dt * (double)a.nTimeSteps;
    const int64_t ntiles = total_tiles(a.batch);
    const int lane = threadIdx.x & 31;
    // per-lane counts stay far below 2^32 (a lane finishes a few thousand points)
    unsigned c_pts = 0, c_fail = 0, c_nan = 0;
    unsigned long long c_visits = 0;
    unsigned visits = 0;  // folded into c_visits after every tile
    int loaded = -1;
    Exact1D e;
    e.A = sA;
    e.ba = s_ba;
    e.ia = s_ia;
    e.lx = s_lx;
    e.nC = nC;
    e.step = 1.0 / (double)nC;
    // the reference gives up after nC crossings
    const int cap = nC;
    // CTAs take groups of G consecutive tiles, strided over the grid (the
    // tiles of a group mostly share an instance, so its tables are built once)
    constexpr int G = CPAB_EXACT1D_TILE_GROUP;
    for (int64_t it = 0;; ++it) {
        const int64_t grp = (int64_t)blockIdx.x + (it / G) * gridDim.x;
        const int64_t tile = grp * G + it % G;
        if (grp * G >= ntiles) break;
        if (tile >= ntiles) continue;
        if ((it & 7) == 0 && cta_cancelled(a.cancel, a.counters)) break;
        if (threadIdx.x == 0) {
            s_tile = decode_tile(a.batch, tile);
            s_claim = 0;
        }
        __syncthreads();
        const TileInfo ti = s_tile;
        if (ti.inst != loaded) {
            const double *gA = a.A + (size_t)ti.inst * nC * 2;
            for (int i = threadIdx.x; i < nC * 2; i += blockDim.x) sA[i] = gA[i];
            for (int c = threadIdx.x; c < nC; c += blockDim.x) {
                const double ac = gA[2 * c], bc = gA[2 * c + 1];
                const double ba = bc / ac;
                s_ba[c] = ba;
                s_ia[c] = 1.0 / ac;
                if (sizeof(Real) == 4) {
                    s_lx[2 * c] = log(fabs(vert(e, c + 1) + 1e-16 + ba));
                    s_lx[2 * c + 1] = log(fabs(vert(e, c) - 1e-16 + ba));
                }
            }
            __syncthreads();
            build_transit(e, tr);
            loaded = ti.inst;
            __syncthreads();
            const int64_t size = a.batch.offsets ? a.batch.offsets[ti.inst + 1] - a.batch.offsets[ti.inst] : a.batch.n_uniform;
            tr.skip = size >= kSkipFew ? skips : nullptr;
            if (tr.skip) {
                build_skip(e, tr, T_total);
                __syncthreads();
            }
        }
        const int n = (int)(ti.end - ti.start);
        // the tile's points: 32-bit offsets from one base pointer
        const Real *tin = static_cast<const Real *>(a.pts_in) + ti.start;
        Real *tout = static_cast<Real *>(a.pts_out) + ti.start;
        if (a.sort) {
            // counting sort by start cell: a warp then takes neighbouring points,
            // which cross the same cells (same walk length).  Points are staged
            // in shared memory so that global loads and stores stay coalesced.
            for (int c = threadIdx.x; c < nC; c += blockDim.x) s_hist[c] = 0;
            __syncthreads();
            for (int j = threadIdx.x; j < n; j += blockDim.x) {
                const Real xin = tin[j];
                s_y[j] = xin;
                atomicAdd(s_hist + sort_key(e, xin), 1);
            }
            __syncthreads();
            warp0_exclusive_scan(s_hist, nC);
            __syncthreads();
            for (int j = threadIdx.x; j < n; j += blockDim.x) {
                const Real xin = s_y[j];
                const int pos = atomicAdd(s_hist + sort_key(e, xin), 1);
                s_perm[pos] = (unsigned short)j;
                s_xs[pos] = xin;
            }
            __syncthreads();
        }
        // warps claim 32 consecutive (sorted) points at a time until the tile is done
        for (;;) {
            int base = 0;
            if (lane == 0) base = atomicAdd(&s_claim, 32);
            base = __shfl_sync(FULL, base, 0);
            if (base >= n) break;
            const int k = base + lane;
            if (k < n) {
                const Real xin = a.sort ? s_xs[k] : tin[k];
                double y;
                bool ok = cf_point<sizeof(Real) == 4>(e, tr, (double)xin, T_total, cap, y, visits);
                if (a.clamp) y = clamp_ref(y, a.clamp_lo, a.clamp_hi);
                Real yo = (Real)y;
                if (a.sort) s_y[s_perm[k]] = yo;
                else tout[k] = yo;
                ++c_pts;
                c_fail += ok ? 0u : 1u;
                c_nan += (y != y) ? 1u : 0u;
            }
        }
        c_visits += visits;
        visits = 0;
        __syncthreads();
        if (a.sort) {
            for (int j = threadIdx.x; j < n; j += blockDim.x) tout[j] = s_y[j];
            // the next tile rewrites s_y only after its first barrier
        }
    }
    if (a.counters) {
        const unsigned long long pts = warp_sum_u64(c_pts), fails = warp_sum_u64(c_fail),
                                 nans = warp_sum_u64(c_nan);
        c_visits = warp_sum_u64(c_visits);
        if ((threadIdx.x & 31) == 0) {
            if (nans) atomicAdd(a.counters + CNT_NAN, nans);
            atomicAdd(a.counters + CNT_FAST, c_visits);  // cell visits (closed-form segments)
            atomicAdd(a.counters + CNT_POINTS, pts);
            atomicAdd(a.counters + CNT_FAILED, fails);
        }
    }
}

// ------------------------------------------------------------ FP32: intervals of the flow map
//
// The map x -> T(x) of one instance is analytic between the points where the
// start cell or the end cell changes: on such an interval every point leaves
// its start cell c after a time it alone decides, crosses the same cells, and
// ends in the same cell d.  With x0 in the interval, y0 = T(x0), and dt the
// flow time from x0 to x inside c,
//     dt = log1p(z) / a_c,  z = a_c (x - x0) / v_c(x0),
//     T(x) = y0 + v_d(y0) (e^{a_d dt} - 1) / a_d,
// i.e. T(x) = y0 + (x - x0) G L(z) phi(w), G = v_d(y0) / v_c(x0),
// L(z) = log1p(z)/z, phi(w) = (e^w - 1)/w, w = a_d (x - x0)/v_c(x0) L(z).
// Points that stay in c: z = w = 0 and G = e^{a_c t}.  An interval is found
// from the start cell's list by bisection (two or three intervals per cell,
// more around a source), so a point costs no walk, no FP64 and no sort.
//
// x0 and y0 come from the FP64 tables of the walk: the ends of an interval are
// where a point reaches a cell's vertex exactly at the end time, one exponential
// each; hitting times stay FP64.  Anchored at the end where v_c is smaller, z is
// >= 0 or small, and the rounding of the float formula is relative to the
// displacement inside d.  Error: float rounding of the result (2.2e-8 of the
// norm on the batched workload, as the walk's).  Intervals that the float
// formula cannot resolve, points outside [0, 1] and NaN take the walk
// (cf_point), and an instance whose intervals come out unordered does so
// altogether.
//
// A point's cost does not depend on its instance, so a CTA takes a contiguous
// range of points and builds each instance's tables once: batched 1D workload
// (88 M points, 4096 instances) 0.77 ms against 2.04 ms for the sorted walk.
// Bound by instruction issue: about a third of the time is table builds, a
// third the two functions, and 8 bytes per point would take 0.11 ms.
struct __align__(16) Interval {
    float x0, y0h, y0l, G, iv, za, ad;
    int visits;  // cells a point visits; 0: take the walk
};

constexpr int kBins = 4;  // lookup bins per cell

// Per cell: A, b/a, 1/a and the transit records (80 bytes), two intervals and
// their lower ends, the list's start (one per side while building) and the bins.
size_t exact1d_interval_bytes(int nC)
{
    return (size_t)nC * (4 * sizeof(double) + 2 * (sizeof(double2) + sizeof(int2))) +
           (size_t)(2 * nC + 2) * (sizeof(Interval) + sizeof(float)) + (size_t)(3 * nC + 1) * sizeof(int) +
           (size_t)(kBins * nC) * sizeof(unsigned short);
}

struct IntervalTables {
    Interval *iv;         // [2 nC + 2]
    float *bp;            // [2 nC + 2] lower ends: a float is >= bp exactly when it is >= the end itself
    int *base;            // [3 nC + 1] while building: first interval of (cell, left / stays / right)
    unsigned short *bin;  // [kBins nC] interval at each bin's lower edge
};

// An interval while it is being built, in its record's place.
struct IntervalSeed {
    int cell_side;  // 4 cell + side (0 left, 1 stays, 2 right)
    int rec;        // the end cell's record
    double cum;     // time from the first exit to entering it
    double t_max;   // longest time a moving point of the cell takes to the exit
};

// The points of cell c that leave it in direction dir (0 right, 1 left).
// Returns the record of the neighbour they enter, -1 when none leave (the
// conditions are cf_crossing's at the exit); t_max as above (infinite when
// the velocity has a zero in the cell).
__device__ int cell_side(const Exact1D &e, const Transit &tr, int c, int dir, double &t_max, bool &odd)
{
    const int cn = c + (dir ? -1 : 1);
    t_max = 0.0;
    if (!(0 <= cn && cn < e.nC)) return -1;
    const double xe = vert(e, c + 1 - dir), xn = dir ? xe - 1e-16 : xe + 1e-16;
    const double vn = cf_v(e, xn, cn), ve = e.A[2 * c] * xe + e.A[2 * c + 1];
    if (xn == 0 || xn == 1 || near0(vn) || (dir ? vn > 0 : vn < 0)) return -1;
    if (!(dir ? ve < 0 : ve > 0)) {
        odd = odd || !near0(ve);  // the velocity changes sign at the vertex (or is NaN)
        return -1;
    }
    const int rec = record_of(cn, c), r = 2 * c + dir;
    // entering at the far vertex leads out here: the whole cell moves this way
    t_max = tr.cn[r].x == c && tr.cn[r].y == rec ? tr.te[r].x : CUDART_INF;
    return rec;
}

// x at time tau before the exit
__device__ __forceinline__ double back_from(double xe, double ve, double a, double tau)
{
    const double z = -a * tau;
    return fabs(z) < 1e-12 ? xe - ve * tau : xe + ve * expm1(z) / a;
}

// All threads of the CTA; barriers inside.  Returns false (in every thread)
// when the instance takes the walk.
__device__ bool build_intervals(const Exact1D &e, const Transit &tr, const IntervalTables &it, double t_total)
{
    __shared__ int s_bad;
    const int nC = e.nC;
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
    // counts per (cell, side): the cells a point may end in, from the one reached from the far end (all of
    // its records' times within t_total - t_max) to the one reached from the exit (within t_total)
    for (int i = threadIdx.x; i < 2 * nC; i += blockDim.x) {
        const int c = i >> 1, dir = i & 1;
        double t_max, cum = 0.0;
        bool odd = false;
        int rec = cell_side(e, tr, c, dir, t_max, odd), n = 0;
        const bool all = rec >= 0 && t_max < t_total;
        while (rec >= 0 && n < nC) {
            cum += tr.te[rec].x;
            n += !all || !(cum < t_total - t_max) ? 1 : 0;
            if (!(cum < t_total) || (unsigned)(rec = tr.cn[rec].y) >= (unsigned)(2 * nC)) break;
        }
        it.base[3 * c + (dir ? 0 : 2)] = n;
        if (odd) s_bad = 1;
    }
    if (threadIdx.x == 0) it.base[3 * nC] = 0;
    __syncthreads();
    for (int c = threadIdx.x; c < nC; c += blockDim.x) {
        // nothing stays where the whole cell leaves in time
        double tl, tr_;
        bool odd = false;
        const int l = cell_side(e, tr, c, 1, tl, odd), r = cell_side(e, tr, c, 0, tr_, odd);
        it.base[3 * c + 1] = (l >= 0 && tl < t_total) || (r >= 0 && tr_ < t_total) ? 0 : 1;
    }
    __syncthreads();
    warp0_exclusive_scan(it.base, 3 * nC + 1);
    __syncthreads();
    const int total = it.base[3 * nC];
    const bool walk = total > 2 * nC + 1 || s_bad != 0;  // bp holds one end more
    __syncthreads();  // s_bad is read by all before it is written again
    if (walk) return false;
    for (int i = threadIdx.x; i < 2 * nC; i += blockDim.x) {
        const int c = i >> 1, dir = i & 1;
        const int k0 = it.base[3 * c + (dir ? 0 : 2)], k1 = it.base[3 * c + (dir ? 1 : 3)];
        double t_max, cum = 0.0;
        bool odd = false;
        int rec = cell_side(e, tr, c, dir, t_max, odd);
        const bool all = t_max < t_total;
        // the walk goes from the farthest interval's end cell on; the farthest interval is the lowest of a
        // right side, the highest of a left one
        int n = 0;
        while (n < k1 - k0) {
            const double t = tr.te[rec].x;
            if (!all || !(cum + t < t_total - t_max)) {
                const int k = dir ? k1 - 1 - n : k0 + n;
                *reinterpret_cast<IntervalSeed *>(it.iv + k) = IntervalSeed{4 * c + (dir ? 0 : 2), rec, cum, t_max};
                ++n;
            }
            cum += t;
            rec = tr.cn[rec].y;
        }
    }
    for (int c = threadIdx.x; c < nC; c += blockDim.x)
        if (it.base[3 * c + 2] > it.base[3 * c + 1])
            *reinterpret_cast<IntervalSeed *>(it.iv + it.base[3 * c + 1]) = IntervalSeed{4 * c + 1, -1, 0.0, 0.0};
    __syncthreads();
    // lower ends
    for (int k = threadIdx.x; k < total; k += blockDim.x) {
        const IntervalSeed q = *reinterpret_cast<const IntervalSeed *>(it.iv + k);
        const int c = q.cell_side >> 2, side = q.cell_side & 3;
        const double a = e.A[2 * c], lo = vert(e, c), hi = vert(e, c + 1);
        double x = lo;
        // times before the exit: a right side's far end, a left side's near end, a staying part's left neighbour
        const double xe = side == 2 ? hi : lo, ve = a * xe + e.A[2 * c + 1];
        if (side == 2) {
            const double tau = fmin(t_total - q.cum, q.t_max);
            if (tau < q.t_max || !(q.t_max < t_total)) x = back_from(xe, ve, a, fmin(tau, t_total));
        } else if (side == 0) {
            const double tau = t_total - q.cum - tr.te[q.rec].x;
            if (tau > 0.0) x = back_from(xe, ve, a, tau);
        } else {
            double t_max;
            bool odd = false;
            if (cell_side(e, tr, c, 1, t_max, odd) >= 0) x = back_from(xe, ve, a, t_total);
        }
        x = fmin(fmax(x, lo), hi);
        float f = __double2float_ru(x);
        // a point at a vertex where the velocity is not positive starts left of it (cf_point)
        if (x == lo && c > 0 && (double)f == lo && !(a * lo + e.A[2 * c + 1] > 0)) f = nextafterf(f, 2.0f);
        it.bp[k] = f;
    }
    if (threadIdx.x == 0) it.bp[total] = 2.0f;
    __syncthreads();
    for (int k = threadIdx.x; k < total; k += blockDim.x) {
        const IntervalSeed q = *reinterpret_cast<const IntervalSeed *>(it.iv + k);
        const int c = q.cell_side >> 2, side = q.cell_side & 3;
        const double a = e.A[2 * c], b = e.A[2 * c + 1];
        if (!(it.bp[k] <= it.bp[k + 1])) s_bad = 1;  // bisection would mean nothing
        Interval o;
        o.iv = o.za = o.ad = 0.0f;
        // stays: the middle; moving: the end where the cell's velocity is smaller.  Ending in the first cell, the
        // low end: results next to zero are then sums of positive terms, right to float rounding of themselves
        // (from the middle or the high end, of the cell's width: 1.7e-4 of results around 1e-6 before)
        const bool first = (side == 1 ? c : tr.cn[q.rec].x) == 0;
        const bool at_low = (a > 0) == (side == 2) || first;
        const float high = fminf(it.bp[k + 1], 1.0f);
        o.x0 = side == 1 && !first ? 0.5f * (it.bp[k] + high) : (at_low ? it.bp[k] : high);
        const double x0 = o.x0, vc = a * x0 + b;
        double y0;
        bool ok;
        if (side == 1) {
            const double em = expm1(a * t_total);
            y0 = a == 0 ? x0 + t_total * b : x0 + vc * em / a;
            o.G = (float)(1.0 + em);
            o.visits = 1;
            ok = true;
        } else {
            const double xe = vert(e, c + (side == 2 ? 1 : 0)), ve = a * xe + b, zc = a * (xe - x0) / vc;
            const double tau = fabs(zc) < 1e-12 ? (xe - x0) / vc : log1p(zc) / a;
            const int d = tr.cn[q.rec].x;
            const double ad = e.A[2 * d], ye = tr.te[q.rec].y, vy = ad * ye + e.A[2 * d + 1];
            const double t = t_total - q.cum - tau, em = expm1(ad * t);
            y0 = fabs(ad * t) < 1e-12 ? ye + vy * t : ye + vy * em / ad;
            o.G = (float)(vy * (1.0 + em) / vc);
            o.iv = (float)(1.0 / vc);
            o.za = (float)(a / vc);
            o.ad = (float)ad;
            // crossed: |end cell - start cell| cells, one more visit
            o.visits = abs((q.rec >> 1) - c) + 1;
            // resolved: the anchor moves as the interval does, away from the zero of the velocity
            ok = fabs(vc) > 1e-6 && (vc > 0) == (ve > 0);
            // log1p far below the anchor's velocity is not
            if (first) ok = ok && fabs(a * (double)high + b) >= 0.1 * fabs(vc);
        }
        o.y0h = (float)y0;
        o.y0l = (float)(y0 - (double)o.y0h);
        if (!(ok && isfinite(o.G) && isfinite(o.za) && isfinite(o.y0h))) o.visits = 0;
        it.iv[k] = o;
    }
    // bins: the interval (the last with bp <= x) a little below each lower edge, as x * bins rounds
    const int nb = kBins * nC;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        const float x = ((float)i - 0.01f) / (float)nb;
        int k = 0, m = total;
        while (m > 1) {
            const int half = m >> 1;
            const bool up = x >= it.bp[k + half];
            k += up ? half : 0;
            m = up ? m - half : half;
        }
        it.bin[i] = (unsigned short)k;
    }
    __syncthreads();
    const bool good = s_bad == 0;
    __syncthreads();
    return good;
}

// log1p(z)/z and (e^w - 1)/w.  Near zero by their series: with t = z/(2 + z),
// log1p(z) = 2 atanh(t) = 2 t (1 + t^2/3 + t^4/5 + ...), so log1p(z)/z =
// 2/(2 + z) (1 + ...) -- t^14/15 < 5e-8 for -0.4 <= z <= 0.85; and
// 1 + w/2 (1 + w/3 (1 + ...)) -- w^10/11! < 3e-8 up to one.
__device__ __forceinline__ float log1p_over(float z)
{
    if (z >= -0.4f && z <= 0.85f) {
        const float r = __fdividef(1.0f, 2.0f + z), t = z * r, t2 = t * t;
        float p = fmaf(t2, 1.0f / 13, 1.0f / 11);
        p = fmaf(t2, p, 1.0f / 9);
        p = fmaf(t2, p, 1.0f / 7);
        p = fmaf(t2, p, 1.0f / 5);
        p = fmaf(t2, p, 1.0f / 3);
        p = fmaf(t2, p, 1.0f);
        return 2.0f * r * p;
    }
    return log1pf(z) / z;
}
__device__ __forceinline__ float expm1_over(float w)
{
    if (fabsf(w) <= 1.0f) {
        float p = fmaf(w, 1.0f / 10, 1.0f);
        p = fmaf(w * (1.0f / 9), p, 1.0f);
        p = fmaf(w * (1.0f / 8), p, 1.0f);
        p = fmaf(w * (1.0f / 7), p, 1.0f);
        p = fmaf(w * (1.0f / 6), p, 1.0f);
        p = fmaf(w * (1.0f / 5), p, 1.0f);
        p = fmaf(w * (1.0f / 4), p, 1.0f);
        p = fmaf(w * (1.0f / 3), p, 1.0f);
        return fmaf(w * 0.5f, p, 1.0f);
    }
    return expm1f(w) / w;
}

__device__ __forceinline__ float eval_interval(const Interval &o, float x)
{
    const float d = x - o.x0;
    const float s = d * log1p_over(o.za * d);
    const float f = expm1_over(o.ad * (o.iv * s));
    return fminf(1.0f, fmaxf(0.0f, o.y0h + fmaf(o.G * s, f, o.y0l)));
}

// First index with off[index + 1] > s, by one warp (32-way search).
__device__ __forceinline__ int find_instance(const int64_t *off, int N, int64_t s)
{
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = N;  // off[lo] <= s < off[hi]
    while (hi - lo > 1) {
        const int step = (hi - lo + 31) / 32;
        const int p = min(lo + (lane + 1) * step, hi);
        const bool below = p < hi && off[p] <= s;
        const int n = __popc(__ballot_sync(FULL, below));
        hi = min(lo + (n + 1) * step, hi);
        lo += n * step;
    }
    return lo;
}

// Instances of fewer points than kIvFew take the walk, whose table is built
// five times as fast: an instance of 1000 points takes as long either way (4096
// instances of 100 cells: 256 points 50 and 108 us, 512 84 and 127, 1000 134 and
// 142).  The number of an instance's own points decides, nothing of the batch,
// so results do not depend on that.
// A CTA's range is at least kIvMinRange points (kWalkMinRange where instances
// are that small on average), which the build of a table is worth; uniform
// instances of up to kIvPart points per CTA are cut into equal parts, so that
// no CTA builds two tables.
constexpr int kIvUnroll = 4, kIvFew = 1024, kIvMinRange = 1024, kWalkMinRange = 32, kIvPart = 4096;

// 4 resident CTAs of 256 threads (64 registers): 0.77 ms on the batch above; 3, 5, 6: 0.86, 0.84, 0.86.
__global__ void __launch_bounds__(256, 4) k_exact1d_intervals(IntegrateArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int nC = a.t.nC;
    double *sA = reinterpret_cast<double *>(smem_raw);
    double *s_ba = sA + 2 * nC, *s_ia = s_ba + nC;
    Transit tr;
    tr.te = reinterpret_cast<double2 *>(s_ia + nC);
    tr.cn = reinterpret_cast<int2 *>(tr.te + 2 * nC);
    tr.skip = nullptr;
    IntervalTables it;
    it.iv = reinterpret_cast<Interval *>(tr.cn + 2 * nC);
    it.bp = reinterpret_cast<float *>(it.iv + 2 * nC + 2);
    it.base = reinterpret_cast<int *>(it.bp + 2 * nC + 2);
    it.bin = reinterpret_cast<unsigned short *>(it.base + 3 * nC + 1);
    __shared__ int s_inst;
    const double T_total = a.dt * (double)a.nTimeSteps;
    Exact1D e;
    e.A = sA;
    e.ba = s_ba;
    e.ia = s_ia;
    e.lx = nullptr;
    e.nC = nC;
    e.step = 1.0 / (double)nC;
    const float bins = (float)(kBins * nC);
    // this CTA's contiguous range of points, whole warps of 32
    const int64_t p0 = a.batch.offsets ? a.batch.offsets[0] : 0;
    const int64_t p1 = a.batch.offsets ? a.batch.offsets[a.batch.N] : (int64_t)a.batch.N * a.batch.n_uniform;
    const int64_t total = p1 - p0, mean = total / max(a.batch.N, 1);
    int64_t len = (total + gridDim.x - 1) / gridDim.x;
    len = (max(len, (int64_t)(mean < kIvFew ? kWalkMinRange : kIvMinRange)) + 31) / 32 * 32;
    int64_t first = p0 + len * blockIdx.x, last = min(first + len, p1);
    if (!a.batch.offsets && (int64_t)a.batch.N <= gridDim.x) {
        const int64_t n = a.batch.n_uniform, cuts = gridDim.x / a.batch.N;
        const int64_t part = max((n + cuts - 1) / cuts, (int64_t)(n < kIvFew ? 64 : kIvMinRange));
        const int64_t parts = (n + part - 1) / part;
        if (part <= kIvPart) {
            const int64_t i = blockIdx.x / parts;
            if (i >= a.batch.N) return;
            first = i * n + (blockIdx.x - i * parts) * part;
            last = min(first + part, (i + 1) * n);
        }
    }
    if (first >= last) return;
    if (a.batch.offsets) {
        if (threadIdx.x < 32) {
            const int i = find_instance(a.batch.offsets, a.batch.N, first);
            if (threadIdx.x == 0) s_inst = i;
        }
    } else if (threadIdx.x == 0) {
        s_inst = (int)(first / a.batch.n_uniform);
    }
    __syncthreads();
    int inst = s_inst;
    const float *in = static_cast<const float *>(a.pts_in);
    float *out = static_cast<float *>(a.pts_out);
    unsigned c_pts = 0, c_fail = 0, c_nan = 0;
    unsigned long long c_visits = 0;
    bool stop = false;
    for (int64_t pos = first; pos < last && inst < a.batch.N && !stop; ++inst) {
        const int64_t end = min(last, a.batch.offsets ? a.batch.offsets[inst + 1] : (int64_t)(inst + 1) * a.batch.n_uniform);
        if (end <= pos) continue;  // an empty instance
        __syncthreads();
        const double *gA = a.A + (size_t)inst * nC * 2;
        for (int i = threadIdx.x; i < nC * 2; i += blockDim.x) sA[i] = gA[i];
        for (int c = threadIdx.x; c < nC; c += blockDim.x) {
            const double ac = gA[2 * c], ba = gA[2 * c + 1] / ac;
            s_ba[c] = ba;
            s_ia[c] = 1.0 / ac;
        }
        __syncthreads();
        build_transit(e, tr);
        __syncthreads();
        const int64_t size = a.batch.offsets ? a.batch.offsets[inst + 1] - a.batch.offsets[inst] : a.batch.n_uniform;
        const bool use = size >= kIvFew && build_intervals(e, tr, it, T_total);
        // the cancel flag is polled every 16 K points
        constexpr int kChunk = 16384;
        for (; pos < end; pos += kChunk) {
            if (cta_cancelled(a.cancel, a.counters)) {
                stop = true;
                break;
            }
            const int n = (int)min((int64_t)kChunk, end - pos);
            const float *tin = in + pos;
            float *tout = out + pos;
            unsigned visits = 0;
            for (int j0 = threadIdx.x; j0 < n; j0 += kIvUnroll * blockDim.x) {
                float x[kIvUnroll];
                int k[kIvUnroll];
#pragma unroll
                for (int u = 0; u < kIvUnroll; ++u) {
                    const int j = j0 + u * blockDim.x;
                    x[u] = j < n ? __ldg(tin + j) : 0.0f;
                }
#pragma unroll
                for (int u = 0; u < kIvUnroll; ++u) {
                    // the bin's first interval, and on while the point lies beyond the next one's lower end
                    // (the last end is above 1)
                    k[u] = 0;
                    if (use && x[u] >= 0.0f && x[u] <= 1.0f) {
                        k[u] = it.bin[min((int)(x[u] * bins), kBins * nC - 1)];
                        while (x[u] >= it.bp[k[u] + 1]) ++k[u];
                    }
                }
#pragma unroll
                for (int u = 0; u < kIvUnroll; ++u) {
                    const int j = j0 + u * blockDim.x;
                    if (j >= n) break;
                    float y;
                    unsigned v = 0;
                    if (use && x[u] >= 0.0f && x[u] <= 1.0f) {
                        const Interval o = it.iv[k[u]];
                        y = eval_interval(o, x[u]);
                        v = o.visits;
                    }
                    if (v == 0) {
                        double yd;
                        c_fail += cf_point<false>(e, tr, (double)x[u], T_total, nC, yd, v) ? 0u : 1u;
                        y = (float)yd;
                    }
                    if (a.clamp) y = clamp_ref(y, a.clamp_lo, a.clamp_hi);
                    tout[j] = y;
                    ++c_pts;
                    visits += v;
                    c_nan += y != y ? 1u : 0u;
                }
            }
            c_visits += visits;
        }
        pos = end;
    }
    if (a.counters) {
        const unsigned long long pts = warp_sum_u64(c_pts), fails = warp_sum_u64(c_fail), nans = warp_sum_u64(c_nan);
        c_visits = warp_sum_u64(c_visits);
        if ((threadIdx.x & 31) == 0) {
            if (nans) atomicAdd(a.counters + CNT_NAN, nans);
            atomicAdd(a.counters + CNT_FAST, c_visits);
            atomicAdd(a.counters + CNT_POINTS, pts);
            atomicAdd(a.counters + CNT_FAILED, fails);
        }
    }
}

template <typename Real>
static cudaError_t launch_exact1d_t(const IntegrateArgs &a, int prec, const LaunchCfg &cfg, cudaStream_t s)
{
    // With the skip table the walks are short and near equal, and sorting the
    // points costs more than it saves (FP64, 11 M points of 512 instances:
    // 0.27 ms; sorted without it 0.33, sorted with it 0.34).  Where its room
    // would leave one CTA per SM (beyond about 900 cells), the sorted walk.
    IntegrateArgs b = a;
    size_t smem = exact1d_smem_bytes(a.t.nC, a.batch.tile_pts, 0, prec) + exact1d_skip_bytes(a.t.nC);
    const bool skip = smem <= 112 * 1024;
    if (skip) b.sort = 0;
    else smem = exact1d_smem_bytes(a.t.nC, a.batch.tile_pts, a.sort, prec);
    auto kern = k_exact1d<Real>;
    if (smem > kSmemOptInAbove) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    const int grid = cfg.grid > 0 ? cfg.grid : persistent_grid(kern, cfg, smem);
    kern<<<grid, cfg.block, smem, s>>>(b, skip);
    return cudaGetLastError();
}

// Whether FP32 takes the intervals: where their tables leave room for two CTAs
// per SM (about 650 cells); beyond, the walk.
bool exact1d_uses_intervals(int nC, int prec)
{
    return prec == PREC_F32 && exact1d_interval_bytes(nC) <= 112 * 1024;
}

cudaError_t launch_integrate_exact1d(const IntegrateArgs &a, int prec, const LaunchCfg &cfg, cudaStream_t s)
{
    if (prec == PREC_F64) return launch_exact1d_t<double>(a, prec, cfg, s);
    if (!exact1d_uses_intervals(a.t.nC, prec)) return launch_exact1d_t<float>(a, prec, cfg, s);
    const size_t smem = exact1d_interval_bytes(a.t.nC);
    if (smem > kSmemOptInAbove) {
        cudaError_t e = cudaFuncSetAttribute(k_exact1d_intervals, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    k_exact1d_intervals<<<persistent_grid(k_exact1d_intervals, cfg, smem), cfg.block, smem, s>>>(a);
    return cudaGetLastError();
}

}  // namespace cpab
