// cpab_grad.cu -- adjoint (reverse-mode) gradient of the midpoint scheme.
//
// Forward (calc_T_simple, cpab/gpu/calc_2Dto2D.cu:412-445): nTimeSteps *
// nStepsODE explicit-midpoint sub-steps, each with the matrix of the cell
// that holds the sub-step's start point,
//     v = L p + t,  pm = p + h/2 v,  v2 = L pm + t,  p' = p + h v2.
// The reference's own sensitivity code (solveODE2 / calc_grad_theta,
// calc_2Dto2D.cu:202-319,448-491; never bound, cpab/gpu/Calcs.py:196) carries
// dp/dtheta forward for every basis vector.  Here the gradient of a scalar
// loss runs backwards instead: given g = dLoss/dT(x) per point,
//     a = h g',  dL += a pm^T, dt += a,  dpm = L^T a,
//     b = h/2 dpm,  dL += b p^T, dt += b,  g = g' + dpm + L^T b,
// summed per cell into dLoss/dA [nC, D, D+1]; dLoss/dtheta = B^T dLoss/dA
// (k_bt_times).  This is the exact gradient of the discrete forward map.
//
// Memory: positions at the start of every `ck`-th time step are kept in
// scratch ([ceil(nT/ck), nPts, D] float64); the start of any other step is
// recomputed from the previous checkpoint (ck = 1 stores all, ck = nT only
// the input).  Inside a time step the sub-steps are replayed once, keeping
// every sub-step's start point and cell in a per-thread array.
//
// k_grad_ref: the same for the reference scheme (calc_T, calc_2Dto2D.cu:
// 348-408), FP64 and FP32, through the composed steps of cpab_jump.cuh.  A
// time step is either the closed-form step, kept when its end stays in the
// cell, or nStepsODE sub-steps; the forward takes runs of either inside one
// cell as one application of the map's power, r' = r + M [r; 1] on the
// position r in the box, and records each move's table row and start.  The
// adjoint runs down that list,
//     dM += g [r; 1]^T,   g = g + M_lin^T g,
// with dM summed per instance, cell and table row.  Once per instance and
// cell, k_level_sums takes the sums down the levels -- D' = 2 D + D_lin D for
// a map applied twice, so dD = 2 dD' + D_lin^T dD' + [dD' D^T | 0] -- to
// dLoss/dT_c and dLoss/d(sub-step map)_c, and these become dLoss/dA_c:
// k_frechet_adjoint:
//     dA_c += dt L(X^T, dT_c),  X = dt [A_c; 0],
// L the Frechet derivative of expm, read off the top-right block of
// expm([[X^T, G], [0, X^T]]), and k_substep_map_adjoint.  This is the exact
// gradient of the discrete map along the branch calc_T takes (kept / fallback,
// cells; Path); where a perturbation flips a branch the map itself jumps
// by the sub-steps' discretisation error.  Nothing is checkpointed: the list
// holds kMoves moves of a trajectory (most take 5 to 30) in local memory, and
// a longer one is replayed in blocks from saved states.
//
// Measured, 3D with 320 cells, FP32, 8 theta x 64^3 points, forward and
// backward: one step at a time 30.8 ms -- 4.8 of 32 lanes active, a fallback
// step holding up its warp -- this 4.1 ms.
#include <algorithm>
#include <climits>

#include "cpab_integrate.cuh"
#include "cpab_jump.cuh"
#include "cpab_grad.h"
#include "cpab_launch.h"

namespace cpab {

constexpr int kMaxSubsteps = 256;  // sub-steps per time step the adjoint keeps (cpab_grad_theta* check)

template <int DIM, int TESS>
__device__ __forceinline__ void substeps(const Tess &t, const double *sA, double *p, double h, int n)
{
    constexpr int NE = DIM * (DIM + 1);
    for (int k = 0; k < n; ++k) {
        int c = exact_cell<DIM, TESS>(t, p);
        exact_midpoint<DIM>(p, sA + c * NE, h);
    }
}

// Per-thread accumulator of one cell's dLoss/d(matrix) entries, added to the
// CTA's shared sums when the cell changes (c = -1: flush).
template <int NE>
__device__ __forceinline__ void acc_switch(double *sG, double *acc, int &acc_cell, int c)
{
    if (c == acc_cell) return;
    if (acc_cell >= 0) {
#pragma unroll
        for (int e = 0; e < NE; ++e) {
            atomicAdd(sG + acc_cell * NE + e, acc[e]);
            acc[e] = 0.0;
        }
    }
    acc_cell = c;
}

// Backwards through the nODE sub-steps of one time step that starts at q
// (q is consumed): g = dLoss/d(end of the step) on entry, dLoss/d(start) on
// return; dLoss/dA of the cells used is accumulated (acc / acc_cell / sG).
// One forward pass keeps every sub-step's start point and cell in a
// per-thread array (nODE <= 256: at most 7 KB of local memory), then the
// adjoint runs down it.
template <int DIM, int TESS>
__device__ __forceinline__ void adjoint_substeps(const Tess &t, const double *sA, double *sG, double *q, double *g,
                                                 double h, int nODE, double *acc, int &acc_cell)
{
    constexpr int NE = DIM * (DIM + 1), NH = DIM + 1;
    double xs[kMaxSubsteps][DIM];
    int cs[kMaxSubsteps];
    for (int k = 0; k < nODE; ++k) {
        const int c = exact_cell<DIM, TESS>(t, q);
#pragma unroll
        for (int i = 0; i < DIM; ++i) xs[k][i] = q[i];
        cs[k] = c;
        exact_midpoint<DIM>(q, sA + c * NE, h);
    }
    for (int k = nODE - 1; k >= 0; --k) {
        double pk[DIM];
#pragma unroll
        for (int i = 0; i < DIM; ++i) pk[i] = xs[k][i];
        const int c = cs[k];
        const double *M = sA + c * NE;
        acc_switch<NE>(sG, acc, acc_cell, c);
        // recompute v and pm of the forward sub-step
        double v[DIM], pm[DIM];
        exact_affine<DIM>(v, M, pk);
#pragma unroll
        for (int i = 0; i < DIM; ++i) pm[i] = pk[i] + h * v[i] / 2.;
        double av[DIM], dpm[DIM], b[DIM];
#pragma unroll
        for (int i = 0; i < DIM; ++i) av[i] = h * g[i];
#pragma unroll
        for (int jj = 0; jj < DIM; ++jj) {
            double s2 = 0.0;
#pragma unroll
            for (int i = 0; i < DIM; ++i) s2 += M[i * NH + jj] * av[i];
            dpm[jj] = s2;
        }
#pragma unroll
        for (int i = 0; i < DIM; ++i) b[i] = 0.5 * h * dpm[i];
#pragma unroll
        for (int i = 0; i < DIM; ++i) {
#pragma unroll
            for (int jj = 0; jj < DIM; ++jj) acc[i * NH + jj] += av[i] * pm[jj] + b[i] * pk[jj];
            acc[i * NH + DIM] += av[i] + b[i];
        }
#pragma unroll
        for (int jj = 0; jj < DIM; ++jj) {
            double s2 = 0.0;
#pragma unroll
            for (int i = 0; i < DIM; ++i) s2 += M[i * NH + jj] * b[i];
            g[jj] += dpm[jj] + s2;
        }
    }
}

template <int DIM, int TESS>
__global__ void __launch_bounds__(128) k_grad_simple(GradArgs a)
{
    constexpr int NE = DIM * (DIM + 1);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *sA = reinterpret_cast<double *>(smem_raw);
    double *sG = sA + a.t.nC * NE;
    const int inst = blockIdx.y;
    const int tab = a.t.nC * NE;
    for (int i = threadIdx.x; i < tab; i += blockDim.x) {
        sA[i] = a.A[(size_t)inst * tab + i];
        sG[i] = 0.0;
    }
    __syncthreads();
    const double h = XDIV(a.dt, (double)a.nStepsODE);
    const int nT = a.nTimeSteps, nODE = a.nStepsODE, ck = a.ck;
    const int64_t n = a.n_per_inst;
    const int64_t total = n * a.N;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
        const int64_t gi = (int64_t)inst * n + j;
        double p[DIM];
        load_pt<DIM, double>(a.pts, gi, p);
        // forward with checkpoints
        for (int s = 0; s < nT; ++s) {
            if (s % ck == 0) store_pt<DIM, double>(a.ckpt, (int64_t)(s / ck) * total + gi, p);
            substeps<DIM, TESS>(a.t, sA, p, h, nODE);
        }
        if (a.out) store_pt<DIM, double>(a.out, gi, p);
        double g[DIM];
        load_pt<DIM, double>(a.grad_out, gi, g);
        double acc[NE];
#pragma unroll
        for (int e = 0; e < NE; ++e) acc[e] = 0.0;
        int acc_cell = -1;
        for (int s = nT - 1; s >= 0; --s) {
            // start of time step s
            double q[DIM];
            load_pt<DIM, double>(a.ckpt, (int64_t)(s / ck) * total + gi, q);
            substeps<DIM, TESS>(a.t, sA, q, h, s % ck * nODE);
            adjoint_substeps<DIM, TESS>(a.t, sA, sG, q, g, h, nODE, acc, acc_cell);
        }
        acc_switch<NE>(sG, acc, acc_cell, -1);
        if (a.grad_in) store_pt<DIM, double>(a.grad_in, gi, g);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < tab; i += blockDim.x) {
        double v = sG[i];
        if (v != 0.0) atomicAdd(a.gA + (size_t)inst * tab + i, v);
    }
}

// ------------------------------------------------------------ adjoint of calc_T

// Moves of a trajectory kept at once, and states saved of a longer one.
constexpr int kMoves = 48, kSaves = 24;
// Lanes that must add to the same sums for them to be added up in the warp
// first (the 3D case above: 8 lanes 3.98 ms, 4 4.11, 16 4.54).
constexpr int kGroup = 8;

// Points a warp may have left for later, and the units of its first go at a
// point (3D, 320 cells, 8 x 262144 points, value and gradient: 4.20 ms without
// the queue, 4.26 with 4 units first, 4.28 with 6, 3.99 with 10, 4.06 with 16; a
// longer queue no better).
constexpr int kGradQueue = 64, kGradUnits = 10;

// Add each lane's NE values to the sums at G (null: nothing to add; `key`
// tells the sums apart).  Lanes with the same key -- neighbouring points make
// the same moves -- are added up in the warp first: the sums are spread over
// the lanes as they are halved (16 shuffles for up to 16 values), and one lane
// per value adds its share.  Added one by one, 32 lanes to one address, the
// additions bound the kernel (7.6 ms of 8.8 on the case above; 3.2 of 4.0 like
// this, where the moves' list and the sums wait on L2).
template <int NE, typename Real>
__device__ __forceinline__ void add_grouped(double *G, int key, const Real *v)
{
    const int lane = threadIdx.x & 31;
    const unsigned same = __match_any_sync(FULL, G ? key : -1 - lane);
    const bool alone = __popc(same) < kGroup;
    if (G && alone) {
#pragma unroll
        for (int e = 0; e < NE; ++e) atomicAdd(G + e, (double)v[e]);
    }
    unsigned todo = __ballot_sync(FULL, !alone);
    while (todo) {
        const int lead = __ffs(todo) - 1;
        const unsigned members = __shfl_sync(FULL, same, lead);
        const bool in = (members >> lane) & 1u;
        todo &= ~members;
        double *base = reinterpret_cast<double *>(__shfl_sync(FULL, reinterpret_cast<unsigned long long>(G), lead));
        constexpr int kSlots = NE <= 2 ? 2 : NE <= 8 ? 8 : 16;
        Real s[kSlots];
#pragma unroll
        for (int e = 0; e < kSlots; ++e) s[e] = e < NE && in ? v[e < NE ? e : 0] : Real(0);
        int slot = 0;
#pragma unroll
        for (int half = kSlots / 2, bit = 16; bit > 0; half /= 2, bit /= 2) {
            if (half > 0) {
                // keep one half of the values, hand the other to the partner
                const bool up = (lane & bit) != 0;
                if (up) slot += half;
#pragma unroll
                for (int e = 0; e < half; ++e) {
                    const Real give = up ? s[e] : s[e + half], keep = up ? s[e + half] : s[e];
                    s[e] = keep + __shfl_xor_sync(FULL, give, bit);
                }
            } else {
                s[0] += __shfl_xor_sync(FULL, s[0], bit);
            }
        }
        // the lanes that differ only in the bits left over hold the same sum
        if ((lane & (32 / kSlots - 1)) == 0 && slot < NE) atomicAdd(base + slot, (double)s[0]);
    }
}

// Where the sums of table row `key` of this instance are.
template <int NE>
__device__ __forceinline__ double *sums_of(const GradArgs &a, int inst, int key)
{
    const int nC = a.t.nC, s_row = a.jump.nT * nC;
    const bool sub = key >= s_row;
    const int rel = key - (sub ? s_row : 0);
    const size_t tab = (size_t)nC * NE;
    if (rel < nC) return (sub ? a.gS : a.gT) + inst * tab + (size_t)rel * NE;
    return a.gL + inst * (a.jump.nT - 1 + a.jump.nS - 1) * tab + (size_t)(rel - nC + (sub ? (a.jump.nT - 1) * nC : 0)) * NE;
}

// Value and adjoint of one point, its doubtful decisions settled in calc_T's arithmetic; mi, r and save are the
// caller's lists.  Out of line, for points so rare that their lanes may go alone.
template <int DIM, int TESS>
__device__ __noinline__ void careful_point(const GradArgs &a, JumpTables<double> jt, int inst, int64_t gi, int *mi,
                                           double (*r)[DIM], Path<DIM, TESS, double> *save)
{
    constexpr int NE = DIM * (DIM + 1), NH = DIM + 1;
    const size_t tab = (size_t)a.t.nC * NE;
    const double *x0 = static_cast<const double *>(a.pts) + gi * DIM;
    double x[DIM], g[DIM];
    load_pt<DIM, double>(a.pts, gi, x);
    load_pt<DIM, double>(a.grad_out, gi, g);
#pragma unroll
    for (int i = 0; i < DIM; ++i) g[i] *= a.t.inc[i];
    Path<DIM, TESS, double> s;
    ExactPath<DIM, TESS> e;
    e.c = -1;
    int k = 0, block = 0;
    auto unit = [&] {
        k += s.settled_unit(a.t, a.jump, jt, a.A + inst * tab, a.T + inst * tab, a.h_sub, a.nTimeSteps, a.nStepsODE, x0, e,
                            mi[k], r[k]) ? 1 : 0;
    };
    int todo = -1;  // blocks to replay, the first time as many as there are
    for (;;) {
        const int from = todo < 0 ? 0 : min(todo, kSaves - 1);
        if (from == 0) s.begin(a.t, a.jump, x, a.nTimeSteps);
        else s = save[from];
        k = 0;
        block = from;
        while (todo < 0 ? !s.done() : block < todo || k < kMoves) {
            if (k == kMoves) {
                ++block;
                k = 0;
                if (todo < 0 && block < kSaves) save[block] = s;
            }
            unit();
        }
        while (k > 0) {
            --k;
            double *G = sums_of<NE>(a, inst, mi[k]);
            const double *M = jt.map + (size_t)mi[k] * NE;
            double gn[DIM];
#pragma unroll
            for (int c = 0; c < DIM; ++c) {
                gn[c] = g[c];
#pragma unroll
                for (int i = 0; i < DIM; ++i) {
                    atomicAdd(G + i * NH + c, g[i] * r[k][c]);
                    gn[c] += M[c * DIM + i] * g[i];
                }
                atomicAdd(G + c * NH + DIM, g[c]);
            }
#pragma unroll
            for (int c = 0; c < DIM; ++c) g[c] = gn[c];
        }
        todo = block - 1;
        if (todo < 0) break;
    }
    if (a.grad_in) {
#pragma unroll
        for (int i = 0; i < DIM; ++i) g[i] *= a.t.inv_inc[i];
        store_pt<DIM, double>(a.grad_in, gi, g);
    }
}

// Resident CTAs per SM the registers must allow (0: the compiler's choice, 48 registers in 1D, 101 in 3D): 2D FP32, 16 x
// 65536 points, 3 CTAs 593 us, 4 633; FP64 as many as without careful_point's registers (1D 64, else 128).
template <int DIM, typename Real>
constexpr int kGradCtas = sizeof(Real) == 4 ? (DIM == 2 ? 3 : 0) : DIM == 1 ? 4 : 2;

template <int DIM, int TESS, typename Real>
__global__ void __launch_bounds__(256, kGradCtas<DIM, Real>) k_grad_ref(const __grid_constant__ GradArgs a)
{
    constexpr int NE = DIM * (DIM + 1), NH = DIM + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int nC = a.t.nC, tab = nC * NE, inst = blockIdx.y, lane = threadIdx.x & 31;
    const JumpCfg jc = a.jump;
    const JumpTables<Real> jt = stage_jump<DIM, TESS, Real>(a.A + (size_t)inst * tab, a.T + (size_t)inst * tab, a.t, jc,
                                                            a.dt, a.h_sub, false, smem_raw);
    __syncthreads();
    // sums of level 0 (steps, sub-steps), and of the levels above in kappa's order
    double *gT = a.gT + (size_t)inst * tab, *gS = a.gS + (size_t)inst * tab;
    double *gL = a.gL + (size_t)inst * (jc.nT - 1 + jc.nS - 1) * tab;
    const int s_row = jc.nT * nC;
    const int64_t n = a.n_per_inst;
    const Real *pts = static_cast<const Real *>(a.pts), *gout = static_cast<const Real *>(a.grad_out);
    Real *gin = static_cast<Real *>(a.grad_in);
    // 32 points per warp at a time: the next 32 of the instance, as far as a
    // few units take them, or 32 of those that this left over (most points
    // make a few moves, some make dozens: together, the few set the pace of
    // the warp).  A warp with one go at the points takes them to their end.
    int64_t *queue = reinterpret_cast<int64_t *>(smem_raw + jump_bytes(jc, DIM, nC, sizeof(Real))) +
                     (threadIdx.x >> 5) * kGradQueue;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t j0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) - lane;
    const bool once = !a.queue || n <= stride;
    int queued = 0;
    for (;;) {
        const bool next = j0 < n && queued <= kGradQueue - 32;
        if (!next && queued == 0) break;
        const int64_t j = next ? j0 + lane : lane < queued ? queue[max(queued - 32, 0) + lane] : 0;
        bool have = next ? j < n : lane < queued;
        const int most_units = next && !once ? kGradUnits : INT_MAX;
        if (next) j0 += stride;
        else queued = max(queued - 32, 0);
        __syncwarp();
        const int64_t gi = (int64_t)inst * n + j;
        Real x[DIM], g[DIM], r[kMoves][DIM];
        int mi[kMoves];
        Path<DIM, TESS, Real> save[kSaves], s;
        int k = 0, block = 0;
        if (have) {
            load_pt<DIM, Real>(pts, gi, x);
            s.begin(a.t, jc, x, a.nTimeSteps);
            for (int u = 0; u < most_units && !s.done(); ++u) {
                if (k == kMoves) {
                    ++block;
                    k = 0;
                    if (block < kSaves) save[block] = s;
                }
                k += s.unit(a.t, jc, jt, a.nStepsODE, mi[k], r[k]) ? 1 : 0;
                if (s.doubtful()) break;
            }
            if (s.done() && a.out) {
                // (FP32: the end calc_T comes to)
                s.w.position(a.t, x);
                store_pt<DIM, Real>(a.out, gi, x);
            }
        }
        if constexpr (sizeof(Real) == 8) {
            if (have && s.doubtful()) {
                careful_point<DIM, TESS>(a, jt, inst, gi, mi, r, save);
                have = false;
                k = block = 0;
            }
        }
        const bool later = have && !s.done();
        const unsigned put = __ballot_sync(FULL, later);
        if (later) {
            queue[queued + __popc(put & ((1u << lane) - 1u))] = j;
            have = false;
            k = block = 0;
        }
        queued += __popc(put);
        __syncwarp();
        if (have) {
            // dLoss/d(position in the box)
            load_pt<DIM, Real>(gout, gi, g);
#pragma unroll
            for (int i = 0; i < DIM; ++i) g[i] *= (Real)a.t.inc[i];
        }
        for (;;) {
            while (__any_sync(FULL, k > 0)) {
                double *G = nullptr;
                Real v[NE];
                int key = 0;
                if (k > 0) {
                    --k;
                    key = mi[k];
                    const bool sub = key >= s_row;
                    const int rel = key - (sub ? s_row : 0);
                    G = rel < nC ? (sub ? gS : gT) + rel * NE
                                 : gL + (size_t)(rel - nC + (sub ? (jc.nT - 1) * nC : 0)) * NE;
#pragma unroll
                    for (int i = 0; i < DIM; ++i) {
#pragma unroll
                        for (int c = 0; c < DIM; ++c) v[i * NH + c] = g[i] * r[k][c];
                        v[i * NH + DIM] = g[i];
                    }
                    const Real *M = jt.map + (size_t)key * NE;
                    Real gn[DIM];
#pragma unroll
                    for (int c = 0; c < DIM; ++c) {
                        Real u = g[c];
#pragma unroll
                        for (int i = 0; i < DIM; ++i) u += M[c * DIM + i] * g[i];
                        gn[c] = u;
                    }
#pragma unroll
                    for (int c = 0; c < DIM; ++c) g[c] = gn[c];
                }
                add_grouped<NE, Real>(G, key, v);
            }
            if (!__any_sync(FULL, block > 0)) break;
            if (block > 0) {
                // the block before, replayed from the latest saved state at or before its start
                --block;
                const int from = min(block, kSaves - 1);
                if (from == 0) {
                    load_pt<DIM, Real>(pts, gi, x);
                    s.begin(a.t, jc, x, a.nTimeSteps);
                } else {
                    s = save[from];
                }
                // whole blocks of moves up to this one, the last in the list
                for (int skip = block - from; skip >= 0; --skip)
                    for (k = 0; k < kMoves;) k += s.unit(a.t, jc, jt, a.nStepsODE, mi[k], r[k]) ? 1 : 0;
            }
        }
        if (gin && have) {
#pragma unroll
            for (int i = 0; i < DIM; ++i) g[i] *= (Real)a.t.inv_inc[i];
            store_pt<DIM, Real>(gin, gi, g);
        }
    }
}

// dLoss/dD from dLoss/d(2 D + D_lin D), in place.
template <int DIM>
__device__ __forceinline__ void twice_adjoint(const double *D, double *G)
{
    constexpr int NH = DIM + 1, NE = DIM * NH;
    double o[NE];
#pragma unroll
    for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int col = 0; col < NH; ++col) {
            double v = 2.0 * G[r * NH + col];
#pragma unroll
            for (int k = 0; k < DIM; ++k) v = fma(D[k * NH + r], G[k * NH + col], v);
            if (col < DIM) {
#pragma unroll
                for (int q = 0; q < NH; ++q) v = fma(G[r * NH + q], D[col * NH + q], v);
            }
            o[r * NH + col] = v;
        }
#pragma unroll
    for (int e = 0; e < NE; ++e) G[e] = o[e];
}

// The sums of all levels, in box coordinates, taken down to level 0 and to
// the coordinates of the tables: gT becomes dLoss/dT, gS dLoss/d(sub-step map).
template <int DIM, int TESS>
__global__ void k_level_sums(GradArgs a)
{
    constexpr int NH = DIM + 1, NE = DIM * NH;
    const int nC = a.t.nC, extra = a.jump.nT - 1 + a.jump.nS - 1;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (int64_t)2 * a.N * nC;
         i += (int64_t)gridDim.x * blockDim.x) {
        const bool sub = (i & 1) != 0;
        const int64_t ic = i >> 1;
        const int inst = (int)(ic / nC), c = (int)(ic - (int64_t)inst * nC);
        const double *A = a.A + ic * NE, *T = a.T + ic * NE;
        double ctr[DIM], P[9][NE], G[NE];
        {
            int kb[DIM];
            cell_box<DIM, TESS>(a.t, c, kb);
#pragma unroll
            for (int r = 0; r < DIM; ++r) ctr[r] = ((double)kb[r] + 0.5) * a.t.inc[r];
        }
        double D[NE];
        if (sub) {
            midpoint_increment<DIM>(A, a.h_sub, D);
        } else {
#pragma unroll
            for (int e = 0; e < NE; ++e) D[e] = T[e] - (e % NH == e / NH ? 1.0 : 0.0);
        }
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
            double off = D[r * NH + DIM];
#pragma unroll
            for (int k = 0; k < DIM; ++k) {
                off = fma(D[r * NH + k], ctr[k], off);
                P[0][r * NH + k] = D[r * NH + k] * a.t.inc[k] * a.t.inv_inc[r];
            }
            P[0][r * NH + DIM] = off * a.t.inv_inc[r];
        }
        const int top = (sub ? a.jump.nS : a.jump.nT) - 1, q0 = sub ? a.jump.nT - 1 : 0, chain = top * a.jump.r;
        for (int q = 0; q < chain; ++q) {
#pragma unroll
            for (int e = 0; e < NE; ++e) P[q + 1][e] = P[q][e];
            twice<DIM>(P[q + 1]);
        }
        double *g0 = (sub ? a.gS : a.gT) + ic * NE;
#pragma unroll
        for (int e = 0; e < NE; ++e) G[e] = 0.0;
        for (int q = chain; q > 0; --q) {
            if (q % a.jump.r == 0) {
                const double *g = a.gL + (((size_t)inst * extra + q0 + q / a.jump.r - 1) * nC + c) * NE;
#pragma unroll
                for (int e = 0; e < NE; ++e) G[e] += g[e];
            }
            twice_adjoint<DIM>(P[q - 1], G);
        }
#pragma unroll
        for (int e = 0; e < NE; ++e) G[e] += g0[e];
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
            const double go = G[r * NH + DIM] * a.t.inv_inc[r];
#pragma unroll
            for (int k = 0; k < DIM; ++k)
                g0[r * NH + k] = G[r * NH + k] * a.t.inc[k] * a.t.inv_inc[r] + go * ctr[k];
            g0[r * NH + DIM] = go;
        }
    }
}

// gA[c] += dt L(X^T, G_c) for every (instance, cell) c, X = dt [A_c; 0]
// (homogeneous) and G_c = [gT_c; 0]: the top-right block of exp(Z),
// Z = [[X^T, G], [0, X^T]].  Scaling and squaring (Moler & Van Loan, "Nineteen
// dubious ways to compute the exponential of a matrix", method 3) with the
// degree-18 Taylor polynomial of Z / 2^s, |Z / 2^s|_1 <= 1/2 (truncation below
// 1e-22 relative).  Powers of Z keep its shape [[P, Q], [0, P]], so only P and
// Q are carried: P' = P X^T, Q' = Q X^T + P G, and (P^2, P Q + Q P) to square.
// L is linear in G, so G is scaled to max |entry| 1 and the block scaled back,
// which keeps the squaring count set by X.
//
// 16 threads per cell, one matrix entry each, matrices in shared memory: a
// thread per cell had the 2 (DIM + 1) square matrices in local memory and
// too few threads (2560 cells: 0.45 ms of the 3D gradient, this 0.02).
template <int DIM>
__global__ void __launch_bounds__(128) k_frechet_adjoint(const double *A, const double *gT, double *gA, int total,
                                                         double dt)
{
    constexpr int M = DIM + 1, NE = DIM * M;
    __shared__ double s_m[8][6][16];
    const int grp = threadIdx.x >> 4, e = threadIdx.x & 15, i = e / M, j = e - i * M;
    const unsigned mask = 0xffffu << ((threadIdx.x & 16) ? 16 : 0);
    double *X = s_m[grp][0], *G = s_m[grp][1], *P = s_m[grp][2], *Q = s_m[grp][3], *P2 = s_m[grp][4], *Q2 = s_m[grp][5];
    const bool on = e < M * M;
    const int idx = blockIdx.x * 8 + grp;
    if (idx >= total) return;  // whole groups; the barriers below are per group
    const double *a = A + (size_t)idx * NE, *g = gT + (size_t)idx * NE;
    double gs = 0.0;
    for (int k = 0; k < NE; ++k) gs = fmax(gs, fabs(g[k]));
    if (!(gs > 0.0)) return;  // no closed-form step in this cell
    // X^T and G, row-major [i][j], last row of G and last column of X^T zero
    if (on) {
        X[e] = j < DIM ? dt * a[j * M + i] : 0.0;
        G[e] = i < DIM ? g[i * M + j] / gs : 0.0;
    }
    __syncwarp(mask);
    double nrm = 0.0;
    for (int c = 0; c < M; ++c) {
        double cx = 0.0, cg = 0.0;
        for (int r = 0; r < M; ++r) {
            cx += fabs(X[r * M + c]);
            cg += fabs(G[r * M + c]);
        }
        nrm = fmax(nrm, cx + cg);
    }
    int sq = 0;
    while (nrm > 0.5 && sq < 60) {
        nrm *= 0.5;
        ++sq;
    }
    const double sc = ldexp(1.0, -sq);
    __syncwarp(mask);
    double p = i == j ? 1.0 : 0.0, q = 0.0;  // the term
    double sp = p, sum = 0.0;                // the sums
    if (on) {
        X[e] *= sc;
        G[e] *= sc;
        P[e] = p;
        Q[e] = q;
    }
    __syncwarp(mask);
    for (int k = 1; k <= 18; ++k) {
        const double inv = 1.0 / (double)k;
        p = q = 0.0;
        if (on) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
                p = fma(P[i * M + m], X[m * M + j], p);
                q = fma(Q[i * M + m], X[m * M + j], fma(P[i * M + m], G[m * M + j], q));
            }
            p *= inv;
            q *= inv;
            sp += p;
            sum += q;
        }
        __syncwarp(mask);
        if (on) {
            P[e] = p;
            Q[e] = q;
        }
        __syncwarp(mask);
    }
    for (int r = 0; r < sq; ++r) {
        if (on) {
            P2[e] = sp;
            Q2[e] = sum;
        }
        __syncwarp(mask);
        p = q = 0.0;
        if (on) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
                p = fma(P2[i * M + m], P2[m * M + j], p);
                q = fma(P2[i * M + m], Q2[m * M + j], fma(Q2[i * M + m], P2[m * M + j], q));
            }
        }
        sp = p;
        sum = q;
        __syncwarp(mask);
    }
    if (on && i < DIM) gA[(size_t)idx * NE + i * M + j] += dt * gs * sum;
}

// gA[c] += dLoss/dA through S - I = [hL + h^2/2 L^2 | hb + h^2/2 Lb] (A = [L | b]):
//     dL = h G + h^2/2 (G L^T + L^T G + g b^T),   db = h g + h^2/2 L^T g,
// G, g the linear and offset parts of gS[c].
template <int DIM>
__global__ void k_substep_map_adjoint(const double *A, const double *gS, double *gA, int total, double h)
{
    constexpr int M = DIM + 1, NE = DIM * M;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
        const double *a = A + (size_t)idx * NE;
        const double *G = gS + (size_t)idx * NE;
        double *o = gA + (size_t)idx * NE;
        const double hh = 0.5 * h * h;
        for (int i = 0; i < DIM; ++i) {
            for (int j = 0; j < DIM; ++j) {
                double s2 = 0.0;
                for (int k = 0; k < DIM; ++k) s2 += G[i * M + k] * a[j * M + k] + a[k * M + i] * G[k * M + j];
                s2 += G[i * M + DIM] * a[j * M + DIM];
                o[i * M + j] += h * G[i * M + j] + hh * s2;
            }
            double s3 = 0.0;
            for (int k = 0; k < DIM; ++k) s3 += a[k * M + i] * G[k * M + DIM];
            o[i * M + DIM] += h * G[i * M + DIM] + hh * s3;
        }
    }
}

// out[n, j] = scale * sum_k B[k, j] * G[n, k]  (dLoss/dtheta = B^T dLoss/dA).
// A CTA takes 32 columns of one instance, its 16 warps a strided share of the
// rows each, added in warp order: one thread per column ran D_A dependent
// loads deep (D_A = 3840, 8 x 225 columns: 0.3 ms, this 0.02).
constexpr int kBtWarps = 16;
__global__ void __launch_bounds__(32 * kBtWarps) k_bt_times(const double *B, const double *G, double *out, int DA, int d,
                                                             double scale)
{
    __shared__ double part[kBtWarps][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, j = blockIdx.x * 32 + lane;
    const double *Gn = G + (int64_t)blockIdx.y * DA;
    double s = 0.0;
    if (j < d)
        for (int k = w; k < DA; k += kBtWarps) s = fma(B[(int64_t)k * d + j], Gn[k], s);
    part[w][lane] = s;
    __syncthreads();
    if (w == 0 && j < d) {
        s = 0.0;
#pragma unroll
        for (int k = 0; k < kBtWarps; ++k) s += part[k][lane];
        out[(int64_t)blockIdx.y * d + j] = scale * s;
    }
}

template <int DIM, int TESS>
static cudaError_t launch_grad_t(const GradArgs &a, cudaStream_t s)
{
    constexpr int NE = DIM * (DIM + 1);
    size_t smem = (size_t)2 * a.t.nC * NE * sizeof(double);
    auto kern = k_grad_simple<DIM, TESS>;
    if (smem > kSmemOptInAbove) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    int64_t bx = (a.n_per_inst + 127) / 128;
    int64_t cap = (int64_t)num_sms() * 8 / (a.N > 0 ? a.N : 1) + 1;
    if (bx > cap) bx = cap;
    if (bx < 1) bx = 1;
    dim3 grid((unsigned)bx, (unsigned)a.N);
    kern<<<grid, 128, smem, s>>>(a);
    return cudaGetLastError();
}

template <int DIM, int TESS, typename Real>
static cudaError_t launch_grad_ref_t(GradArgs a, cudaStream_t s)
{
    LaunchCfg cfg;
    cfg.block = a.n_per_inst * a.N >= (int64_t)num_sms() * 512 ? 256 : 64;
    // the warps' queues, where they fit beside the tables and two CTAs do not become one
    size_t smem = jump_bytes(a.jump, DIM, a.t.nC, sizeof(Real));
    const size_t with = smem + cfg.block / 32 * kGradQueue * sizeof(int64_t);
    const size_t most = (size_t)max_smem_optin() - 1024;
    a.queue = with <= most && (with <= most / 2 || smem > most / 2);
    if (a.queue) smem = with;
    auto kern = k_grad_ref<DIM, TESS, Real>;
    if (smem > kSmemOptInAbove) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    // one wave: a CTA over it would run alone after all others
    int64_t bx = (a.n_per_inst + cfg.block - 1) / cfg.block;
    const int64_t cap = std::max<int64_t>(1, persistent_grid(kern, cfg, smem) / a.N);
    if (bx > cap) bx = cap;
    dim3 grid((unsigned)bx, (unsigned)a.N);
    kern<<<grid, cfg.block, smem, s>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const int total = a.N * a.t.nC;
    k_level_sums<DIM, TESS><<<(2 * total + 63) / 64, 64, 0, s>>>(a);
    k_frechet_adjoint<DIM><<<(total + 7) / 8, 128, 0, s>>>(a.A, a.gT, a.gA, total, a.dt);
    k_substep_map_adjoint<DIM><<<(total + 127) / 128, 128, 0, s>>>(a.A, a.gS, a.gA, total, a.h_sub);
    return cudaGetLastError();
}

template <typename Real>
static cudaError_t launch_grad_ref_r(const GradArgs &a, cudaStream_t s)
{
    const int dim = a.t.dim, tess = a.t.tess;
    if (dim == 1) return launch_grad_ref_t<1, 2, Real>(a, s);
    if (dim == 2) return tess == 1 ? launch_grad_ref_t<2, 1, Real>(a, s) : launch_grad_ref_t<2, 2, Real>(a, s);
    return tess == 1 ? launch_grad_ref_t<3, 1, Real>(a, s) : launch_grad_ref_t<3, 2, Real>(a, s);
}

cudaError_t launch_grad_ref(const GradArgs &a, int prec, cudaStream_t s)
{
    return prec == PREC_F64 ? launch_grad_ref_r<double>(a, s) : launch_grad_ref_r<float>(a, s);
}

cudaError_t launch_grad_simple(const GradArgs &a, cudaStream_t s)
{
    const int dim = a.t.dim, tess = a.t.tess;
    if (dim == 1) return launch_grad_t<1, 2>(a, s);
    if (dim == 2) return tess == 1 ? launch_grad_t<2, 1>(a, s) : launch_grad_t<2, 2>(a, s);
    return tess == 1 ? launch_grad_t<3, 1>(a, s) : launch_grad_t<3, 2>(a, s);
}

cudaError_t launch_bt_times(const double *B, const double *G, double *out, int DA, int d, int N, double scale,
                            cudaStream_t s)
{
    // N <= 65535 (checked by the caller)
    k_bt_times<<<dim3((unsigned)((d + 31) / 32), (unsigned)N), 32 * kBtWarps, 0, s>>>(B, G, out, DA, d, scale);
    return cudaGetLastError();
}

}  // namespace cpab
