// cpab_launch.h -- host-side launchers of cpab_kernels.cu / cpab_remap.cu.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "cpab_internal.h"

namespace cpab {

// Launch shape of the integration kernel (chosen by the autotuner).
struct LaunchCfg {
    int block = 256;       // threads per CTA (multiple of 32, <= 256)
    int ctas_per_sm = 32;  // cap on resident CTAs per SM of the persistent grid (occupancy decides below it)
    int grid = 0;          // explicit grid (0 = persistent default)
    int tile_pts = 2048;   // points per CTA tile
    int sort = 0;          // cell-sort the points of each tile
    int max_ctas = 0;      // cap on the CTAs of every persistent launch of the context (0 = none)
};

// Kernels opt in to more than the default 48 KB of shared memory when their
// dynamic size exceeds this (their static shared memory comes on top).
constexpr size_t kSmemOptInAbove = 40 * 1024;

// Static shared memory of k_integrate* (48 bytes), and at most of any kernel that integrates.
constexpr size_t kIntegrateStatic = 48, kStaticSmem = 320;

int num_sms();
int max_smem_optin();

// Points per tile of a uniform 1D exact or a likelihood launch over `total`
// points: the configured tile, or a smaller one (a multiple of 32, at least 64)
// when the launch has too few points to give every SM four tiles -- one
// transform of a few hundred thousand points would otherwise occupy fewer SMs
// than the GPU has.  Per-point results do not depend on the tiling.
inline int small_launch_tile(int64_t total, int tile_pts)
{
    const int64_t want = 4 * (int64_t)num_sms();
    if (total >= want * tile_pts) return tile_pts;
    int64_t t = (total + want - 1) / want;
    t = (t + 31) / 32 * 32;
    if (t < 64) t = 64;
    return (int)(t < tile_pts ? t : tile_pts);
}
// Points per tile of an integration of `total` points by `ctas` persistent
// CTAs: the configured tile where every CTA gets two of them or more; for
// fewer points one or two tiles for every CTA, all of one size (a multiple of
// 32, at least 64), of N ragged instances with room for as many half empty
// last tiles.  A few CTAs with a tile more than the others would set
// the launch's time.  Measured, us, with tiles of 2048 points (uniform: a
// quarter of an SM's share) before and these: FP32 ragged, 16 x 10 k points
// 116 and 87, 200 x 2.7 k 321 and 212, 48 x 28 k 300 and 278; exact scheme, 64 x
// 5 k 308 and 171; 3D, 262144 points 205 and 163; FP64, 64 x 8192 551 and 458.
// From two tiles per CTA on, larger tiles or shares of consecutive points lose
// more to points that cost alike side by side than they save at their ends
// (1024 x 8192: 793 with tiles of 2048, 841 in one share per CTA).
__host__ __device__ inline int balanced_tile(int64_t total, int N, bool ragged, int tile_pts, int ctas)
{
    const int64_t most = (int64_t)ctas * tile_pts;
    if (total >= 2 * most || N < 1) return tile_pts;
    const int64_t slots = total > most ? 2 * (int64_t)ctas : ctas;
    int64_t t;
    if (ragged) {
        const int64_t n = N / 2 < slots / 2 ? slots - N / 2 : slots - slots / 2;
        t = (total + n - 1) / n;
    } else {  // a whole number of tiles per instance
        const int64_t n = slots > N ? slots / N : 1, len = total / N;
        t = (len + n - 1) / n;
    }
    t = (t + 31) / 32 * 32;
    if (t < 64) t = 64;
    return (int)(t < tile_pts ? t : tile_pts);
}
// Room for the warps' queues of an FP32 integration (integrate_jump), `bytes`,
// behind its other shared memory; false, and none, where that fills an SM.
inline bool add_queue(size_t &smem, size_t bytes)
{
    if (smem + bytes + kStaticSmem > (size_t)max_smem_optin()) return false;
    smem += bytes;
    return true;
}
int persistent_grid_impl(const void *kern, const LaunchCfg &cfg, size_t smem);
template <typename K>
inline int persistent_grid(K kern, const LaunchCfg &cfg, size_t smem)
{
    return persistent_grid_impl(reinterpret_cast<const void *>(kern), cfg, smem);
}

cudaError_t launch_integrate(const IntegrateArgs &a, int prec, int scheme, const LaunchCfg &cfg, cudaStream_t s);
cudaError_t launch_integrate_exact1d(const IntegrateArgs &a, int prec, const LaunchCfg &cfg, cudaStream_t s);
size_t exact1d_smem_bytes(int nC, int tile_pts, int sort, int prec);
bool exact1d_uses_intervals(int nC, int prec);
cudaError_t launch_tile_prefix(const int64_t *offsets, int64_t *prefix, int N, int tile_pts, int ctas, cudaStream_t s);
cudaError_t launch_trajectory(const IntegrateArgs &a, int64_t nPts, cudaStream_t s);
cudaError_t launch_cell_idx(const Tess &t, const double *pts, int32_t *out, int64_t n, cudaStream_t s);
cudaError_t launch_calc_v(const Tess &t, const double *A, const double *pts, double *out, int64_t n, cudaStream_t s);
cudaError_t launch_expm(int dim, const double *A, double *signedA, double *T, int64_t n_cells, double dt,
                        double sign, cudaStream_t s);
cudaError_t launch_theta_to_trels(int dim, const double *B, const double *theta, int d, int nC, int N, double dt,
                                  double sign, double *A, double *signedA, double *T, cudaStream_t s);

}  // namespace cpab
