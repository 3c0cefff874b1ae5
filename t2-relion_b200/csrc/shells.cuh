// Shell indices of a padded grid and per-shell sums, shared by the reconstruction kernels.
#pragma once
#include "t2b_internal.cuh"

namespace t2b {
namespace {

// floor(sqrt(r2) / pad) and ROUND(sqrt(r2) / pad) for integers r2 >= 0, pad >= 1: an FP32 estimate
// corrected by exact integer comparisons, the values the FP64 expressions give (sqrt(r2) is exact
// where r2 is a square, and otherwise far more than an FP64 rounding away from a multiple of pad / 2)
__device__ __forceinline__ int shell_floor(int r2, int pad)
{
    int c = (int)(sqrtf((float)r2) / (float)pad);
    while ((long long)(c + 1) * (c + 1) * pad * pad <= r2) ++c;
    while ((long long)c * c * pad * pad > r2) --c;
    return c;
}
__device__ __forceinline__ int shell_round(int r2, int pad)
{
    int c = (int)(sqrtf((float)r2) / (float)pad + 0.5f);
    while ((long long)(2 * c + 1) * (2 * c + 1) * pad * pad <= 4LL * r2) ++c;
    while (c > 0 && (long long)(2 * c - 1) * (2 * c - 1) * pad * pad > 4LL * r2) --c;
    return c;
}

// the MAP term of one voxel (src/backprojector.cpp:1412-1455): inv_tau2[shell] = 1 / (tscale tau2),
// or -1 where tau2 is not positive
__device__ __forceinline__ double map_weight(double w, int r2, int pad, const double* inv_tau2, int minres_map)
{
    const int im = shell_round(r2, pad);
    if (im < minres_map) return w;
    const double it = inv_tau2[im];
    return w + (it >= 0. ? it : (w > 1e-20 ? 1. / (0.001 * w) : 0.));
}

// Sums per shell of a grid: NV values of each voxel inside r2 < rmax2 into acc[NV * shell + v]
// (FP64).  value(n, r2, shell, out) gives the voxel's values; index(r2) its shell.
// Bound by reading the grid's weights (35 MB at 259 x 259 x 130).  A thread takes RUN consecutive x
// of a row: r changes by less than one voxel per step, so a shell of pad voxels holds for several of
// them, and only where the shell changes does the run's sum go to the block's bins in shared memory
// (then one global atomic per bin and block).  With one shared atomic per value and voxel the SSNR
// passes took 100 us each, with global atomics the decentering pass 1.56 ms (8.7 M voxels).
constexpr int RUN = 16;
template <int NV, class Index, class Value>
__device__ __forceinline__ void shell_sums(const Volume& g, int rmax2, int nb, double* sb, double* acc, Index index,
                                           Value value)
{
    for (int i = threadIdx.x; i < NV * nb; i += blockDim.x) sb[i] = 0.;
    __syncthreads();
    const int per = (g.xdim + RUN - 1) / RUN;
    const long long items = (long long)g.zdim * g.ydim * per;
    for (long long it = (long long)blockIdx.x * blockDim.x + threadIdx.x; it < items;
         it += (long long)gridDim.x * blockDim.x) {
        const long long row = it / per;
        const int j0 = (int)(it - row * per) * RUN, j1 = min(g.xdim, j0 + RUN);
        const int y = (int)(row % g.ydim) + g.inity, z = g.ref_dim == 3 ? (int)(row / g.ydim) + g.initz : 0;
        const int yz2 = y * y + z * z;
        if (yz2 + j0 * j0 >= rmax2) continue;
        int cur = -1;
        double s[NV];
        const auto flush = [&] {
            if (cur < 0) return;
#pragma unroll
            for (int v = 0; v < NV; ++v)
                if (s[v] != 0.) atomicAdd(&sb[NV * cur + v], s[v]);
        };
        for (int j = j0; j < j1; ++j) {
            const int r2 = yz2 + j * j;
            if (r2 >= rmax2) break;
            const int sh = index(r2);
            if (sh != cur) {
                flush();
                cur = sh;
#pragma unroll
                for (int v = 0; v < NV; ++v) s[v] = 0.;
            }
            double x[NV];
            value(row * g.xdim + j, r2, sh, x);
#pragma unroll
            for (int v = 0; v < NV; ++v) s[v] += x[v];
        }
        flush();
    }
    __syncthreads();
    for (int i = threadIdx.x; i < NV * nb; i += blockDim.x)
        if (sb[i] != 0.) atomicAdd(&acc[i], sb[i]);
}

}  // namespace
}  // namespace t2b
