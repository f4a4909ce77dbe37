// cfd_reduce.cuh -- deterministic per-case reductions over a tile table.
//
// Every CTA of a tile kernel reduces its values and writes one partial row per tile
// (tile_partial); k_fin, one CTA per case, launched right after, sums that case's rows in a fixed
// order and runs the finaliser. The result does not depend on CTA scheduling or on which
// other cases share the launch, so a case gives the same bits alone and inside any batch.
// Finding the last CTA of a case inside the tile kernel instead (a fence, an arrival
// counter, its answer) held every CTA's registers for two more memory round trips: k_diag 189
// us against 152 + 7 for k_fin, k_correct 220 against 196, on the 256-case sweep.
#pragma once
#include "cfd_common.cuh"

namespace cfd {

constexpr int PSTRIDE = 8;  // doubles per tile partial

// op bit k set => value k is a max, else a sum
template <int NV, unsigned MAXMASK>
__device__ __forceinline__ void block_reduce_mixed(double (&v)[NV], double* smem) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        const bool mx = (MAXMASK >> k) & 1u;
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            double y = __shfl_down_sync(0xffffffffu, x, o);
            x = mx ? fmax(x, y) : x + y;
        }
        if (lane == 0) smem[k * 32 + warp] = x;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) {
            const bool mx = (MAXMASK >> k) & 1u;
            double x = lane < nw ? smem[k * 32 + lane] : (mx ? -1.0e300 : 0.0);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                double y = __shfl_down_sync(0xffffffffu, x, o);
                x = mx ? fmax(x, y) : x + y;
            }
            v[k] = x;
        }
    }
    __syncthreads();
}

// a CTA's partial of its tile: NV values from column `col` of row `tile` (thread 0 writes)
template <int NV, unsigned MAXMASK>
__device__ __forceinline__ void tile_partial(const BatchDev& b, int tile, int col, const double (&v)[NV]) {
    static_assert(NV <= PSTRIDE, "too many reduction values");
    __shared__ double smem[NV * 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        const bool mx = (MAXMASK >> k) & 1u;
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            double y = __shfl_down_sync(0xffffffffu, x, o);
            x = mx ? fmax(x, y) : x + y;
        }
        if (lane == 0) smem[k * 32 + warp] = x;
    }
    __syncthreads();
    if (warp != 0) return;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        const bool mx = (MAXMASK >> k) & 1u;
        double x = lane < nw ? smem[k * 32 + lane] : (mx ? -1.0e300 : 0.0);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            double y = __shfl_down_sync(0xffffffffu, x, o);
            x = mx ? fmax(x, y) : x + y;
        }
        if (lane == 0) b.partial[(long long)tile * PSTRIDE + col + k] = x;
    }
}

// the case's totals of columns 0 .. NV-1, in thread 0
template <int NV, unsigned MAXMASK>
__device__ __forceinline__ void case_total(const BatchDev& b, int tile_begin, int tile_count, double (&v)[NV]) {
    __shared__ double smem[NV * 32];
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = ((MAXMASK >> k) & 1u) ? -1.0e300 : 0.0;
    for (int t = threadIdx.x; t < tile_count; t += blockDim.x) {
        const double* src = b.partial + (long long)(tile_begin + t) * PSTRIDE;
#pragma unroll
        for (int k = 0; k < NV; k++) {
            const double x = src[k];
            v[k] = ((MAXMASK >> k) & 1u) ? fmax(v[k], x) : v[k] + x;
        }
    }
    block_reduce_mixed<NV, MAXMASK>(v, smem);
}

}  // namespace cfd
