// Deterministic FP64 grid reduction: every block sums its threads' values
// (warp shuffles, then the warps in order), writes one partial, and the last
// block to finish sums the partials in block order.  The result does not
// depend on which blocks ran when, unlike one atomic add per warp, and only
// one atomic per block touches a shared address.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace lbm {

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums (a, b) over the grid into out[0], out[1].  scratch: 2 doubles per
// block, then a u32 ticket that starts at zero (the last block resets it).
// Every thread of every block calls this once, with NT threads per block.
template <int NT>
__device__ __forceinline__ void grid_sum2(double a, double b, double *scratch, double *out) {
    __shared__ double sh[NT / 32][2];
    __shared__ bool last;
    uint32_t *ticket = reinterpret_cast<uint32_t *>(scratch + 2 * (size_t)gridDim.x);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    a = warp_sum_d(a);
    b = warp_sum_d(b);
    if (lane == 0) { sh[warp][0] = a; sh[warp][1] = b; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double sa = 0, sb = 0;
        for (int w = 0; w < NT / 32; w++) { sa += sh[w][0]; sb += sh[w][1]; }
        scratch[2 * blockIdx.x] = sa;
        scratch[2 * blockIdx.x + 1] = sb;
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double sa = 0, sb = 0;
    for (uint32_t k = threadIdx.x; k < gridDim.x; k += NT) {
        sa += __ldcg(&scratch[2 * k]);
        sb += __ldcg(&scratch[2 * k + 1]);
    }
    sa = warp_sum_d(sa);
    sb = warp_sum_d(sb);
    __syncthreads();
    if (lane == 0) { sh[warp][0] = sa; sh[warp][1] = sb; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ta = 0, tb = 0;
        for (int w = 0; w < NT / 32; w++) { ta += sh[w][0]; tb += sh[w][1]; }
        out[0] = ta;
        out[1] = tb;
        *ticket = 0u;
    }
}

// The force and moment of each step of a batch from the wall kernel's block
// partials (6 doubles, 8 apart; nblk blocks per step, the steps one after
// another): block k sums step slot0 + k in block order into hist.  Left to one
// launch per batch: summed by the wall kernel's last block, every step paid
// for the fence, the counter and the second pass (3-5 us) before the bulk.
template <int NT>
__global__ void __launch_bounds__(NT) k_force_sum(const double *__restrict__ partials, uint32_t nblk, double *__restrict__ hist, uint32_t slot0) {
    __shared__ double sh[NT / 32][6];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double *part = partials + (uint64_t)blockIdx.x * nblk * 8;
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (uint32_t b = threadIdx.x; b < nblk; b += NT)
        for (int j = 0; j < 6; j++) acc[j] += part[(uint64_t)b * 8 + j];
#pragma unroll
    for (int j = 0; j < 6; j++) acc[j] = warp_sum_d(acc[j]);
    if (lane == 0)
        for (int j = 0; j < 6; j++) sh[warp][j] = acc[j];
    __syncthreads();
    if (threadIdx.x < 6) {
        double t = 0;
        for (int w = 0; w < NT / 32; w++) t += sh[w][threadIdx.x];
        hist[(uint64_t)(slot0 + blockIdx.x) * 8 + threadIdx.x] = t;
    }
}

// A block's 6 sums into its partial (warp shuffles, then the warps in order).
template <int NT>
__device__ __forceinline__ void block_partial6(double *v, double *out) {
    __shared__ double sh[NT / 32][6];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < 6; j++) v[j] = warp_sum_d(v[j]);
    if (lane == 0)
        for (int j = 0; j < 6; j++) sh[warp][j] = v[j];
    __syncthreads();
    if (threadIdx.x < 6) {
        double t = 0;
        for (int w = 0; w < NT / 32; w++) t += sh[w][threadIdx.x];
        out[threadIdx.x] = t;
    }
}

// steps whose partials are kept before they are summed: as many of `most` as
// 16 MB hold
inline uint32_t force_ring(uint64_t nblk, uint32_t most) {
    const uint64_t n = (16ull << 20) / (nblk * 64);
    return n < 1 ? 1u : (n > most ? most : (uint32_t)n);
}

}  // namespace lbm
