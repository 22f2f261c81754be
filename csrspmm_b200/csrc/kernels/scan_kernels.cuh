// Exclusive scan of int32 counts (row offsets of a conversion, digit offsets of a sort): counts[0..n) into
// offsets[0..n], with the total and the largest count.  scan_tiles: every CTA scans kScanTile counts of its own and
// leaves their sum and maximum; scan_finish: every CTA adds up the sums of the tiles before its own (a few
// thousand values at most) and adds that to its tile.  One tile needs no second launch.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace csrspmm_b200 {

constexpr int kScanThreads = 1024;
constexpr int kScanPer = 8;
constexpr int kScanTile = kScanThreads * kScanPer;

__device__ __forceinline__ long long block_inclusive_scan(long long v, long long* warp_sums)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) warp_sums[warp] = v;
    __syncthreads();
    if (warp == 0) {
        long long w = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        warp_sums[lane] = w;
    }
    __syncthreads();
    if (warp > 0) v += warp_sums[warp - 1];
    return v;
}

__device__ __forceinline__ int block_max(int v, int* warp_max)
{
    v = __reduce_max_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = v;
    __syncthreads();
    int m = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = max(m, warp_max[w]);
    return m;
}

__global__ void __launch_bounds__(kScanThreads) scan_tiles_kernel(const int* __restrict__ counts, long long n, int* __restrict__ offsets,
                                                                  long long* __restrict__ tile_sum, int* __restrict__ tile_max,
                                                                  long long* results)
{
    wait_for_previous_grid();
    release_next_grid();
    __shared__ long long warp_sums[32];
    __shared__ int warp_max[32];
    const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanPer;
    int c[kScanPer];
    long long sum = 0;
    int mx = 0;
    if (base + kScanPer <= n && (reinterpret_cast<uintptr_t>(counts) & 15u) == 0) {
#pragma unroll
        for (int k = 0; k < kScanPer; k += 4) {
            const int4 q = __ldg(reinterpret_cast<const int4*>(counts + base + k));
            c[k] = q.x, c[k + 1] = q.y, c[k + 2] = q.z, c[k + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kScanPer; ++k) c[k] = base + k < n ? counts[base + k] : 0;
    }
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        sum += c[k];
        mx = max(mx, c[k]);
    }
    const long long incl = block_inclusive_scan(sum, warp_sums);
    mx = block_max(mx, warp_max);
    long long run = incl - sum;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        run += c[k];
        if (base + k < n) offsets[base + k + 1] = (int)run;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) offsets[0] = 0;
    if (threadIdx.x == kScanThreads - 1) {
        if (gridDim.x == 1) {
            results[0] = incl;
            results[1] = mx;
        } else {
            tile_sum[blockIdx.x] = incl;
            tile_max[blockIdx.x] = mx;
        }
    }
}

__global__ void __launch_bounds__(kScanThreads) scan_finish_kernel(long long n, int* __restrict__ offsets,
                                                                   const long long* __restrict__ tile_sum,
                                                                   const int* __restrict__ tile_max, long long* results)
{
    wait_for_previous_grid();
    release_next_grid();
    __shared__ long long warp_sums[32];
    __shared__ int warp_max[32];
    __shared__ long long before;
    long long sum = 0;
    int mx = 0;
    const bool last = blockIdx.x == gridDim.x - 1;
    for (int t = threadIdx.x; t < (int)gridDim.x; t += kScanThreads) {
        if (t < (int)blockIdx.x) sum += tile_sum[t];
        if (last) mx = max(mx, tile_max[t]);
    }
    const long long incl = block_inclusive_scan(sum, warp_sums);
    if (last) mx = block_max(mx, warp_max);
    if (threadIdx.x == kScanThreads - 1) {
        before = incl;
        if (last) {
            results[0] = incl + tile_sum[blockIdx.x];
            results[1] = mx;
        }
    }
    __syncthreads();
    const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanPer;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k)
        if (base + k < n) offsets[base + k + 1] = (int)(offsets[base + k + 1] + before);
}

}  // namespace csrspmm_b200
