// Device-side dense <-> CSR conversion.
//
// The reference converts on one host core (src/host/csr_utils.cpp:70-145: count, allocate, fill
// row by row with fabs(v) > tol, ascending columns, max_row_nnz; and zero-fill + scatter for the
// way back), which is O(M * Kd) and sized with 32-bit products.  These kernels produce the same
// arrays, bit for bit, from a device-resident matrix.
//
// Both directions of the conversion read (or clear) the whole dense matrix and are bound by that.  A row is
// cut into chunks of 512 columns, one warp each, WPR warps of a CTA side by side on one row: every lane has four
// 16-byte loads in flight before anything is tested, where one warp stepping through a row 32 columns at a
// time spent its life waiting (4096 x 4096 at 10 %: 400 us a pass, now 12-15).  An entry's place is the number of kept
// entries before it: ballots inside the chunk, the other warps' totals through shared memory, a running base
// from chunk to chunk, so the order inside a row is ascending.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace csrspmm_b200 {

constexpr int kConvertThreads = 256;
constexpr int kChunkQuads = 4;                      // float4 per lane and chunk
constexpr int kChunkCols = 32 * 4 * kChunkQuads;    // columns per warp and chunk

// Warps side by side on one row: as many as there are chunks, at most the CTA.
inline int convert_warps_per_row(int W)
{
    return W <= kChunkCols ? 1 : (W <= 2 * kChunkCols ? 2 : (W <= 4 * kChunkCols ? 4 : 8));
}

// This lane's 16 entries of the chunk that starts at column c0: quad k, element e is column
//   c0 + 128k + 4*lane + e (VEC: rows start on 16 bytes)   or   c0 + 128k + 32e + lane (any alignment).
// Columns at or beyond W read as 0 and are reported not kept.  (Unsigned: a chunk can end beyond 2^31 - 1.)
template <bool VEC>
__device__ __forceinline__ void load_chunk(const float* __restrict__ src, unsigned c0, unsigned W, int lane, float (&v)[kChunkQuads][4])
{
#pragma unroll
    for (int k = 0; k < kChunkQuads; ++k) {
        if constexpr (VEC) {
            const unsigned c = c0 + 128 * k + 4 * lane;
            if (c + 3 < W) {
                const float4 q = __ldg(reinterpret_cast<const float4*>(src + c));
                v[k][0] = q.x, v[k][1] = q.y, v[k][2] = q.z, v[k][3] = q.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) v[k][e] = c + e < W ? __ldg(src + c + e) : 0.0f;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const unsigned c = c0 + 128 * k + 32 * e + lane;
                v[k][e] = c < W ? __ldg(src + c) : 0.0f;
            }
        }
    }
}

template <bool VEC>
__device__ __forceinline__ unsigned chunk_column(unsigned c0, int k, int e, int lane)
{
    return VEC ? c0 + 128 * k + 4 * lane + e : c0 + 128 * k + 32 * e + lane;
}

// counts[r] = number of entries of row r with |v| > tol
template <bool VEC>
__global__ void __launch_bounds__(kConvertThreads) dense_count_kernel(int H, int W, const float* __restrict__ dense,
                                                                      long long ld, float tol, int wpr, int* __restrict__ counts)
{
    wait_for_previous_grid();
    release_next_grid();
    __shared__ int s_count[kConvertThreads / 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rows_per_cta = (kConvertThreads / 32) / wpr;
    const long long row = (long long)blockIdx.x * rows_per_cta + warp / wpr;
    int count = 0;
    if (row < H) {
        const float* src = dense + row * ld;
        for (unsigned c0 = (warp % wpr) * kChunkCols; c0 < (unsigned)W; c0 += wpr * kChunkCols) {
            float v[kChunkQuads][4];
            load_chunk<VEC>(src, c0, W, lane, v);
#pragma unroll
            for (int k = 0; k < kChunkQuads; ++k)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (fabsf(v[k][e]) > tol && chunk_column<VEC>(c0, k, e, lane) < (unsigned)W) ++count;
        }
    }
    count = __reduce_add_sync(0xffffffffu, count);
    if (wpr == 1) {
        if (lane == 0 && row < H) counts[row] = count;
        return;
    }
    if (lane == 0) s_count[warp] = count;
    __syncthreads();
    if (lane == 0 && warp % wpr == 0 && row < H) {
        for (int w = 1; w < wpr; ++w) count += s_count[warp + w];
        counts[row] = count;
    }
}

template <bool VEC>
__global__ void __launch_bounds__(kConvertThreads) dense_fill_kernel(int H, int W, const float* __restrict__ dense, long long ld,
                                                                     float tol, int wpr, const int* __restrict__ row_ptr,
                                                                     int* __restrict__ col_idx, float* __restrict__ values)
{
    wait_for_previous_grid();
    release_next_grid();
    __shared__ int s_count[2][kConvertThreads / 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rows_per_cta = (kConvertThreads / 32) / wpr;
    const long long row = (long long)blockIdx.x * rows_per_cta + warp / wpr;
    const int first = warp - warp % wpr;  // the row's first warp
    const bool live = row < H;
    const float* src = dense + (live ? row : 0) * ld;
    int base = live ? row_ptr[row] : 0;  // where the current round of chunks starts in the output
    int round = 0;
    for (unsigned r0 = 0; r0 < (unsigned)W; r0 += wpr * kChunkCols, round ^= 1) {
        const unsigned c0 = r0 + (warp % wpr) * kChunkCols;
        float v[kChunkQuads][4];
        unsigned kept[kChunkQuads][4];
        int count = 0;
        if (live && c0 < (unsigned)W) {
            load_chunk<VEC>(src, c0, W, lane, v);
#pragma unroll
            for (int k = 0; k < kChunkQuads; ++k)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    kept[k][e] = __ballot_sync(0xffffffffu, fabsf(v[k][e]) > tol && chunk_column<VEC>(c0, k, e, lane) < (unsigned)W);
                    count += __popc(kept[k][e]);
                }
        }
        int at = base;
        if (wpr > 1) {
            // two sets of totals in turn, so that one barrier a round is enough
            if (lane == 0) s_count[round][warp] = count;
            __syncthreads();
            for (int w = 0; w < wpr; ++w) {
                const int c = s_count[round][first + w];
                if (first + w < warp) at += c;
                base += c;
            }
        } else {
            base += count;
        }
        if (live && c0 < (unsigned)W) {
            const unsigned below = (1u << lane) - 1u;
#pragma unroll
            for (int k = 0; k < kChunkQuads; ++k) {
                if constexpr (VEC) {
                    int mine = at;
#pragma unroll
                    for (int e = 0; e < 4; ++e) mine += __popc(kept[k][e] & below);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if ((kept[k][e] >> lane) & 1u) {
                            col_idx[mine] = (int)chunk_column<VEC>(c0, k, e, lane);
                            values[mine] = v[k][e];
                            ++mine;
                        }
                        at += __popc(kept[k][e]);
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if ((kept[k][e] >> lane) & 1u) {
                            const int mine = at + __popc(kept[k][e] & below);
                            col_idx[mine] = (int)chunk_column<VEC>(c0, k, e, lane);
                            values[mine] = v[k][e];
                        }
                        at += __popc(kept[k][e]);
                    }
                }
            }
        }
    }
}

__global__ void csr_scatter_kernel(int H, int W, const int* __restrict__ row_ptr, const int* __restrict__ col_idx,
                                   const float* __restrict__ values, float* __restrict__ dense, long long ld)
{
    const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= H) return;
    float* dst = dense + row * ld;
    // a repeated column index keeps the last stored value, like the sequential host loop
    const unsigned rs = (unsigned)max(row_ptr[row], 0), re = (unsigned)max(row_ptr[row + 1], 0);
    for (unsigned j0 = rs; j0 < re; j0 += 32) {
        const unsigned j = j0 + lane;
        const int c = j < re ? col_idx[j] : -1;
        const float v = j < re ? values[j] : 0.0f;
        // later lanes win over earlier ones with the same column
        bool last = c >= 0 && c < W;
        for (int o = 1; o < 32; ++o) {
            const int other = __shfl_down_sync(0xffffffffu, c, o);
            if (lane + o < 32 && other == c) last = false;
        }
        if (last) dst[c] = v;
        __syncwarp();
    }
}

}  // namespace csrspmm_b200
