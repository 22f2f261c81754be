// Device-side dense <-> CSR conversion.
//
// The reference converts on one host core (src/host/csr_utils.cpp:70-145: count, allocate, fill
// row by row with fabs(v) > tol, ascending columns, max_row_nnz; and zero-fill + scatter for the
// way back), which is O(M * Kd) and sized with 32-bit products.  These kernels produce the same
// arrays, bit for bit, from a device-resident matrix.
//
// Counting reads the whole dense matrix and is bound by that.  A row is cut into chunks of 512 columns, one warp each,
// WPR warps of a CTA side by side on one row: every lane has four 16-byte loads in flight before anything is tested, where
// one warp stepping through a row 32 columns at a time spent its life waiting (4096 x 4096 at 10 %: 400 us, now 15; asking for
// a warp's next chunk before this one is done with changes nothing).  It leaves one bit per element, a thirty-second of
// the matrix, for the fill.
//
// The fill takes those bits (or makes them again from the matrix) 1024 columns to a warp, one word per lane: the words' counts say
// where a lane's entries go, the kept columns are listed in order in shared memory, and the warp walks the list -- 32
// neighbouring entries of the result at a time, so that columns and values are written in whole sectors and only the
// sectors of the matrix that hold an entry are read.  Reading the matrix again and writing each element from the lane that
// read it was 23 us for 4096 x 4096 at 10 %, this is 10.5.  Both and the scan between, with the host's wait: 51 -> 40 us there,
// 47 -> 37 at 1 %, 55 -> 47 at 30 %, 16 384 x 6000 with 100 per row 210 -> 146.  Without the bits (dense2csr_count and _fill, which the
// C++ API's dense2csr_device calls) the fill alone goes 22 -> 13.4, count and fill 50 -> 43, at 1 % 48 -> 41, at 50 % 69 -> 57, 16 384 x
// 16 384 at 0.5 % 443 -> 338, 100 000 x 64 the same.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace csrspmm_b200 {

constexpr int kConvertThreads = 256;
constexpr int kChunkQuads = 4;                      // float4 per lane and chunk
constexpr int kChunkCols = 32 * 4 * kChunkQuads;    // columns per warp and chunk
constexpr int kSpanCols = 32 * 32;                  // columns per warp and round of the fill

// Warps side by side on one row: as many as there are chunks (spans, for the fill) of `cols` columns, at most the CTA.
inline int convert_warps_per_row(int W, int cols)
{
    return W <= cols ? 1 : (W <= 2LL * cols ? 2 : (W <= 4LL * cols ? 4 : 8));
}

__host__ __device__ inline long long words_per_row(int W) { return ((long long)W + 31) / 32; }

// This lane's 16 entries of the chunk that starts at column c0: quad k, element e is column
//   c0 + 128k + 4*lane + e (VEC: rows start on 16 bytes)   or   c0 + 128k + 32e + lane (any alignment).
// Columns at or beyond W read as NaN, which no tolerance keeps.  (Unsigned: a chunk can end beyond 2^31 - 1.)
template <bool VEC>
__device__ __forceinline__ void load_chunk(const float* __restrict__ src, unsigned c0, unsigned W, int lane, float (&v)[kChunkQuads][4])
{
    const float nan = __int_as_float(0x7fffffff);
#pragma unroll
    for (int k = 0; k < kChunkQuads; ++k) {
        if constexpr (VEC) {
            const unsigned c = c0 + 128 * k + 4 * lane;
            if (c + 3 < W) {
                const float4 q = __ldg(reinterpret_cast<const float4*>(src + c));
                v[k][0] = q.x, v[k][1] = q.y, v[k][2] = q.z, v[k][3] = q.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) v[k][e] = c + e < W ? __ldg(src + c + e) : nan;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const unsigned c = c0 + 128 * k + 32 * e + lane;
                v[k][e] = c < W ? __ldg(src + c) : nan;
            }
        }
    }
}

// Which of a loaded chunk's entries are kept, as 16 words of 32 columns: the lane's word is number chunk_word_of<VEC>(lane) of them,
// 0 where it has none (-1).
template <bool VEC>
__device__ __forceinline__ int chunk_word_of(int lane)
{
    if (VEC) return (lane & 1) ? -1 : ((lane >> 1) & 3) * 4 + (lane >> 3);
    return lane < 4 * kChunkQuads ? lane : -1;
}

template <bool VEC>
__device__ __forceinline__ unsigned chunk_words(const float (&v)[kChunkQuads][4], float tol, int lane)
{
    unsigned mine = 0;
    if constexpr (VEC) {
        // byte k: this lane's four columns of quad k; eight lanes' half-bytes are a word
#pragma unroll
        for (int k = 0; k < kChunkQuads; ++k)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (fabsf(v[k][e]) > tol) mine |= 1u << (8 * k + e);
        static_assert(kChunkQuads == 4, "one byte per quad");
        const unsigned pair = __shfl_xor_sync(0xffffffffu, mine, 1);
        mine = (lane & 1) ? pair | (mine << 4) : mine | (pair << 4);
        // bytes of four pairs of lanes, transposed: pair j gets byte j of each
        const unsigned far = __shfl_xor_sync(0xffffffffu, mine, 4);
        mine = __byte_perm(mine, far, (lane & 4) ? 0x3276 : 0x5410);
        const unsigned near = __shfl_xor_sync(0xffffffffu, mine, 2);
        mine = __byte_perm(mine, near, (lane & 2) ? 0x3715 : 0x6240);
        if (lane & 1) mine = 0;
    } else {
#pragma unroll
        for (int k = 0; k < kChunkQuads; ++k)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const unsigned word = __ballot_sync(0xffffffffu, fabsf(v[k][e]) > tol);
                if (lane == k * 4 + e) mine = word;
            }
    }
    return mine;
}

// counts[r] = number of entries of row r with |v| > tol; mask (may be null): a bit for each of them, words_per_row words a row
template <bool VEC>
__global__ void __launch_bounds__(kConvertThreads) dense_count_kernel(int H, int W, const float* __restrict__ dense, long long ld, float tol,
                                                                      int wpr, int* __restrict__ counts, unsigned* __restrict__ mask)
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
        const int word = chunk_word_of<VEC>(lane);
        for (unsigned c0 = (warp % wpr) * kChunkCols; c0 < (unsigned)W; c0 += wpr * kChunkCols) {
            float v[kChunkQuads][4];
            load_chunk<VEC>(src, c0, W, lane, v);
            const unsigned bits = chunk_words<VEC>(v, tol, lane);
            count += __popc(bits);
            if (mask != nullptr && word >= 0 && c0 / 32 + word < (unsigned)words_per_row(W)) mask[row * words_per_row(W) + c0 / 32 + word] = bits;
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

// mask: the bits that dense_count_kernel left, or null to make them from the matrix.
template <bool VEC>
__global__ void __launch_bounds__(kConvertThreads) dense_fill_kernel(int H, int W, const float* __restrict__ dense, long long ld, float tol,
                                                                     int wpr, const unsigned* __restrict__ mask, const int* __restrict__ row_ptr,
                                                                     int* __restrict__ col_idx, float* __restrict__ values)
{
    wait_for_previous_grid();
    release_next_grid();
    __shared__ int s_count[2][kConvertThreads / 32];
    __shared__ unsigned s_words[kConvertThreads / 32][32];
    __shared__ unsigned short s_list[kConvertThreads / 32][kSpanCols];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rows_per_cta = (kConvertThreads / 32) / wpr;
    const long long row = (long long)blockIdx.x * rows_per_cta + warp / wpr;
    const int first = warp - warp % wpr;  // the row's first warp
    const bool live = row < H;
    const float* src = dense + (live ? row : 0) * ld;
    int base = live ? __ldg(row_ptr + row) : 0;  // where the current round of spans starts in the output
    int round = 0;
    for (unsigned r0 = 0; r0 < (unsigned)W; r0 += wpr * kSpanCols, round ^= 1) {
        const unsigned c0 = r0 + (warp % wpr) * kSpanCols;
        unsigned word = 0;  // of columns c0 + 32 * lane and up
        if (live && c0 < (unsigned)W) {
            if (mask != nullptr) {
                if (c0 / 32 + lane < (unsigned)words_per_row(W)) word = __ldg(mask + row * words_per_row(W) + c0 / 32 + lane);
            } else {
                s_words[warp][lane] = 0;
                __syncwarp();
#pragma unroll
                for (int h = 0; h < kSpanCols / kChunkCols; ++h) {
                    const unsigned at = c0 + h * kChunkCols;
                    if (at < (unsigned)W) {
                        float v[kChunkQuads][4];
                        load_chunk<VEC>(src, at, W, lane, v);
                        const unsigned bits = chunk_words<VEC>(v, tol, lane);
                        if (chunk_word_of<VEC>(lane) >= 0) s_words[warp][h * (kChunkCols / 32) + chunk_word_of<VEC>(lane)] = bits;
                    }
                }
                __syncwarp();
                word = s_words[warp][lane];
            }
        }
        int incl = __popc(word);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const int count = __shfl_sync(0xffffffffu, incl, 31);
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
        // the kept columns in order
        for (int k = incl - __popc(word); word != 0; word &= word - 1) s_list[warp][k++] = (unsigned short)(lane * 32 + __ffs(word) - 1);
        __syncwarp();
        for (int i = lane; i < count; i += 4 * 32) {
            unsigned c[4];
            float v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                c[q] = c0 + (i + q * 32 < count ? s_list[warp][i + q * 32] : 0);
                v[q] = __ldg(src + c[q]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (i + q * 32 < count) {
                    col_idx[at + i + q * 32] = (int)c[q];
                    values[at + i + q * 32] = v[q];
                }
            }
        }
        __syncwarp();  // the list is rewritten by the next round
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
