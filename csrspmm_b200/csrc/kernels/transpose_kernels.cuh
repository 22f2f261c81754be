// CSR of A^T from the CSR of A: a stable radix sort of the entries by column.
//
// No counterpart in the reference, which has no gradients.  The backward product of a matrix that is new at
// each step (a sampled subgraph) needs A^T every time, so the transposition is part of the step: sorting 64-bit
// keys with a general sort, gathering and counting took 520 us for 1 M entries and 65 536 columns.
//
// An entry's key is its column; entries of one column keep their stored order, so the result has ascending
// rows in each column and is the same on every run (no atomics decide a place).  One to four passes over
// digits of up to eight bits, least significant first.  A pass is three steps:
//   count    every CTA counts the digits of its tile of entries -> counts[digit][tile]
//   scan     exclusive scan of the counts in that order (scan_kernels.cuh): where each tile's entries with
//            each digit begin
//   scatter  every CTA puts its tile in digit order in shared memory and writes it out, a run of one digit after
//            the other
// The first pass reads the columns from the matrix and finds each entry's row by a search in row_ptr bounded by
// the rows of the warp's first and last entry; the last writes the arrays of A^T.  Between passes an entry is a
// 4-byte key and an 8-byte (row, value).
//
// What bounds it: launches up to about a million entries, then the writes.  Written straight to their places
// by digits of ten bits (two passes for a million columns) the entries cost one L2 sector write for every 4 or 8 bytes,
// 0.36-0.54 ms per pass over 16.8 M entries and 1.35 ms in all; in runs, with three passes of seven bits, 0.18-0.23 ms per
// pass and 0.77 ms in all.  1 M entries, 65 536 columns: 520 us with torch's sort, 115 written straight, 70 in runs.
#pragma once

#include "common.cuh"

namespace csrspmm_b200 {

constexpr int kTransposeThreads = 256;
constexpr int kTransposeWarps = kTransposeThreads / 32;
constexpr int kMaxDigitBits = 8;
constexpr int kMaxDigits = 1 << kMaxDigitBits;

struct DigitPass {
    int shift, bits, digits;  // digit of key k = (k >> shift) & (digits - 1); digits = 1 << bits
    int tiles;
    long long n;        // entries
};

__device__ __forceinline__ int clamp_col(int c, int Kd) { return (unsigned)c < (unsigned)Kd ? c : min(max(c, 0), Kd - 1); }

// keys: columns of A on the first pass (clamped to [0, Kd)), keys of the pass before on the others
// BY_TILE: counts[tile][digit], for a scatter that adds them up itself.
template <int ITEMS, bool BY_TILE>
__global__ void __launch_bounds__(kTransposeThreads) transpose_count_kernel(const DigitPass ps, const int* __restrict__ keys, int Kd,
                                                                            int* __restrict__ counts)
{
    wait_for_previous_grid();
    release_next_grid();
    __shared__ int hist[kMaxDigits];
    for (int d = threadIdx.x; d < ps.digits; d += kTransposeThreads) hist[d] = 0;
    __syncthreads();
    const long long base = (long long)blockIdx.x * (kTransposeThreads * ITEMS) + threadIdx.x;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const long long j = base + (long long)i * kTransposeThreads;
        if (j < ps.n) atomicAdd(&hist[(clamp_col(__ldg(keys + j), Kd) >> ps.shift) & (ps.digits - 1)], 1);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < ps.digits; d += kTransposeThreads) counts[BY_TILE ? (long long)blockIdx.x * ps.digits + d : (long long)d * ps.tiles + blockIdx.x] = hist[d];
}

// Lanes of the warp with this lane's digit (-1: none), one vote per bit.  Faster here than a match instruction,
// whose time grows with the number of different values in the warp.
__device__ __forceinline__ unsigned same_digit(int d, int bits)
{
    unsigned same = __ballot_sync(0xffffffffu, d >= 0);
    if (d < 0) same = ~same;
    for (int b = 0; b < bits; ++b) {
        const unsigned set = __ballot_sync(0xffffffffu, (d >> b) & 1);
        same &= ((d >> b) & 1) ? set : ~set;
    }
    return same;
}

// Last row r in [lo, hi] with row_ptr[r] <= j (the row of entry j when the offsets ascend)
__device__ __forceinline__ int row_of_entry(const int* __restrict__ row_ptr, int lo, int hi, long long j)
{
    while (lo < hi) {
        const int mid = lo + (hi - lo + 1) / 2;
        if (__ldg(row_ptr + mid) <= j) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// FIRST: entries come from (col_idx, row_ptr, values), else from (keys, pairs).
// LAST: entries go to (t_keys, t_col, t_val), else to (out_keys, out_pairs).
// The same over [0, hi] for two entries at once, one per half warp, sixteen probes a step.
__device__ __forceinline__ int row_of_entry_by_half_warp(const int* __restrict__ row_ptr, int hi, long long j)
{
    const int lane = threadIdx.x & 31;
    int lo = 0;
    while (__any_sync(0xffffffffu, lo < hi)) {
        const int step = (hi - lo + 15) / 16;
        const long long at = (long long)lo + (long long)((lane & 15) + 1) * step;
        const bool below = step > 0 && at <= hi && __ldg(row_ptr + at) <= j;
        const unsigned votes = __ballot_sync(0xffffffffu, below);
        lo += __popc((votes >> (lane & 16)) & 0xffffu) * step;
        hi = step > 0 ? min(hi, lo + step - 1) : lo;
    }
    return lo;
}

// Exclusive scan over the CTA's threads; ends with a barrier behind the last read of warp_sums.
__device__ __forceinline__ int exclusive_over_cta(int v, int* warp_sums)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    int begin = incl - v;
    for (int w = 0; w < warp; ++w) begin += warp_sums[w];
    __syncthreads();
    return begin;
}

// Shared memory of the scatter: the tile's entries in digit order, then the counters.
template <int ITEMS>
struct ScatterSmem {
    static constexpr int TILE = kTransposeThreads * ITEMS;
    int2 pair[TILE];
    int key[TILE];
    int delta[kMaxDigits];   // output position of the tile's entry i in digit order, minus i, per digit
    int start[kMaxDigits];   // where the tile's entries of the digit begin in that order
    int warp_sums[kTransposeWarps];
    unsigned short seen[kTransposeWarps][kMaxDigits];  // the warp's entries of the digit so far, later those of the warps before
};

// SELF: `offsets` holds the counts[tile][digit] and every CTA adds up what lies before its own: up to kSelfTiles tiles that
// costs less than the two scan launches (43 us for 65 K entries and 4096 columns with them).
constexpr int kSelfTiles = 64;

template <int ITEMS, bool FIRST, bool LAST, bool SELF>
__global__ void __launch_bounds__(kTransposeThreads) transpose_scatter_kernel(
    const DigitPass ps, const int* __restrict__ keys, const int2* __restrict__ pairs, const int* __restrict__ row_ptr, int M, int Kd,
    const float* __restrict__ values, const int* __restrict__ offsets, int* __restrict__ out_keys, int2* __restrict__ out_pairs,
    int* __restrict__ t_col, float* __restrict__ t_val)
{
    wait_for_previous_grid();
    release_next_grid();
    extern __shared__ __align__(16) char smem_bytes[];
    ScatterSmem<ITEMS>& s = *reinterpret_cast<ScatterSmem<ITEMS>*>(smem_bytes);
    constexpr int TILE = ScatterSmem<ITEMS>::TILE;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long tile0 = (long long)blockIdx.x * TILE;
    const long long w0 = tile0 + warp * (32 * ITEMS);  // a warp's entries are consecutive
    for (int d = lane; d < ps.digits; d += 32) s.seen[warp][d] = 0;

    int key[ITEMS];
    int2 pair[ITEMS];  // (row, value)
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const long long j = w0 + i * 32 + lane;
        key[i] = j < ps.n ? clamp_col(__ldg(keys + j), Kd) : -1;
        if constexpr (FIRST) pair[i] = make_int2(0, j < ps.n ? __float_as_int(__ldg(values + j)) : 0);
        else pair[i] = j < ps.n ? __ldg(pairs + j) : make_int2(0, 0);
    }
    // where the tile's entries of digit threadIdx.x go (digits <= threads)
    int out0 = 0;
    if constexpr (SELF) {
        int before = 0, all = 0;
        if ((int)threadIdx.x < ps.digits) {
#pragma unroll 8
            for (int t = 0; t < ps.tiles; ++t) {
                const int c = __ldg(offsets + (long long)t * ps.digits + threadIdx.x);
                if (t < (int)blockIdx.x) before += c;
                all += c;
            }
        }
        out0 = exclusive_over_cta(all, s.warp_sums) + before;
    } else if ((int)threadIdx.x < ps.digits) {
        out0 = __ldg(offsets + (long long)threadIdx.x * ps.tiles + blockIdx.x);
    }
    if constexpr (FIRST) {
        if (w0 < ps.n) {
            // rows of the warp's first and last entry; every row that begins between them marks its first entry,
            // and an entry belongs to the last mark at or before it
            const long long w1 = min(w0 + 32 * ITEMS, ps.n);
            const int r = row_of_entry_by_half_warp(row_ptr, M - 1, lane < 16 ? w0 : w1 - 1);
            const int lo = __shfl_sync(0xffffffffu, r, 0);
            const int hi = max(__shfl_sync(0xffffffffu, r, 16), lo);
            if (hi - lo <= 8 * 32 * ITEMS) {
                int* const mark = reinterpret_cast<int*>(s.pair) + warp * (32 * ITEMS);
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) mark[i * 32 + lane] = -1;
                __syncwarp();
                for (int q = lo + 1 + lane; q <= hi; q += 32) {
                    const long long at = (long long)__ldg(row_ptr + q) - w0;
                    if (at >= 0 && at < 32 * ITEMS) atomicMax(mark + at, q);  // empty rows: the last one holds the entry
                }
                __syncwarp();
                int open = lo;  // the row that holds the entry before
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) {
                    const int m = mark[i * 32 + lane];
                    const unsigned marks = __ballot_sync(0xffffffffu, m >= 0) & (0xffffffffu >> (31 - lane));
                    const int got = __shfl_sync(0xffffffffu, m, 31 - __clz(marks | 1u));
                    pair[i].x = marks != 0 ? got : open;
                    open = __shfl_sync(0xffffffffu, pair[i].x, 31);
                }
            } else {  // thousands of empty rows in between: one search per entry
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) pair[i].x = row_of_entry(row_ptr, lo, hi, min(w0 + i * 32 + lane, w1 - 1));
            }
        }
    }
    __syncwarp();

    unsigned short rank[ITEMS];  // among the warp's entries of the same digit, in stored order
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const bool live = key[i] >= 0;
        const int d = live ? (key[i] >> ps.shift) & (ps.digits - 1) : -1;
        const unsigned same = same_digit(d, ps.bits);
        const int before = live ? s.seen[warp][d] : 0;
        rank[i] = (unsigned short)(before + __popc(same & ((1u << lane) - 1u)));
        __syncwarp();
        if (live && lane == __ffs(same) - 1) s.seen[warp][d] = (unsigned short)(before + __popc(same));
        __syncwarp();
    }
    __syncthreads();
    {
        int total = 0;
        if ((int)threadIdx.x < ps.digits) {
#pragma unroll
            for (int w = 0; w < kTransposeWarps; ++w) {
                const int c = s.seen[w][threadIdx.x];
                s.seen[w][threadIdx.x] = (unsigned short)total;
                total += c;
            }
        }
        const int begin = exclusive_over_cta(total, s.warp_sums);
        if ((int)threadIdx.x < ps.digits) {
            s.start[threadIdx.x] = begin;
            s.delta[threadIdx.x] = out0 - begin;
        }
    }
    __syncthreads();

    // the tile in digit order in shared memory
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        if (key[i] < 0) continue;
        const int d = (key[i] >> ps.shift) & (ps.digits - 1);
        rank[i] = (unsigned short)(rank[i] + s.start[d] + s.seen[warp][d]);
        s.key[rank[i]] = key[i];
    }
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
        if (key[i] >= 0) s.pair[rank[i]] = pair[i];
    __syncthreads();

    // and out, runs of one digit side by side
    const int count = (int)min((long long)TILE, ps.n - tile0);
    for (int i = threadIdx.x; i < count; i += kTransposeThreads) {
        const int k = s.key[i];
        const int2 p = s.pair[i];
        const int at = s.delta[(k >> ps.shift) & (ps.digits - 1)] + i;
        out_keys[at] = k;
        if constexpr (LAST) {
            t_col[at] = p.x;
            t_val[at] = __int_as_float(p.y);
        } else {
            out_pairs[at] = p;
        }
    }
}

// Row offsets from the sorted keys: position p begins every column above the key before it, up to its own.  Four
// positions per thread; a long run of empty columns is written by the whole warp.
__global__ void __launch_bounds__(256) transpose_row_ptr_kernel(int Kd, int n, const int* __restrict__ keys, int* __restrict__ t_row_ptr)
{
    wait_for_previous_grid();
    release_next_grid();
    const long long pos0 = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
    const int lane = threadIdx.x & 31;
    int k[4];
    if (pos0 + 3 < n) {
        const int4 q = __ldg(reinterpret_cast<const int4*>(keys + pos0));
        k[0] = q.x, k[1] = q.y, k[2] = q.z, k[3] = q.w;
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) k[e] = pos0 + e < n ? __ldg(keys + pos0 + e) : Kd;
    }
    int before = __shfl_up_sync(0xffffffffu, k[3], 1);
    if (lane == 0) before = pos0 == 0 ? -1 : (pos0 <= n ? __ldg(keys + pos0 - 1) : Kd);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int pos = (int)(pos0 + e);
        const int from = before + 1, to = pos0 + e <= n ? k[e] : -1;  // columns [from, to] begin at pos
        before = k[e];
        const bool many = to - from >= 16;
        if (!many)
            for (int c = from; c <= to; ++c) t_row_ptr[c] = pos;
        for (unsigned left = __ballot_sync(0xffffffffu, many); left != 0; left &= left - 1) {
            const int src = __ffs(left) - 1;
            const int f = __shfl_sync(0xffffffffu, from, src), t = __shfl_sync(0xffffffffu, to, src), p = __shfl_sync(0xffffffffu, pos, src);
            for (int c = f + lane; c <= t; c += 32) t_row_ptr[c] = p;
        }
    }
}

// The same by one search per column, for matrices with fewer entries than columns.
// t_row_ptr[c] = first position whose key is c or more
__global__ void __launch_bounds__(256) transpose_row_ptr_search_kernel(int Kd, int n, const int* __restrict__ keys, int* __restrict__ t_row_ptr)
{
    wait_for_previous_grid();
    release_next_grid();
    const int c = blockIdx.x * 256 + threadIdx.x;
    if (c > Kd) return;
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = lo + (hi - lo) / 2;
        if (__ldg(keys + mid) < c) lo = mid + 1;
        else hi = mid;
    }
    t_row_ptr[c] = lo;
}

}  // namespace csrspmm_b200
