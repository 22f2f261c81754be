// CSR of A^T from the CSR of A: a stable radix sort of the entries by column.
//
// No counterpart in the reference, which has no gradients.  The backward product of a matrix that is new at
// each step (a sampled subgraph) needs A^T every time, so the transposition is part of the step: sorting 64-bit
// keys with a general sort, gathering and counting took 520 us for 1 M entries and 65 536 columns.
//
// An entry's key is its column; entries of one column keep their stored order, so the result has ascending
// rows in each column and is the same on every run (no atomics decide a place).  Matrices whose buckets are small enough
// for a CTA each go through buckets (second half of this file): up to 2^19 columns, and up to 4096 entries for each of at most
// 1024 runs of columns, so 4.2 million entries with 1024 columns and more, 262 144 with 64.  The others take one to four passes
// over digits of up to eight bits, least significant first.  A pass is three steps:
//   count    every CTA counts the digits of its tile of entries -> counts[digit][tile]
//   scan     exclusive scan of the counts in that order (scan_kernels.cuh): where each tile's entries with
//            each digit begin
//   scatter  every CTA puts its tile in digit order in shared memory and writes it out, a run of one digit after
//            the other
// The first pass reads the columns from the matrix and finds each entry's row by a search in row_ptr bounded by
// the rows of the warp's first and last entry; the last writes the arrays of A^T.  Between passes an entry is a
// 4-byte key and an 8-byte (row, value).
//
// What bounds it: the writes.  Written straight to their places
// by digits of ten bits (two passes for a million columns) the entries cost one L2 sector write for every 4 or 8 bytes,
// 0.36-0.54 ms per pass over 16.8 M entries and 1.35 ms in all; in runs, with three passes of seven bits, 0.18-0.23 ms per
// pass and 0.77 ms in all.
#pragma once

#include "common.cuh"

namespace csrspmm_b200 {

constexpr int kTransposeThreads = 256;
constexpr int kTransposeWarps = kTransposeThreads / 32;
constexpr int kMaxDigitBits = 8;
constexpr int kMaxDigits = 1 << kMaxDigitBits;

struct DigitPass {
    int shift, digits;  // digit of key k = (k >> shift) & (digits - 1); digits a power of two
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

// Rows of the 32 * ITEMS consecutive entries that begin at w0 and end before w1 (at most 32 * ITEMS of them), entry w0 + i * 32 + lane in
// row[i]; one warp.  The first lies in row lo, the last in row hi or before; every row that begins between them marks its
// first entry, and an entry belongs to the last mark at or before it.  mark: 32 * ITEMS words of shared memory.
template <int ITEMS>
__device__ __forceinline__ void rows_of_entries(const int* __restrict__ row_ptr, int lo, int hi, long long w0, long long w1, int* mark,
                                                int (&row)[ITEMS])
{
    const int lane = threadIdx.x & 31;
    if (hi - lo <= 8 * 32 * ITEMS) {
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
            row[i] = marks != 0 ? got : open;
            open = __shfl_sync(0xffffffffu, row[i], 31);
        }
    } else {  // thousands of empty rows in between: one search per entry
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) row[i] = row_of_entry(row_ptr, lo, hi, min(w0 + i * 32 + lane, w1 - 1));
    }
}

// rank[i] of digit[i] (-1: no entry) among the warp's entries of that digit, in stored order (i, then lane).  seen: the warp's
// counters, one per digit; mask: as many words of shared memory of the warp's own.  Items from `count` on are nobody's (the same
// for the whole warp).  Every lane sets its bit in its digit's word, and the bits say which lanes share the digit: two
// instructions of the load-store unit, where one vote per bit of the digit is four instructions each on the integer pipe (256 items
// of 32 warps on one SM, 512 digits: 4800 cycles, 9100 with votes, 14 600 with match instructions).
template <int ITEMS>
__device__ __forceinline__ void rank_in_warp(const int (&digit)[ITEMS], int count, int digits, unsigned short* seen, unsigned* mask,
                                             unsigned short (&rank)[ITEMS])
{
    const int lane = threadIdx.x & 31;
    for (int d = lane; d < digits; d += 32) {
        seen[d] = 0;
        mask[d] = 0;
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        if (i >= count) break;
        const bool live = digit[i] >= 0;
        if (live) atomicOr(mask + digit[i], 1u << lane);
        __syncwarp();
        const unsigned same = live ? mask[digit[i]] : 0u;
        const int before = live ? seen[digit[i]] : 0;
        rank[i] = (unsigned short)(before + __popc(same & ((1u << lane) - 1u)));
        __syncwarp();
        if (live && (same >> lane) == 1u) {  // the last of them
            seen[digit[i]] = (unsigned short)(before + __popc(same));
            mask[digit[i]] = 0;
        }
        __syncwarp();
    }
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
    int sum = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0;  // every warp scans the warps' sums for itself
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += t;
    }
    const int before = __shfl_sync(0xffffffffu, sum, max(warp - 1, 0));
    __syncthreads();
    return incl - v + (warp > 0 ? before : 0);
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

// FIRST: entries come from (col_idx, row_ptr, values), else from (keys, pairs).
// LAST: entries go to (out_keys, t_col, t_val), else to (out_keys, out_pairs).
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
    // words of the warp's own, until the entries go to s.pair
    unsigned* const words = reinterpret_cast<unsigned*>(s.pair) + warp * (32 * ITEMS);
    static_assert(32 * ITEMS >= kMaxDigits, "one word per digit");

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
            int row[ITEMS];
            const long long w1 = min(w0 + 32 * ITEMS, ps.n);
            const int r = row_of_entry_by_half_warp(row_ptr, M - 1, lane < 16 ? w0 : w1 - 1);
            const int lo = __shfl_sync(0xffffffffu, r, 0);
            rows_of_entries<ITEMS>(row_ptr, lo, max(__shfl_sync(0xffffffffu, r, 16), lo), w0, w1, reinterpret_cast<int*>(words), row);
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) pair[i].x = row[i];
        }
    }
    __syncwarp();

    int digit[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) digit[i] = key[i] < 0 ? -1 : (key[i] >> ps.shift) & (ps.digits - 1);
    unsigned short rank[ITEMS];
    rank_in_warp<ITEMS>(digit, ITEMS, ps.digits, s.seen[warp], words, rank);
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

// ---- two steps through buckets ------------------------------------------------------------------------
//
// Up to some four million entries the passes above are mostly launches and their ramps: nine of them for 1 M entries and 65 536
// columns, 68 us.  Here the most significant bits of the column come first: the entries are put into 2^high_bits buckets of about
// 2000 entries, stably, and then one CTA takes a bucket whole, sorts it by the remaining bits in shared memory and
// writes a contiguous piece of A^T -- without counts, a scan or a second scattered write, and the row offsets of the
// bucket's columns come out of its own counters.
//   count    counts[tile][bucket], tiles of 1024 threads, and the row of each warp's first entry
//   offsets  for each bucket, what the tiles before hold of it; its total
//   scatter  the tile in bucket order, written out run by run
//   sort     one CTA per bucket
// A bucket of more entries than a CTA holds (a hub column) is cut into chunks, a CTA each, whose digits a kernel of
// its own counts before the sort; without such a bucket that kernel has nothing to do (2.5 us).  Up to one chunk of entries there is
// none, so two launches; up to one tile three (nothing to count across tiles), else five.
//
// Measured against the passes (us): 1 M entries and 65 536 columns 68 -> 31, 5 % of them in one column 69 -> 38, all in one 68 -> 54,
// columns by a power law 67 -> 49; 250 000 entries 50 -> 20; 600 000 and 200 000 columns 80 -> 27; 2 M and 262 144 columns 150 ->
// 54; 3.9 M 207 -> 108; 1500 entries 21 -> 10.  Of the 31 us the scatter is 13 (one CTA of 1024 threads per SM, whose
// phases wait for one another: loads 4000 cycles, ranks 4800, staging 4000, writing 4900) and the sort 10.

constexpr int kBucketThreads = 1024;
constexpr int kMaxBucketBits = 10;  // buckets <= kBucketThreads
constexpr int kMaxColumnBits = 9;   // columns per bucket <= threads of the sort
constexpr int kMaxBuckets = 1 << kMaxBucketBits;
constexpr int kMaxBucketColumns = 1 << kMaxColumnBits;
constexpr int kBucketItems = 8;
constexpr int kMaxBucketTiles = 4 * kSms;  // four waves of the scatter; 32 warps of the offsets kernel with 19 each

struct BucketPass {
    int high_bits, low_bits;  // column = bucket << low_bits | digit
    int tiles;
    int items;    // entries per thread and tile, at most kBucketItems
    int chunk;    // entries a CTA of the sort holds
    int n;        // entries
    int large;    // CTAs of the sort for chunks of larger buckets
};

// first_row[w]: row of the first entry of the w-th warp's entries (32 * ps.items each), and behind the last one that of the last entry
__global__ void __launch_bounds__(kBucketThreads) transpose_bucket_count_kernel(const BucketPass ps, const int* __restrict__ keys,
                                                                                const int* __restrict__ row_ptr, int M, int Kd,
                                                                                int* __restrict__ counts, int* __restrict__ first_row)
{
    wait_for_previous_grid();
    release_next_grid();
    __shared__ int hist[kMaxBuckets];
    const int buckets = 1 << ps.high_bits;
    if ((int)threadIdx.x < buckets) hist[threadIdx.x] = 0;
    int key[kBucketItems];
    const int base = blockIdx.x * (kBucketThreads * ps.items) + threadIdx.x;
    const int end = min((blockIdx.x + 1) * (kBucketThreads * ps.items), ps.n);
#pragma unroll
    for (int i = 0; i < kBucketItems; ++i) key[i] = base + i * kBucketThreads < end ? __ldg(keys + base + i * kBucketThreads) : 0;
    const int w = blockIdx.x * (kBucketThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int w0 = w * (32 * ps.items);
    if (w0 < ps.n) {
        const bool last = w0 + 32 * ps.items >= ps.n;
        const int r = row_of_entry_by_half_warp(row_ptr, M - 1, lane < 16 ? w0 : ps.n - 1);
        if (lane == 0) first_row[w] = r;
        if (lane == 16 && last) first_row[w + 1] = r;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kBucketItems; ++i)
        if (base + i * kBucketThreads < end) atomicAdd(&hist[clamp_col(key[i], Kd) >> ps.low_bits], 1);
    __syncthreads();
    if ((int)threadIdx.x < buckets) counts[blockIdx.x * buckets + threadIdx.x] = hist[threadIdx.x];
}

// counts[tile][bucket] -> the bucket's entries in the tiles before, and total[bucket].  A CTA takes 32 buckets, a warp a run of tiles.
__global__ void __launch_bounds__(1024) transpose_bucket_offsets_kernel(const BucketPass ps, int* __restrict__ counts, int* __restrict__ total)
{
    wait_for_previous_grid();
    release_next_grid();
    __shared__ int sums[32][33];
    constexpr int RUN = (kMaxBucketTiles + 31) / 32;
    const int buckets = 1 << ps.high_bits, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bucket = blockIdx.x * 32 + lane;
    const int run = (ps.tiles + 31) / 32, t0 = warp * run;
    int c[RUN], sum = 0;
#pragma unroll
    for (int k = 0; k < RUN; ++k) {
        c[k] = k < run && t0 + k < ps.tiles && bucket < buckets ? counts[(t0 + k) * buckets + bucket] : 0;
        sum += c[k];
    }
    sums[warp][lane] = sum;
    __syncthreads();
    int v = sums[lane][warp];  // warp: bucket, lane: run
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    if (lane == 31 && blockIdx.x * 32 + warp < buckets) total[blockIdx.x * 32 + warp] = incl;
    __syncthreads();
    sums[lane][warp] = incl - v;
    __syncthreads();
    int before = sums[warp][lane];
#pragma unroll
    for (int k = 0; k < RUN; ++k) {
        if (k < run && t0 + k < ps.tiles && bucket < buckets) counts[(t0 + k) * buckets + bucket] = before;
        before += c[k];
    }
}

// Shared memory of the scatter.  The first part holds the tile in bucket order; before that, words of each warp's own.
struct BucketSmem {
    static constexpr int TILE = kBucketThreads * kBucketItems, WARPS = kBucketThreads / 32;
    int2* pair;
    int* key;
    int* delta;
    int* start;
    int* warp_sums;
    unsigned short* seen;  // [WARPS][buckets]
    unsigned* words;       // [WARPS][words_per_warp]
    static __host__ __device__ int words_per_warp(int buckets) { return buckets > 32 * kBucketItems ? buckets : 32 * kBucketItems; }
    static __host__ __device__ int first_part(int buckets)
    {
        const int words = WARPS * words_per_warp(buckets) * 4;
        return words > TILE * 12 ? words : TILE * 12;
    }
    static __host__ __device__ int bytes(int buckets) { return first_part(buckets) + buckets * 8 + 128 + WARPS * buckets * 2; }
    __device__ BucketSmem(char* at, int buckets)
        : pair(reinterpret_cast<int2*>(at)), key(reinterpret_cast<int*>(at + TILE * 8)), delta(reinterpret_cast<int*>(at + first_part(buckets))),
          start(delta + buckets), warp_sums(start + buckets), seen(reinterpret_cast<unsigned short*>(warp_sums + 32)),
          words(reinterpret_cast<unsigned*>(at))
    {
    }
};

// first_entry[b], first_slot[b], b = 0 .. buckets: where bucket b begins in (out_low, out_pairs), and the number of its first chunk
// among the chunks of buckets with more than one.  One tile: without counts, totals and first_row.
__global__ void __launch_bounds__(kBucketThreads, 1) transpose_bucket_scatter_kernel(
    const BucketPass ps, const int* __restrict__ col_idx, const int* __restrict__ row_ptr, int M, int Kd, const float* __restrict__ values,
    const int* __restrict__ counts, const int* __restrict__ totals, const int* __restrict__ first_row, unsigned short* __restrict__ out_low,
    int2* __restrict__ out_pairs, int* __restrict__ first_entry, int* __restrict__ first_slot)
{
    wait_for_previous_grid();
    release_next_grid();
    extern __shared__ __align__(16) char smem_bytes[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int buckets = 1 << ps.high_bits;
    const BucketSmem s(smem_bytes, buckets);
    unsigned* const words = s.words + warp * s.words_per_warp(buckets);
    unsigned short* const seen = s.seen + warp * buckets;
    constexpr int ITEMS = kBucketItems;
    const int tile0 = blockIdx.x * (kBucketThreads * ps.items);
    // a warp's entries are consecutive
    const int w0 = tile0 + warp * (32 * ps.items), w1 = min(w0 + 32 * ps.items, ps.n);

    int key[ITEMS], row[ITEMS];
    float value[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int j = w0 + i * 32 + lane;
        key[i] = j < w1 ? __ldg(col_idx + j) : 0;
        value[i] = j < w1 ? __ldg(values + j) : 0.0f;
    }
    int all = 0, before = 0;  // bucket tid: its entries, those in the tiles before this one
    if (ps.tiles > 1 && tid < buckets) {
        all = __ldg(totals + tid);
        before = __ldg(counts + blockIdx.x * buckets + tid);
    }
    if (w0 < w1) {
        int lo, hi;
        if (ps.tiles > 1) {
            lo = __ldg(first_row + blockIdx.x * BucketSmem::WARPS + warp);
            hi = __ldg(first_row + blockIdx.x * BucketSmem::WARPS + warp + 1);
        } else {
            const int r = row_of_entry_by_half_warp(row_ptr, M - 1, lane < 16 ? w0 : w1 - 1);
            lo = __shfl_sync(0xffffffffu, r, 0);
            hi = __shfl_sync(0xffffffffu, r, 16);
        }
        rows_of_entries<ITEMS>(row_ptr, lo, max(hi, lo), w0, w1, reinterpret_cast<int*>(words), row);
        __syncwarp();
    }
    int digit[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        key[i] = w0 + i * 32 + lane < w1 ? clamp_col(key[i], Kd) : -1;
        digit[i] = key[i] >> ps.low_bits;
    }
    unsigned short rank[ITEMS];
    rank_in_warp<ITEMS>(digit, ps.items, buckets, seen, words, rank);
    __syncthreads();
    int total = 0;
    if (tid < buckets) {
#pragma unroll
        for (int w = 0; w < BucketSmem::WARPS; ++w) {
            const int c = s.seen[w * buckets + tid];
            s.seen[w * buckets + tid] = (unsigned short)total;
            total += c;
        }
        if (ps.tiles == 1) all = total;
    }
    const int bucket0 = exclusive_over_cta(all, s.warp_sums);
    const int begin = exclusive_over_cta(total, s.warp_sums);
    if (tid < buckets) {
        s.start[tid] = begin;
        s.delta[tid] = bucket0 + before - begin;
    }
    if (blockIdx.x == 0) {
        const int slots = all > ps.chunk ? (all + ps.chunk - 1) / ps.chunk : 0;
        const int slot0 = exclusive_over_cta(slots, s.warp_sums);
        if (tid < buckets) {
            first_entry[tid] = bucket0;
            first_slot[tid] = slot0;
        }
        if (tid == buckets - 1) {
            first_entry[buckets] = ps.n;
            first_slot[buckets] = slot0 + slots;
        }
    }
    __syncthreads();

    // the tile in bucket order in shared memory
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        if (key[i] < 0) continue;
        const int at = rank[i] + s.start[digit[i]] + seen[digit[i]];
        s.key[at] = key[i];
        s.pair[at] = make_int2(row[i], __float_as_int(value[i]));
    }
    __syncthreads();

    // and out, runs of one bucket side by side
    const int count = min(kBucketThreads * ps.items, ps.n - tile0);
#pragma unroll 4
    for (int i = tid; i < count; i += kBucketThreads) {
        const int k = s.key[i];
        const int at = s.delta[k >> ps.low_bits] + i;
        out_low[at] = (unsigned short)(k & ((1 << ps.low_bits) - 1));
        out_pairs[at] = s.pair[i];
    }
}

// Chunk `slot` of the buckets with more than one chunk: its bucket and its entries [begin, end).
__device__ __forceinline__ int bucket_of_slot(const BucketPass& ps, const int* __restrict__ first_entry, const int* __restrict__ first_slot,
                                              int slot, int& begin, int& end)
{
    int lo = 0, hi = (1 << ps.high_bits) - 1;  // the last bucket whose first slot is not beyond (those without slots share the next one's)
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(first_slot + mid) <= slot) lo = mid;
        else hi = mid - 1;
    }
    begin = __ldg(first_entry + lo) + (slot - __ldg(first_slot + lo)) * ps.chunk;
    end = min(begin + ps.chunk, __ldg(first_entry + lo + 1));
    return lo;
}

// chunk_counts[slot][digit] of every chunk of a bucket with more than one
__global__ void __launch_bounds__(512) transpose_chunk_count_kernel(const BucketPass ps, const unsigned short* __restrict__ low,
                                                                    const int* __restrict__ first_entry, const int* __restrict__ first_slot,
                                                                    int* __restrict__ chunk_counts)
{
    wait_for_previous_grid();
    release_next_grid();
    __shared__ int hist[kMaxBucketColumns];
    const int slots = __ldg(first_slot + (1 << ps.high_bits)), digits = 1 << ps.low_bits;
    for (int slot = blockIdx.x; slot < slots; slot += gridDim.x) {
        int begin, end;
        bucket_of_slot(ps, first_entry, first_slot, slot, begin, end);
        if ((int)threadIdx.x < digits) hist[threadIdx.x] = 0;
        __syncthreads();
        for (int j = begin + threadIdx.x; j < end; j += 512) atomicAdd(&hist[__ldg(low + j)], 1);
        __syncthreads();
        if ((int)threadIdx.x < digits) chunk_counts[(slot << ps.low_bits) + threadIdx.x] = hist[threadIdx.x];
        __syncthreads();
    }
}

template <int THREADS, int ITEMS>
struct BucketSortSmem {
    static constexpr int CHUNK = THREADS * ITEMS, WARPS = THREADS / 32;
    static_assert(CHUNK * 2 >= THREADS * (int)sizeof(int2), "partial sums in `words`");
    int2* pair;              // [CHUNK], as they come
    unsigned* words;         // [WARPS][digits], the warps' own
    unsigned short* source;  // [CHUNK], in the same place later: which of the pairs is entry i in column order
    int* start;              // [digits]
    int* warp_sums;          // [32]
    unsigned short* seen;    // [WARPS][digits]
    static __host__ __device__ int bytes(int digits)
    {
        return CHUNK * 8 + words_bytes(digits) + digits * 4 + 128 + WARPS * digits * 2;
    }
    static __host__ __device__ int words_bytes(int digits) { return WARPS * digits * 4 > CHUNK * 2 ? WARPS * digits * 4 : CHUNK * 2; }
    __device__ BucketSortSmem(char* at, int digits)
        : pair(reinterpret_cast<int2*>(at)), words(reinterpret_cast<unsigned*>(at + CHUNK * 8)), source(reinterpret_cast<unsigned short*>(words)),
          start(reinterpret_cast<int*>(at + CHUNK * 8 + words_bytes(digits))), warp_sums(start + digits),
          seen(reinterpret_cast<unsigned short*>(warp_sums + 32))
    {
    }
};

// Entries [begin, end) of `bucket` (at most a chunk) in column order into A^T.  LARGE: they are chunk `slot` of a bucket with more
// than one, [slot0, slot1).
template <int THREADS, int ITEMS, bool LARGE>
__device__ __forceinline__ void sort_chunk(const BucketPass& ps, const BucketSortSmem<THREADS, ITEMS>& s, int bucket, int begin, int end,
                                           int bucket0, int slot, int slot0, int slot1, int Kd, const unsigned short* __restrict__ low,
                                           const int2* __restrict__ pairs, const int* __restrict__ chunk_counts, int* __restrict__ t_row_ptr,
                                           int* __restrict__ t_col, float* __restrict__ t_val)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, digits = 1 << ps.low_bits;
    unsigned short* const seen = s.seen + warp * digits;
    const int n = end - begin;
    // a warp's entries are consecutive: the same whole number of 32 for every warp
    const int per_warp = (n + THREADS - 1) / THREADS;  // in units of 32, at most ITEMS
    const int w0 = warp * 32 * per_warp;
    int key[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int j = w0 + i * 32 + lane;
        key[i] = i < per_warp && j < n ? (int)__ldg(low + begin + j) : -1;
    }
    for (int j = tid; j < n; j += THREADS)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(s.pair + j)), "l"(pairs + begin + j) : "memory");
    async_commit();
    // where the digits of a chunk go: behind the whole bucket's entries of the digits below and those of the chunks before
    int before = 0, all = 0;
    if constexpr (LARGE) {
        const int step = THREADS >> ps.low_bits;  // threads of a digit share the chunks
#pragma unroll 8
        for (int q = slot0 + (tid >> ps.low_bits); q < slot1; q += step) {
            const int c = __ldg(chunk_counts + (q << ps.low_bits) + (tid & (digits - 1)));
            if (q < slot) before += c;
            all += c;
        }
        int2* const part = reinterpret_cast<int2*>(s.words);
        part[tid] = make_int2(before, all);
        __syncthreads();
        before = all = 0;
        for (int q = tid; q < THREADS && tid < digits; q += digits) {
            before += part[q].x;
            all += part[q].y;
        }
        __syncthreads();
    }
    unsigned short rank[ITEMS];
    rank_in_warp<ITEMS>(key, per_warp, digits, seen, s.words + warp * digits, rank);
    __syncthreads();
    int total = 0;
    if (tid < digits) {
#pragma unroll
        for (int w = 0; w < THREADS / 32; ++w) {
            const int c = s.seen[w * digits + tid];
            s.seen[w * digits + tid] = (unsigned short)total;
            total += c;
        }
    }
    const int in_bucket = exclusive_over_cta(LARGE ? all : total, s.warp_sums);
    if (tid < digits) {
        s.start[tid] = LARGE ? bucket0 + in_bucket + before : in_bucket;
        const int column = (bucket << ps.low_bits) + tid;
        if (column < Kd && begin == bucket0) t_row_ptr[column] = bucket0 + in_bucket;
    }
    if constexpr (LARGE) {  // its digits do not lie side by side in A^T: straight to their places
        async_wait<0>();
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (key[i] < 0) continue;
            const int at = s.start[key[i]] + rank[i] + seen[key[i]];
            const int2 p = s.pair[w0 + i * 32 + lane];
            t_col[at] = p.x;
            t_val[at] = __int_as_float(p.y);
        }
        __syncthreads();  // the next chunk reuses all of it
    } else {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (key[i] >= 0) s.source[rank[i] + s.start[key[i]] + seen[key[i]]] = (unsigned short)(w0 + i * 32 + lane);
        async_wait<0>();
        __syncthreads();
        for (int i = tid; i < n; i += THREADS) {
            const int2 p = s.pair[s.source[i]];
            t_col[begin + i] = p.x;
            t_val[begin + i] = __int_as_float(p.y);
        }
    }
}

// The first ps.large CTAs take the chunks of larger buckets in turn (first: they are the longer ones), the others a bucket each
// if it is one chunk.
template <int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS, THREADS > 512 ? 1 : 4) transpose_bucket_sort_kernel(
    const BucketPass ps, int Kd, const unsigned short* __restrict__ low, const int2* __restrict__ pairs, const int* __restrict__ first_entry,
    const int* __restrict__ first_slot, const int* __restrict__ chunk_counts, int* __restrict__ t_row_ptr, int* __restrict__ t_col,
    float* __restrict__ t_val)
{
    wait_for_previous_grid();
    release_next_grid();
    extern __shared__ __align__(16) char smem_bytes[];
    const BucketSortSmem<THREADS, ITEMS> s(smem_bytes, 1 << ps.low_bits);
    if ((int)blockIdx.x < ps.large) {
        const int slots = __ldg(first_slot + (1 << ps.high_bits));
        for (int slot = blockIdx.x; slot < slots; slot += ps.large) {
            int begin, end;
            const int bucket = bucket_of_slot(ps, first_entry, first_slot, slot, begin, end);
            sort_chunk<THREADS, ITEMS, true>(ps, s, bucket, begin, end, __ldg(first_entry + bucket), slot, __ldg(first_slot + bucket),
                                             __ldg(first_slot + bucket + 1), Kd, low, pairs, chunk_counts, t_row_ptr, t_col, t_val);
        }
        return;
    }
    const int bucket = blockIdx.x - ps.large;
    if (bucket == 0 && threadIdx.x == 0) t_row_ptr[Kd] = ps.n;
    const int begin = __ldg(first_entry + bucket), end = __ldg(first_entry + bucket + 1);
    if (end - begin <= ps.chunk)
        sort_chunk<THREADS, ITEMS, false>(ps, s, bucket, begin, end, begin, 0, 0, 0, Kd, low, pairs, chunk_counts, t_row_ptr, t_col, t_val);
}

}  // namespace csrspmm_b200
