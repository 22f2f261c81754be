// extern "C" transposition of a device-resident CSR matrix (declared in include/csrspmm_b200.h).
#include <cuda_runtime.h>

#include <type_traits>

#include "../kernels/transpose_kernels.cuh"
#include "csrspmm_b200.h"
#include "pdl.h"
#include "plan.h"
#include "scan.h"

using namespace csrspmm_b200;

#define CUDA_TRY(expr)                                                                        \
    do {                                                                                      \
        cudaError_t e__ = (expr);                                                             \
        if (e__ != cudaSuccess) {                                                             \
            set_last_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e__), __FILE__, \
                           __LINE__);                                                         \
            return CSRSPMM_B200_ERR_CUDA;                                                     \
        }                                                                                     \
    } while (0)

namespace {

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

struct TransposePlan {
    bool by_buckets;
    BucketPass bucket;
    int passes, digit_bits, items;
    int tiles;
    long long counters;
    // workspace, in this order
    size_t keys, buffer[2], pairs[2], first_row, totals, first_entry, first_slot, chunk_counts, counts, offsets, scan, results, total;
};

// Up to here one CTA makes the buckets and there is nothing to count across tiles: two launches less (1500 entries
// 14.1 -> 9.9 us, 5000 15.6 -> 12.1, 8000 15.7 -> 14.8).
constexpr int64_t kOneTile = kBucketThreads * kBucketItems;

// The sort's CTAs: 512 threads and 4096 entries, or 1024 and 8192 where the buckets are twice as large.
constexpr int kBucketChunk = 4096;

// Through buckets where a bucket and its columns fit a CTA of the sort: the mean bucket fills half of the CTA's room, so that
// uniform columns leave it some, and no bucket is wider than kMaxBucketColumns.
bool plan_buckets(int bits, int64_t nnz, BucketPass* b)
{
    const int most = bits < kMaxBucketBits ? bits : kMaxBucketBits;
    int high = bits > kMaxColumnBits ? bits - kMaxColumnBits : 0;
    if (high > most || nnz == 0) return false;
    b->chunk = (nnz >> most) > kBucketChunk / 2 ? 2 * kBucketChunk : kBucketChunk;
    while (high < most && (nnz >> high) > b->chunk / 2) ++high;
    if ((nnz >> high) > b->chunk / 2 || nnz > (int64_t)kMaxBucketTiles * kBucketThreads * kBucketItems) return false;
    b->high_bits = high;
    b->low_bits = bits - high;
    b->n = (int)nnz;
    return true;
}

TransposePlan plan_transpose(int32_t Kd, int64_t nnz)
{
    TransposePlan p = {};
    int bits = 1;
    while (bits < 31 && ((int64_t)1 << bits) < Kd) ++bits;
    p.by_buckets = plan_buckets(bits, nnz, &p.bucket);
    // eight entries per thread (runs of 8 with 256 digits) while sixteen would leave fewer than three CTAs per SM
    p.items = nnz < (long long)kSms * 3 * kTransposeThreads * 16 ? 8 : 16;
    p.passes = (bits + kMaxDigitBits - 1) / kMaxDigitBits;
    p.digit_bits = (bits + p.passes - 1) / p.passes;
    const int64_t tile = (int64_t)kTransposeThreads * p.items;
    p.tiles = (int)((nnz + tile - 1) / tile);
    p.counters = ((long long)p.tiles) << p.digit_bits;
    if (p.by_buckets) {
        // tiles of whole waves: 1.7 M entries are 280 tiles of 6 entries per thread, not 210 of 8 (one CTA per SM)
        const long long wave = (long long)kSms * kBucketThreads, waves = (nnz + wave * kBucketItems - 1) / (wave * kBucketItems);
        p.bucket.items = (int)((nnz + wave * waves - 1) / (wave * waves));
        if (nnz <= kOneTile) p.bucket.items = (int)((nnz + kBucketThreads - 1) / kBucketThreads);
        const long long tile = (long long)kBucketThreads * p.bucket.items;
        p.tiles = p.bucket.tiles = (int)((nnz + tile - 1) / tile);
        // CTAs for the chunks of larger buckets: as many as there can be, or two per SM that take several each
        const long long most = nnz > p.bucket.chunk ? nnz / p.bucket.chunk * 2 + 1 : 0;
        p.bucket.large = (int)(most < 2 * kSms ? most : 2 * kSms);
        p.counters = ((long long)p.tiles) << p.bucket.high_bits;
    }
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t here = at;
        at += align256(bytes);
        return here;
    };
    if (p.by_buckets) {
        const size_t buckets = (size_t)1 << p.bucket.high_bits;
        p.keys = take((size_t)nnz * 2);
        p.pairs[0] = take((size_t)nnz * 8);
        p.first_row = take(((size_t)p.tiles * (kBucketThreads / 32) + 1) * 4);
        p.totals = take(buckets * 4);
        p.first_entry = take((buckets + 1) * 4);
        p.first_slot = take((buckets + 1) * 4);
        // a bucket of more than one chunk holds more than half of what its chunks could
        p.chunk_counts = take(nnz > p.bucket.chunk ? (((size_t)nnz / p.bucket.chunk * 2 + 2) << p.bucket.low_bits) * 4 : 0);
    } else {
        p.keys = take((size_t)nnz * 4);
        for (int b = 0; b < 2; ++b) {  // one buffer between two passes, two in turn between more
            p.buffer[b] = take(p.passes > b + 1 ? (size_t)nnz * 4 : 0);
            p.pairs[b] = take(p.passes > b + 1 ? (size_t)nnz * 8 : 0);
        }
    }
    p.counts = take((size_t)p.counters * 4);
    p.offsets = take(((size_t)p.counters + 1) * 4);
    p.scan = take(scan_scratch_bytes(p.counters));
    p.results = take(16);
    p.total = at;
    return p;
}

template <int ITEMS>
cudaError_t run_transpose(const TransposePlan& p, int32_t M, int32_t Kd, int64_t nnz, const int32_t* row_ptr, const int32_t* col_idx,
                          const float* values, int32_t* t_row_ptr, int32_t* t_col_idx, float* t_values, char* ws, cudaStream_t st)
{
    auto ints = [&](size_t off) { return reinterpret_cast<int*>(ws + off); };
    auto pairs = [&](size_t off) { return reinterpret_cast<int2*>(ws + off); };
    long long* results = reinterpret_cast<long long*>(ws + p.results);
    constexpr bool kCanSelf = ITEMS == 8;  // sixteen entries per thread are for more tiles than that (plan_transpose)
    for (int k = 0; k < p.passes; ++k) {
        const DigitPass ps = {k * p.digit_bits, 1 << p.digit_bits, p.tiles, nnz};
        const bool first = k == 0, last = k == p.passes - 1;
        const int* keys = first ? col_idx : ints(p.buffer[(k - 1) & 1]);
        const int2* in = first ? nullptr : pairs(p.pairs[(k - 1) & 1]);
        int* out_keys = last ? ints(p.keys) : ints(p.buffer[k & 1]);
        int2* out = last ? nullptr : pairs(p.pairs[k & 1]);
        const bool self = kCanSelf && p.tiles <= kSelfTiles;
        cudaError_t e = launch_overlapped(self ? transpose_count_kernel<ITEMS, kCanSelf> : transpose_count_kernel<ITEMS, false>, (unsigned)p.tiles,
                                          kTransposeThreads, 0, st, ps, keys, Kd, ints(p.counts));
        if (e == cudaSuccess && !self) e = exclusive_scan(ints(p.counts), p.counters, ints(p.offsets), ws + p.scan, results, st);
        if (e != cudaSuccess) return e;
        auto scatter = [&](auto first_c, auto last_c, auto self_c) {
            constexpr auto kernel = transpose_scatter_kernel<ITEMS, decltype(first_c)::value, decltype(last_c)::value, decltype(self_c)::value>;
            const cudaError_t e = allow_dynamic_smem<kernel>(sizeof(ScatterSmem<ITEMS>));
            if (e != cudaSuccess) return e;
            return launch_overlapped(kernel, (unsigned)p.tiles, kTransposeThreads, sizeof(ScatterSmem<ITEMS>), st, ps, keys, in, row_ptr, M, Kd,
                                     values, ints(self ? p.counts : p.offsets), out_keys, out, t_col_idx, t_values);
        };
        using T = std::true_type;
        using F = std::false_type;
        auto pick = [&](auto first_c, auto last_c) {
            return self ? scatter(first_c, last_c, std::bool_constant<kCanSelf>()) : scatter(first_c, last_c, F());
        };
        e = first && last ? pick(T(), T()) : first ? pick(T(), F()) : last ? pick(F(), T()) : pick(F(), F());
        if (e != cudaSuccess) return e;
    }
    if (nnz >= Kd)
        return launch_overlapped(transpose_row_ptr_kernel, (unsigned)((nnz + 1024) / 1024), 256, 0, st, Kd, (int)nnz, ints(p.keys), t_row_ptr);
    return launch_overlapped(transpose_row_ptr_search_kernel, (unsigned)(((long long)Kd + 256) / 256), 256, 0, st, Kd, (int)nnz, ints(p.keys),
                             t_row_ptr);
}

cudaError_t run_buckets(const TransposePlan& p, int32_t M, int32_t Kd, const int32_t* row_ptr, const int32_t* col_idx, const float* values,
                        int32_t* t_row_ptr, int32_t* t_col_idx, float* t_values, char* ws, cudaStream_t st)
{
    auto ints = [&](size_t off) { return reinterpret_cast<int*>(ws + off); };
    const BucketPass& ps = p.bucket;
    const int buckets = 1 << ps.high_bits;
    unsigned short* low = reinterpret_cast<unsigned short*>(ws + p.keys);
    int2* pairs = reinterpret_cast<int2*>(ws + p.pairs[0]);
    cudaError_t e = cudaSuccess;
    if (p.tiles > 1) {
        e = launch_overlapped(transpose_bucket_count_kernel, (unsigned)p.tiles, kBucketThreads, 0, st, ps, col_idx, row_ptr, M, Kd,
                              ints(p.counts), ints(p.first_row));
        if (e == cudaSuccess)
            e = launch_overlapped(transpose_bucket_offsets_kernel, (unsigned)((buckets + 31) / 32), 1024, 0, st, ps, ints(p.counts), ints(p.totals));
    }
    constexpr auto scatter = transpose_bucket_scatter_kernel;
    const size_t scatter_smem = (size_t)BucketSmem::bytes(buckets);
    if (e == cudaSuccess) e = allow_dynamic_smem<scatter>(scatter_smem);
    if (e == cudaSuccess)
        e = launch_overlapped(scatter, (unsigned)p.tiles, kBucketThreads, scatter_smem, st, ps, col_idx, row_ptr, M, Kd, values, ints(p.counts),
                              ints(p.totals), ints(p.first_row), low, pairs, ints(p.first_entry), ints(p.first_slot));
    if (e != cudaSuccess) return e;
    if (ps.large > 0)
        e = launch_overlapped(transpose_chunk_count_kernel, (unsigned)ps.large, 512, 0, st, ps, low, ints(p.first_entry), ints(p.first_slot),
                              ints(p.chunk_counts));
    if (e != cudaSuccess) return e;
    auto sort = [&](auto threads_c) {
        constexpr int threads = decltype(threads_c)::value;
        using Smem = BucketSortSmem<threads, kBucketChunk / 512>;
        constexpr auto kernel = transpose_bucket_sort_kernel<threads, kBucketChunk / 512>;
        const size_t smem = (size_t)Smem::bytes(1 << ps.low_bits);
        const cudaError_t se = allow_dynamic_smem<kernel>(smem);
        if (se != cudaSuccess) return se;
        return launch_overlapped(kernel, buckets + ps.large, threads, smem, st, ps, Kd, low, pairs, ints(p.first_entry), ints(p.first_slot),
                                 ints(p.chunk_counts), t_row_ptr, t_col_idx, t_values);
    };
    return ps.chunk == kBucketChunk ? sort(std::integral_constant<int, 512>()) : sort(std::integral_constant<int, 1024>());
}

}  // namespace

extern "C" {

size_t csrspmm_b200_transpose_workspace_bytes(int32_t Kd, int64_t nnz)
{
    if (Kd < 0 || nnz < 0 || nnz > 0x7fffffffLL) return 0;
    return plan_transpose(Kd, nnz).total;
}

int csrspmm_b200_transpose(int32_t M, int32_t Kd, int64_t nnz, const int32_t* row_ptr, const int32_t* col_idx, const float* values,
                           int32_t* t_row_ptr, int32_t* t_col_idx, float* t_values, void* workspace, size_t workspace_bytes,
                           csrspmm_b200_stream_t stream)
{
    if (M < 0 || Kd < 0 || nnz < 0 || nnz > 0x7fffffffLL || t_row_ptr == nullptr || (nnz > 0 && (M == 0 || Kd == 0)) ||
        (nnz > 0 && (row_ptr == nullptr || col_idx == nullptr || values == nullptr || t_col_idx == nullptr || t_values == nullptr))) {
        set_last_error("transpose: bad argument");
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (nnz == 0) {
        CUDA_TRY(cudaMemsetAsync(t_row_ptr, 0, ((size_t)Kd + 1) * 4, st));
        return CSRSPMM_B200_OK;
    }
    const TransposePlan p = plan_transpose(Kd, nnz);
    if (workspace == nullptr || workspace_bytes < p.total || (reinterpret_cast<uintptr_t>(workspace) & 255u) != 0) {
        set_last_error("transpose: workspace of %zu bytes at %p: need %zu bytes, 256-byte aligned", workspace_bytes, workspace, p.total);
        return CSRSPMM_B200_ERR_WORKSPACE;
    }
    char* ws = static_cast<char*>(workspace);
    if (p.by_buckets) {
        CUDA_TRY(run_buckets(p, M, Kd, row_ptr, col_idx, values, t_row_ptr, t_col_idx, t_values, ws, st));
        return CSRSPMM_B200_OK;
    }
    const cudaError_t e = p.items == 8 ? run_transpose<8>(p, M, Kd, nnz, row_ptr, col_idx, values, t_row_ptr, t_col_idx, t_values, ws, st)
                                       : run_transpose<16>(p, M, Kd, nnz, row_ptr, col_idx, values, t_row_ptr, t_col_idx, t_values, ws, st);
    CUDA_TRY(e);
    return CSRSPMM_B200_OK;
}

}  // extern "C"
