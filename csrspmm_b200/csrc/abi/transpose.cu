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
    int passes, digit_bits, items;
    int tiles;
    long long counters;
    // workspace, in this order
    size_t keys, buffer[2], pairs[2], counts, offsets, scan, results, total;
};

TransposePlan plan_transpose(int32_t Kd, int64_t nnz)
{
    TransposePlan p = {};
    int bits = 1;
    while (bits < 31 && ((int64_t)1 << bits) < Kd) ++bits;
    // eight entries per thread (runs of 8 with 256 digits) while sixteen would leave fewer than three CTAs per SM
    p.items = nnz < (long long)kSms * 3 * kTransposeThreads * 16 ? 8 : 16;
    p.passes = (bits + kMaxDigitBits - 1) / kMaxDigitBits;
    p.digit_bits = (bits + p.passes - 1) / p.passes;
    const int64_t tile = (int64_t)kTransposeThreads * p.items;
    p.tiles = (int)((nnz + tile - 1) / tile);
    p.counters = ((long long)p.tiles) << p.digit_bits;
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t here = at;
        at += align256(bytes);
        return here;
    };
    p.keys = take((size_t)nnz * 4);
    for (int b = 0; b < 2; ++b) {  // one buffer between two passes, two in turn between more
        p.buffer[b] = take(p.passes > b + 1 ? (size_t)nnz * 4 : 0);
        p.pairs[b] = take(p.passes > b + 1 ? (size_t)nnz * 8 : 0);
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
    for (int k = 0; k < p.passes; ++k) {
        const DigitPass ps = {k * p.digit_bits, p.digit_bits, 1 << p.digit_bits, p.tiles, nnz};
        const bool first = k == 0, last = k == p.passes - 1;
        const int* keys = first ? col_idx : ints(p.buffer[(k - 1) & 1]);
        const int2* in = first ? nullptr : pairs(p.pairs[(k - 1) & 1]);
        int* out_keys = last ? ints(p.keys) : ints(p.buffer[k & 1]);
        int2* out = last ? nullptr : pairs(p.pairs[k & 1]);
        const bool self = p.tiles <= kSelfTiles;
        cudaError_t e = launch_overlapped(self ? transpose_count_kernel<ITEMS, true> : transpose_count_kernel<ITEMS, false>, (unsigned)p.tiles,
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
        auto pick = [&](auto first_c, auto last_c) { return self ? scatter(first_c, last_c, T()) : scatter(first_c, last_c, F()); };
        e = first && last ? pick(T(), T()) : first ? pick(T(), F()) : last ? pick(F(), T()) : pick(F(), F());
        if (e != cudaSuccess) return e;
    }
    if (nnz >= Kd)
        return launch_overlapped(transpose_row_ptr_kernel, (unsigned)((nnz + 1024) / 1024), 256, 0, st, Kd, (int)nnz, ints(p.keys), t_row_ptr);
    return launch_overlapped(transpose_row_ptr_search_kernel, (unsigned)(((long long)Kd + 256) / 256), 256, 0, st, Kd, (int)nnz, ints(p.keys),
                             t_row_ptr);
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
    const cudaError_t e = p.items == 8 ? run_transpose<8>(p, M, Kd, nnz, row_ptr, col_idx, values, t_row_ptr, t_col_idx, t_values, ws, st)
                                       : run_transpose<16>(p, M, Kd, nnz, row_ptr, col_idx, values, t_row_ptr, t_col_idx, t_values, ws, st);
    CUDA_TRY(e);
    return CSRSPMM_B200_OK;
}

}  // extern "C"
