// Small device-side helpers around the SpMM kernels: CSR validation and row statistics.
// Neither has a counterpart in the reference, whose host layer checks nothing
// (src/host/spmm_launcher.cu:11-171) and leaves max_row_nnz to the caller
// (src/host/csr_utils.cpp:105-110).
#pragma once

#include "common.cuh"

namespace csrspmm_b200 {

// problems: OR of the CSRSPMM_B200_CSR_* bits.
__global__ void validate_csr_kernel(int M, int Kd, long long nnz, const int* __restrict__ row_ptr,
                                    const int* __restrict__ col_idx, unsigned* problems)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned bad = 0;
    if (tid == 0) {
        if (row_ptr[0] != 0) bad |= 1u;
        if ((long long)row_ptr[M] != nnz) bad |= 2u;
    }
    for (long long r = tid; r < M; r += stride) {
        const int rs = row_ptr[r], re = row_ptr[r + 1];
        if (re < rs) {
            bad |= 4u;
            continue;
        }
        if (rs < 0 || (long long)re > nnz) continue;  // already reported through the end checks
        int prev = -1;
        for (int j = rs; j < re; ++j) {
            const int c = col_idx[j];
            if (c < 0 || c >= Kd) bad |= 8u;
            if (c <= prev) bad |= 16u;
            prev = c;
        }
    }
    if (bad) atomicOr(problems, bad);
}

// Of the above what keeps a product from placing an entry: bits 2 (row_ptr's end) and 8 (a column out of range), without a
// look at the rows.  *problems is zero before; whoever sees something writes all it saw.
constexpr int kBoundsThreads = 256;

__global__ void __launch_bounds__(kBoundsThreads) check_bounds_kernel(int M, int Kd, long long nnz, const int* __restrict__ row_ptr,
                                                                      const int* __restrict__ col_idx, volatile long long* problems)
{
    wait_for_previous_grid();
    release_next_grid();
    constexpr int PER = 8;
    unsigned bad = __ldg(row_ptr + M) != nnz ? 2u : 0u;
    for (long long j = (long long)blockIdx.x * (kBoundsThreads * PER) + threadIdx.x; j < nnz; j += (long long)gridDim.x * (kBoundsThreads * PER)) {
#pragma unroll
        for (int k = 0; k < PER; ++k)
            if (j + k * kBoundsThreads < nnz && (unsigned)__ldg(col_idx + j + k * kBoundsThreads) >= (unsigned)Kd) bad |= 8u;
    }
    if (__syncthreads_or(bad & 2u)) bad |= 2u;
    if (__syncthreads_or(bad & 8u)) bad |= 8u;
    if (threadIdx.x == 0 && bad) *problems = bad;
}

// A copy of B whose rows are whole vectors of four, zeros behind the last column.
__global__ void __launch_bounds__(256) pad_rows_kernel(long long vectors, int vectors_per_row, int Nd, const float* __restrict__ B, long long ldb,
                                                       float4* __restrict__ out)
{
    wait_for_previous_grid();
    release_next_grid();
    for (long long k = (long long)blockIdx.x * 256 + threadIdx.x; k < vectors; k += (long long)gridDim.x * 256) {
        const long long row = k / vectors_per_row;
        const int c = (int)(k - row * vectors_per_row) * 4;
        const float* src = B + row * ldb + c;
        float4 v = make_float4(__ldg(src), 0.f, 0.f, 0.f);
        if (c + 1 < Nd) v.y = __ldg(src + 1);
        if (c + 2 < Nd) v.z = __ldg(src + 2);
        if (c + 3 < Nd) v.w = __ldg(src + 3);
        out[k] = v;
    }
}

// Four numbers over all threads of a CTA: v[0] maximum, v[1..3] sums; valid in thread 0.
constexpr int kStatsThreads = 256;
constexpr int kStatsMaxCtas = kSms * 4;

__device__ __forceinline__ void stats_of_cta(long long (&v)[4])
{
    __shared__ long long part[kStatsThreads / 32][4];
    for (int o = 16; o > 0; o >>= 1) {
        v[0] = max(v[0], __shfl_xor_sync(0xffffffffu, v[0], o));
#pragma unroll
        for (int k = 1; k < 4; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    }
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 4; ++k) part[threadIdx.x >> 5][k] = v[k];
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kStatsThreads / 32; ++w) {
            v[0] = max(v[0], part[w][0]);
            for (int k = 1; k < 4; ++k) v[k] += part[w][k];
        }
    }
}

// Per CTA: longest row, empty rows, rows longer than 32 * (mean + 1), entries in those rows.
__global__ void __launch_bounds__(kStatsThreads) row_stats_kernel(int M, const int* __restrict__ row_ptr, long long* __restrict__ part)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long nnz = (long long)row_ptr[M] - row_ptr[0];
    const long long threshold = 32 * ((M > 0 ? nnz / M : 0) + 1);
    long long v[4] = {0, 0, 0, 0};
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < M; r += stride) {
        const long long len = (long long)row_ptr[r + 1] - row_ptr[r];
        if (len <= 0) ++v[1];
        v[0] = max(v[0], len);
        if (len > threshold) {
            ++v[2];
            v[3] += len;
        }
    }
    stats_of_cta(v);
    if (threadIdx.x == 0)
        for (int k = 0; k < 4; ++k) part[4 * blockIdx.x + k] = v[k];
}

__global__ void __launch_bounds__(kStatsThreads) row_stats_sum_kernel(int num, const long long* __restrict__ part, long long* stats)
{
    long long v[4] = {0, 0, 0, 0};
    for (int b = threadIdx.x; b < num; b += kStatsThreads) {
        v[0] = max(v[0], part[4 * b]);
        for (int k = 1; k < 4; ++k) v[k] += part[4 * b + k];
    }
    stats_of_cta(v);
    if (threadIdx.x == 0)
        for (int k = 0; k < 4; ++k) stats[k] = v[k];
}

}  // namespace csrspmm_b200
