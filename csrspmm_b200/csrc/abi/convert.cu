// extern "C" entry points for device-side dense <-> CSR conversion (declared in
// include/csrspmm_b200.h).  Counterparts of the reference's host-only dense2csr / csr2dense
// (src/host/csr_utils.cpp:70-145); results are identical, the matrices stay on the device.
#include <cuda_runtime.h>

#include <cstring>

#include "../kernels/codec_kernels.cuh"
#include "../kernels/convert_kernels.cuh"
#include "csrspmm_b200.h"
#include "pdl.h"
#include "plan.h"
#include "scan.h"
#include "scratch.h"

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

bool rows_on_16_bytes(const float* dense, int64_t ld) { return ld % 4 == 0 && (reinterpret_cast<uintptr_t>(dense) & 15u) == 0; }

unsigned convert_grid(int32_t H, int wpr)
{
    const int rows = (kConvertThreads / 32) / wpr;
    return (unsigned)(((long long)H + rows - 1) / rows);
}

// CTAs of the e2m1 kernels: enough to fill the chip, each with several 16-byte loads per thread
unsigned codec_grid(int64_t n)
{
    const long long want = (n + kCodecThreads * kCodecPer - 1) / (kCodecThreads * kCodecPer);
    return (unsigned)(want < kCodecMaxCtas ? want : kCodecMaxCtas);
}

float scale_from(float absmax) { return absmax > 0.0f ? absmax / 6.0f : 1.0f; }

}  // namespace

extern "C" {

size_t csrspmm_b200_dense2csr_mask_bytes(int32_t H, int32_t W) { return H > 0 && W > 0 ? (size_t)H * (size_t)words_per_row(W) * 4 : 0; }

int csrspmm_b200_dense2csr_count(int32_t H, int32_t W, const float* dense, int64_t ld, float tol, int32_t* row_ptr,
                                 int64_t* nnz_out, int32_t* max_row_nnz_out, csrspmm_b200_stream_t stream)
{
    return csrspmm_b200_dense2csr_count_mask(H, W, dense, ld, tol, row_ptr, nullptr, nnz_out, max_row_nnz_out, stream);
}

int csrspmm_b200_dense2csr_count_mask(int32_t H, int32_t W, const float* dense, int64_t ld, float tol, int32_t* row_ptr, uint32_t* mask,
                                      int64_t* nnz_out, int32_t* max_row_nnz_out, csrspmm_b200_stream_t stream)
{
    if (H < 0 || W < 0 || ld < W || row_ptr == nullptr || nnz_out == nullptr || (H > 0 && W > 0 && dense == nullptr)) {
        set_last_error("dense2csr_count: bad argument");
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    *nnz_out = 0;
    if (max_row_nnz_out) *max_row_nnz_out = 0;
    if (H == 0) {
        CUDA_TRY(cudaMemsetAsync(row_ptr, 0, sizeof(int), st));
        CUDA_TRY(cudaStreamSynchronize(st));
        return CSRSPMM_B200_OK;
    }
    const size_t scan_bytes = (scan_scratch_bytes(H) + 255) / 256 * 256;
    Scratch scratch(st);  // the scan's, then one count per row
    CUDA_TRY(scratch.alloc(scan_bytes + sizeof(int) * (size_t)H));
    int* counts = reinterpret_cast<int*>(scratch.as<char>() + scan_bytes);
    Results results(st);
    CUDA_TRY(results.init());
    const int wpr = convert_warps_per_row(W, kChunkCols);
    const unsigned grid = convert_grid(H, wpr);
    CUDA_TRY(launch_overlapped(rows_on_16_bytes(dense, ld) ? dense_count_kernel<true> : dense_count_kernel<false>, grid, kConvertThreads, 0, st,
                               H, W, dense, ld, tol, wpr, counts, mask));
    CUDA_TRY(exclusive_scan(counts, H, row_ptr, scratch.as<void>(), results.ptr(), st));
    long long out[2] = {0, 0};
    CUDA_TRY(results.wait(out, 2));
    if (out[0] > 0x7fffffffLL) {  // the int32 offsets wrapped
        set_last_error("dense2csr_count: more than 2^31-1 non-zeros");
        return CSRSPMM_B200_ERR_UNSUPPORTED;
    }
    *nnz_out = out[0];
    if (max_row_nnz_out) *max_row_nnz_out = (int32_t)out[1];
    return CSRSPMM_B200_OK;
}

int csrspmm_b200_dense2csr_fill(int32_t H, int32_t W, const float* dense, int64_t ld, float tol, const int32_t* row_ptr,
                                int32_t* col_idx, float* values, csrspmm_b200_stream_t stream)
{
    return csrspmm_b200_dense2csr_fill_mask(H, W, dense, ld, tol, nullptr, row_ptr, col_idx, values, stream);
}

int csrspmm_b200_dense2csr_fill_mask(int32_t H, int32_t W, const float* dense, int64_t ld, float tol, const uint32_t* mask, const int32_t* row_ptr,
                                     int32_t* col_idx, float* values, csrspmm_b200_stream_t stream)
{
    if (H < 0 || W < 0 || ld < W || row_ptr == nullptr) {
        set_last_error("dense2csr_fill: bad argument");
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (H == 0 || W == 0) return CSRSPMM_B200_OK;
    if (dense == nullptr || col_idx == nullptr || values == nullptr) {
        set_last_error("dense2csr_fill: null pointer");
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    const int wpr = convert_warps_per_row(W, kSpanCols);
    CUDA_TRY(launch_overlapped(rows_on_16_bytes(dense, ld) ? dense_fill_kernel<true> : dense_fill_kernel<false>, convert_grid(H, wpr), kConvertThreads,
                               0, reinterpret_cast<cudaStream_t>(stream), H, W, dense, ld, tol, wpr, mask, row_ptr, col_idx, values));
    return CSRSPMM_B200_OK;
}

int csrspmm_b200_csr2dense(int32_t H, int32_t W, const int32_t* row_ptr, const int32_t* col_idx, const float* values,
                           float* dense, int64_t ld, csrspmm_b200_stream_t stream)
{
    if (H < 0 || W < 0 || ld < W || (H > 0 && (row_ptr == nullptr || (W > 0 && dense == nullptr)))) {
        set_last_error("csr2dense: bad argument");
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (H == 0 || W == 0) return CSRSPMM_B200_OK;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    CUDA_TRY(cudaMemset2DAsync(dense, (size_t)ld * 4, 0, (size_t)W * 4, (size_t)H, st));
    csr_scatter_kernel<<<(unsigned)(((long long)H + 7) / 8), 256, 0, st>>>(H, W, row_ptr, col_idx, values, dense, ld);
    CUDA_TRY(cudaGetLastError());
    return CSRSPMM_B200_OK;
}

// ---- e2m1 codec on the device ------------------------------------------------------------------

int csrspmm_b200_e2m1_scale_device(int64_t n, const float* values, float* scale_out, csrspmm_b200_stream_t stream)
{
    if (n < 0 || scale_out == nullptr || (n > 0 && values == nullptr)) {
        set_last_error("e2m1_scale_device: bad argument");
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    *scale_out = 1.0f;
    if (n == 0) return CSRSPMM_B200_OK;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    Scratch partial(st);
    CUDA_TRY(partial.alloc(sizeof(float) * kCodecMaxCtas));
    const unsigned grid = codec_grid(n);
    CUDA_TRY(launch_overlapped(e2m1_absmax_kernel, grid, kCodecThreads, 0, st, n, values, partial.as<float>()));
    float h[kCodecMaxCtas];
    CUDA_TRY(cudaMemcpyAsync(h, partial.as<float>(), sizeof(float) * grid, cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    float mx = 0.0f;
    for (unsigned k = 0; k < grid; ++k) mx = h[k] > mx ? h[k] : mx;
    *scale_out = scale_from(mx);
    return CSRSPMM_B200_OK;
}

int csrspmm_b200_e2m1_encode_device(int64_t n, const float* values, float scale, uint8_t* packed,
                                    csrspmm_b200_stream_t stream)
{
    if (n < 0 || (n > 0 && (values == nullptr || packed == nullptr)) || !(scale > 0.0f)) {
        set_last_error("e2m1_encode_device: bad argument");
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (n == 0) return CSRSPMM_B200_OK;
    CUDA_TRY(launch_overlapped(e2m1_encode_kernel, codec_grid(n), kCodecThreads, 0, reinterpret_cast<cudaStream_t>(stream), n, values, scale,
                               nullptr, 0, packed, nullptr));
    return CSRSPMM_B200_OK;
}

int csrspmm_b200_e2m1_quantize_device(int64_t n, const float* values, float* scale_out, uint8_t* packed,
                                      csrspmm_b200_stream_t stream)
{
    if (n < 0 || scale_out == nullptr || (n > 0 && (values == nullptr || packed == nullptr))) {
        set_last_error("e2m1_quantize_device: bad argument");
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    *scale_out = 1.0f;
    if (n == 0) return CSRSPMM_B200_OK;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    Scratch partial(st);
    CUDA_TRY(partial.alloc(sizeof(float) * kCodecMaxCtas));
    Results results(st);
    CUDA_TRY(results.init());
    const unsigned grid = codec_grid(n);
    CUDA_TRY(launch_overlapped(e2m1_absmax_kernel, grid, kCodecThreads, 0, st, n, values, partial.as<float>()));
    CUDA_TRY(launch_overlapped(e2m1_encode_kernel, grid, kCodecThreads, 0, st, n, values, 1.0f, partial.as<float>(), (int)grid, packed,
                               results.ptr()));
    long long bits = 0;
    CUDA_TRY(results.wait(&bits, 1));
    const unsigned word = (unsigned)bits;
    memcpy(scale_out, &word, sizeof(word));
    if (!(*scale_out > 0.0f)) {  // the largest magnitude is under 6 times the smallest denormal: no scale to divide by
        set_last_error("e2m1_quantize_device: the scale underflows");
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    return CSRSPMM_B200_OK;
}

int csrspmm_b200_e2m1_decode_device(int64_t n, const uint8_t* packed, float scale, float* values,
                                    csrspmm_b200_stream_t stream)
{
    if (n < 0 || (n > 0 && (values == nullptr || packed == nullptr))) {
        set_last_error("e2m1_decode_device: bad argument");
        return CSRSPMM_B200_ERR_BAD_ARG;
    }
    if (n == 0) return CSRSPMM_B200_OK;
    const long long want = (n + 255) / 256;
    const unsigned grid = (unsigned)(want < kSms * 16 ? want : kSms * 16);
    e2m1_decode_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(n, packed, scale, values);
    CUDA_TRY(cudaGetLastError());
    return CSRSPMM_B200_OK;
}

}  // extern "C"
