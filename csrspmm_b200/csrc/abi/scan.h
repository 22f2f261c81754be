// Exclusive scan on the device (kernels/scan_kernels.cuh).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace csrspmm_b200 {

// Bytes of scratch exclusive_scan needs for n counts (8-byte aligned).
size_t scan_scratch_bytes(long long n);

// offsets[0..n] = exclusive scan of counts[0..n); results[0] = total, results[1] = largest count.  One or two launches.
cudaError_t exclusive_scan(const int* counts, long long n, int* offsets, void* scratch, long long* results, cudaStream_t st);

}  // namespace csrspmm_b200
