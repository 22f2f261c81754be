// Launches whose start overlaps the end of the kernel before them in the stream (programmatic dependent launch).
//
// A kernel started this way may begin as soon as every CTA of its predecessor has called
// release_next_grid() (kernels/common.cuh) or ended, and must call wait_for_previous_grid() before it touches
// global memory: that waits until the predecessor has completed and its writes are visible.  Every kernel here
// calls it first thing in every thread, so that completion stays transitive along the stream.  What overlaps is
// the launch itself: 2 to 3 us of a small product.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>
#include <mutex>

namespace csrspmm_b200 {

// The opt-in to more than 48 KB of dynamic shared memory, once per device and kernel and again when a launch needs more, so
// that later launches (in a stream capture too) are plain ones.  Threads that race with different sizes end with the larger.
template <auto kernel>
cudaError_t allow_dynamic_smem(size_t bytes)
{
    constexpr int kMaxDevices = 64;
    static std::atomic<size_t> granted[kMaxDevices] = {};
    static std::mutex mutex;
    int device = -1;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const bool known = device >= 0 && device < kMaxDevices;
    if (known && granted[device].load(std::memory_order_acquire) >= bytes) return cudaSuccess;
    std::lock_guard<std::mutex> lock(mutex);
    if (known && granted[device].load(std::memory_order_relaxed) >= bytes) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && known) granted[device].store(bytes, std::memory_order_release);
    return e;
}

template <class... Params, class... Args>
cudaError_t launch_overlapped(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, Args... args)
{
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

}  // namespace csrspmm_b200
