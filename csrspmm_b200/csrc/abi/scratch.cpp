// Call-length scratch (see scratch.h).
#include "scratch.h"

#include <mutex>

namespace csrspmm_b200 {

namespace {

constexpr int kMaxDevices = 64;

std::mutex g_mutex;
cudaMemPool_t g_pool[kMaxDevices] = {};
bool g_pool_tried[kMaxDevices] = {};

constexpr int kSlots = 64;
long long* g_page = nullptr;
bool g_page_tried = false;
unsigned long long g_busy = 0;  // bit k: slot k is in use

cudaMemPool_t pool_of(int device)
{
    if (device < 0 || device >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_pool_tried[device]) {
        g_pool_tried[device] = true;
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool = nullptr;
        if (cudaMemPoolCreate(&pool, &props) == cudaSuccess) {
            unsigned long long keep = kScratchKept;
            if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess) g_pool[device] = pool;
            else cudaMemPoolDestroy(pool);
        }
        if (g_pool[device] == nullptr) cudaGetLastError();  // the default pool serves instead
    }
    return g_pool[device];
}

}  // namespace

cudaError_t scratch_alloc(void** ptr, size_t bytes, cudaStream_t st)
{
    int device = -1;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (bytes == 0) bytes = 1;
    cudaMemPool_t pool = pool_of(device);
    return pool != nullptr ? cudaMallocFromPoolAsync(ptr, bytes, pool, st) : cudaMallocAsync(ptr, bytes, st);
}

cudaError_t product_scratch_alloc(void** ptr, size_t bytes, cudaStream_t st)
{
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    const cudaError_t e = cudaStreamIsCapturing(st, &capture);
    if (e != cudaSuccess) return e;
    return capture == cudaStreamCaptureStatusNone ? scratch_alloc(ptr, bytes, st) : cudaMallocAsync(ptr, bytes, st);
}

cudaError_t scratch_release(size_t* bytes)
{
    if (bytes) *bytes = 0;
    std::lock_guard<std::mutex> lock(g_mutex);
    for (cudaMemPool_t pool : g_pool) {
        if (pool == nullptr) continue;
        unsigned long long before = 0, after = 0;
        cudaError_t e = cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &before);
        if (e == cudaSuccess) e = cudaMemPoolTrimTo(pool, 0);
        if (e == cudaSuccess) e = cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &after);
        if (e != cudaSuccess) return e;
        if (bytes) *bytes += (size_t)(before - after);
    }
    return cudaSuccess;
}

PinnedSlot::PinnedSlot()
{
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_page_tried) {
        g_page_tried = true;
        if (cudaHostAlloc(reinterpret_cast<void**>(&g_page), kSlots * kPinnedWords * sizeof(long long),
                          cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
            cudaGetLastError();
            g_page = nullptr;
        }
    }
    if (g_page == nullptr || g_busy == ~0ull) return;
    index_ = __builtin_ctzll(~g_busy);
    g_busy |= 1ull << index_;
    words_ = g_page + index_ * kPinnedWords;
}

PinnedSlot::~PinnedSlot()
{
    if (index_ < 0) return;
    std::lock_guard<std::mutex> lock(g_mutex);
    g_busy &= ~(1ull << index_);
}

}  // namespace csrspmm_b200
