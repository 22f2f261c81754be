// Memory the entry points need for the length of one call: device scratch and a few pinned bytes for a
// result the host waits for.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace csrspmm_b200 {

// Stream-ordered device scratch out of the library's own pool on the current device.  The default pool hands
// everything back to the driver at each synchronisation, and mapping memory anew made a call that
// waits for its result (row statistics, dense -> CSR, quantisation) cost 0.3 to 2 ms; this pool keeps up to
// kScratchKept bytes per device for the next call (and what is above goes back as it does there), until scratch_release.
constexpr size_t kScratchKept = (size_t)64 << 20;
cudaError_t scratch_alloc(void** ptr, size_t bytes, cudaStream_t st);
// The same for scratch of a product, which may be under stream capture: there it comes from cudaMallocAsync (a
// graph owns its allocations, and making a pool is no call for a capture).
cudaError_t product_scratch_alloc(void** ptr, size_t bytes, cudaStream_t st);
// Gives back what the pools keep and nobody uses, on all devices; *bytes (may be null): how much that was.
cudaError_t scratch_release(size_t* bytes);
inline cudaError_t scratch_free(void* ptr, cudaStream_t st) { return cudaFreeAsync(ptr, st); }

// Scratch that goes back to the pool when the scope ends, in stream order.
class Scratch {
public:
    explicit Scratch(cudaStream_t st) : st_(st) {}
    Scratch(const Scratch&) = delete;
    Scratch& operator=(const Scratch&) = delete;
    ~Scratch()
    {
        if (ptr_) scratch_free(ptr_, st_);
    }
    cudaError_t alloc(size_t bytes) { return scratch_alloc(&ptr_, bytes, st_); }
    template <class T>
    T* as() const
    {
        return static_cast<T*>(ptr_);
    }

private:
    cudaStream_t st_;
    void* ptr_ = nullptr;
};

// kPinnedWords 8-byte words of page-locked memory that kernels write to directly and the host reads after
// waiting for the stream: one write over the link instead of a staged copy.  Slots come from one page per
// process (64 of them) and go back when the scope ends; words() is null when all are in use.
constexpr int kPinnedWords = 8;
class PinnedSlot {
public:
    PinnedSlot();
    ~PinnedSlot();
    PinnedSlot(const PinnedSlot&) = delete;
    PinnedSlot& operator=(const PinnedSlot&) = delete;
    volatile long long* words() const { return words_; }

private:
    volatile long long* words_ = nullptr;
    int index_ = -1;
};

// Up to kPinnedWords results of a call: kernels write ptr()[k], wait() waits for the stream and reads them.  A call that
// fails in between waits here all the same: a kernel that it did launch must not write to the slot of the next call.
class Results {
public:
    explicit Results(cudaStream_t st) : st_(st), dev_(st) {}
    Results(const Results&) = delete;
    Results& operator=(const Results&) = delete;
    ~Results()
    {
        if (lent_) cudaStreamSynchronize(st_);
    }
    cudaError_t init()
    {
        lent_ = slot_.words() != nullptr;
        if (slot_.words() != nullptr) return cudaSuccess;
        return dev_.alloc(kPinnedWords * sizeof(long long));  // every slot taken: plain scratch, copied back
    }
    // word 0 = 0, for kernels that only write what they find
    cudaError_t clear()
    {
        if (slot_.words() == nullptr) return cudaMemsetAsync(dev_.as<long long>(), 0, sizeof(long long), st_);
        slot_.words()[0] = 0;
        return cudaSuccess;
    }
    long long* ptr() const { return slot_.words() != nullptr ? const_cast<long long*>(slot_.words()) : dev_.as<long long>(); }
    cudaError_t wait(long long* out, int count)
    {
        if (slot_.words() == nullptr) {
            const cudaError_t e = cudaMemcpyAsync(out, dev_.as<long long>(), count * sizeof(long long), cudaMemcpyDeviceToHost, st_);
            return e != cudaSuccess ? e : cudaStreamSynchronize(st_);
        }
        const cudaError_t e = cudaStreamSynchronize(st_);
        lent_ = e != cudaSuccess;
        for (int k = 0; k < count; ++k) out[k] = slot_.words()[k];
        return e;
    }

private:
    cudaStream_t st_;
    PinnedSlot slot_;
    Scratch dev_;
    bool lent_ = false;  // kernels may be writing to the slot
};

}  // namespace csrspmm_b200
