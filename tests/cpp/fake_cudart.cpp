// A CUDA runtime for tests of the library's host code without a GPU: device memory is host memory, kernels do
// nothing, and one chosen call fails.  Linked with the library's objects in place of the real runtime
// (csrspmm_b200/build.py), so that every way out of a failed call can be walked through on the CPU.
#include <cuda_runtime_api.h>
#include <cxxabi.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>

namespace {

std::mutex g_mutex;
std::set<void*> g_live;           // allocations not freed yet
std::map<void*, bool> g_busy;     // streams with work that nobody has waited for
std::map<void*, void*> g_event;   // the stream an event was recorded on
std::map<void*, std::set<void*>> g_after;  // the streams whose work a stream's work comes after
long g_calls = 0, g_fail_at = 0;  // the call that fails, counted from 1; 0: none
long g_bad_frees = 0;
std::map<const void*, int> g_smem;  // the dynamic shared memory a kernel may take, where it was set
long g_settings = 0;                // how often it was
long g_refused = 0;                 // launches that asked for more
std::atomic<long> g_streams{0};  // made and not destroyed
cudaError_t g_last = cudaSuccess;
char g_handles[4096];
size_t g_next_handle = 0;
std::set<std::string> g_launched;  // names of the kernels launched since the last reset

// The library's kernels by the address they are launched with.  Registered while its objects are loaded, which may be before this
// file's own variables are.
std::map<const void*, std::string>& kernels()
{
    static std::map<const void*, std::string> by_address;
    return by_address;
}

// Copies the names, a line each, to `out` (null: only asks for the room they take).
template <class Names>
size_t list_names(const Names& names, char* out)
{
    std::string all;
    for (const std::string& n : names) all += n + "\n";
    if (out != nullptr) std::memcpy(out, all.c_str(), all.size() + 1);
    return all.size() + 1;
}

// Counts a call that can fail.
cudaError_t call(cudaError_t error = cudaErrorUnknown)
{
    if (++g_calls != g_fail_at) return cudaSuccess;
    g_last = error;
    return error;
}

template <class T>
void new_handle(T* out)
{
    *out = reinterpret_cast<T>(&g_handles[g_next_handle++ % sizeof(g_handles)]);
}

cudaError_t allocate(void** out, size_t bytes)
{
    std::lock_guard<std::mutex> lock(g_mutex);
    if (const cudaError_t e = call(cudaErrorMemoryAllocation)) return e;
    *out = std::aligned_alloc(256, (bytes + 255) / 256 * 256);
    g_live.insert(*out);
    return cudaSuccess;
}

cudaError_t release(void* p)
{
    std::lock_guard<std::mutex> lock(g_mutex);
    if (p == nullptr) return cudaSuccess;
    if (g_live.erase(p) == 0) {
        ++g_bad_frees;
        return cudaErrorInvalidValue;
    }
    std::free(p);
    return cudaSuccess;
}

template <class F>
cudaError_t work_on(cudaStream_t st, F&& body)
{
    std::lock_guard<std::mutex> lock(g_mutex);
    if (const cudaError_t e = call()) return e;
    body();
    g_busy[st] = true;
    return cudaSuccess;
}

cudaError_t simple(cudaError_t error = cudaErrorUnknown)
{
    std::lock_guard<std::mutex> lock(g_mutex);
    return call(error);
}

}  // namespace

extern "C" {

void fake_reset(long fail_at)
{
    std::lock_guard<std::mutex> lock(g_mutex);
    g_calls = 0;
    g_fail_at = fail_at;
    g_bad_frees = 0;
    g_last = cudaSuccess;
    g_busy.clear();
    g_after.clear();
    g_launched.clear();
}
size_t fake_kernels(char* out)
{
    std::set<std::string> names;
    for (const auto& k : kernels()) names.insert(k.second);
    return list_names(names, out);
}
size_t fake_launched(char* out) { return list_names(g_launched, out); }
long fake_calls() { return g_calls; }
long fake_live() { return (long)g_live.size(); }
long fake_settings() { return g_settings; }
long fake_refused() { return g_refused; }
long fake_streams() { return g_streams; }
long fake_bad_frees() { return g_bad_frees; }
long fake_busy()
{
    long n = 0;
    for (const auto& s : g_busy) n += s.second;
    return n;
}

// ---- memory ----------------------------------------------------------------------------------------
cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return allocate(p, n); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return allocate(p, n); }
cudaError_t cudaFree(void* p) { return release(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return release(p); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
    *p = std::calloc(1, n);
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* pool, const cudaMemPoolProps*)
{
    new_handle(pool);
    return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return simple(); }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void* v)
{
    *static_cast<unsigned long long*>(v) = 0;
    return simple();
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st)
{
    return work_on(st, [&] { std::memset(p, v, n); });
}
cudaError_t cudaMemset2DAsync(void* p, size_t pitch, int v, size_t w, size_t h, cudaStream_t st)
{
    return work_on(st, [&] {
        for (size_t r = 0; r < h; ++r) std::memset(static_cast<char*>(p) + r * pitch, v, w);
    });
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
    return work_on(st, [&] { std::memcpy(d, s, n); });
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind)
{
    if (const cudaError_t e = simple()) return e;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t st)
{
    return work_on(st, [&] {
        for (size_t r = 0; r < h; ++r) std::memcpy(static_cast<char*>(d) + r * dp, static_cast<const char*>(s) + r * sp, w);
    });
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*)
{
    std::memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*)
{
    static char scratch[8 << 20];
    *p = scratch;
    return cudaSuccess;
}

// ---- device, streams, events -------------------------------------------------------------------------
cudaError_t cudaGetDevice(int* d)
{
    *d = 0;
    return simple();
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int)
{
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize()
{
    std::lock_guard<std::mutex> lock(g_mutex);
    g_busy.clear();
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st)
{
    std::lock_guard<std::mutex> lock(g_mutex);
    if (const cudaError_t e = call()) return e;
    g_busy[st] = false;
    for (void* before : g_after[st]) g_busy[before] = false;
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s)
{
    *s = cudaStreamCaptureStatusNone;
    return simple();
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* st, unsigned)
{
    if (const cudaError_t e = simple()) return e;
    new_handle(st);
    ++g_streams;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t)
{
    --g_streams;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
    if (const cudaError_t f = simple()) return f;
    new_handle(e);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st)
{
    std::lock_guard<std::mutex> lock(g_mutex);
    if (const cudaError_t f = call()) return f;
    g_event[e] = st;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned)
{
    std::lock_guard<std::mutex> lock(g_mutex);
    if (const cudaError_t f = call()) return f;
    const std::set<void*> before = g_after[g_event[e]];
    g_after[st].insert(before.begin(), before.end());
    g_after[st].insert(g_event[e]);
    return cudaSuccess;
}

// ---- kernels ---------------------------------------------------------------------------------------
cudaError_t cudaFuncSetAttribute(const void* kernel, cudaFuncAttribute, int value)
{
    std::lock_guard<std::mutex> lock(g_mutex);
    if (const cudaError_t e = call()) return e;
    g_smem[kernel] = value;
    ++g_settings;
    return cudaSuccess;
}
cudaError_t launch(const void* kernel, size_t smem, cudaStream_t st)
{
    return work_on(st, [&] {
        g_launched.insert(kernels()[kernel]);
        const auto allowed = g_smem.find(kernel);
        if (smem > (size_t)(allowed != g_smem.end() ? allowed->second : 48 << 10)) ++g_refused;
    });
}
cudaError_t cudaLaunchKernel(const void* kernel, dim3, dim3, void**, size_t smem, cudaStream_t st) { return launch(kernel, smem, st); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* kernel, void**) { return launch(kernel, c->dynamicSmemBytes, c->stream); }
cudaError_t cudaGetLastError()
{
    std::lock_guard<std::mutex> lock(g_mutex);
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "injected"; }

// ---- what compiled kernels register at load time and push before a launch ------------------------------
void** __cudaRegisterFatBinary(void*) { return reinterpret_cast<void**>(g_handles); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* address, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*)
{
    char* plain = abi::__cxa_demangle(name, nullptr, nullptr, nullptr);
    kernels()[address] = plain != nullptr ? plain : name;
    std::free(plain);
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
static thread_local struct { dim3 grid, block; size_t smem; void* stream; } t_launch;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* stream)
{
    t_launch = {grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream)
{
    *grid = t_launch.grid;
    *block = t_launch.block;
    *smem = t_launch.smem;
    *static_cast<void**>(stream) = t_launch.stream;
    return cudaSuccess;
}

}  // extern "C"
