// CPython/torch binding of the C ABI: what csrspmm_b200/ops.py calls on its per-product path.
//
// A small product is over in 3 to 10 us on the GPU, so what a call costs on the host is what the caller
// waits for.  Reading a tensor's address, sizes and device through Python attributes, filling a ctypes
// structure field by field and allocating C through torch.empty took 17 us per call; the same work here takes
// about 4 us, most of it the kernel launch and the allocation of C (1024 x 1024 matrix, 10 entries per row,
// 64 columns).  Plays the part of the reference's pybind wrappers (torch_csrspmm/binding.cpp:26-32,
// torch_csrspmm/torch_csrspmm_naive.cpp:11-58) with its argument checks and messages, on the current stream.
//
// The library's functions arrive as addresses (init), so that the library itself stays free of torch and the
// one ctypes loaded is the one used here.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/VariableTypeUtils.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/library.h>

#include <algorithm>
#include <chrono>
#include <cstdint>
#include <mutex>
#include <optional>

#include "csrspmm_b200.h"

namespace {

struct Library {
    int (*spmm)(const csrspmm_b200_args*, csrspmm_b200_stream_t);
    int (*spmm_sync)(const csrspmm_b200_args*, csrspmm_b200_stream_t);
    int (*uses_workspace)(const csrspmm_b200_args*);
    size_t (*workspace_bytes)(const csrspmm_b200_args*);
    size_t (*least_workspace_bytes)(const csrspmm_b200_args*);
    int (*row_stats)(int32_t, const int32_t*, int64_t*, csrspmm_b200_stream_t);
    size_t (*dense2csr_mask_bytes)(int32_t, int32_t);
    int (*dense2csr_count)(int32_t, int32_t, const float*, int64_t, float, int32_t*, uint32_t*, int64_t*, int32_t*, csrspmm_b200_stream_t);
    int (*dense2csr_fill)(int32_t, int32_t, const float*, int64_t, float, const uint32_t*, const int32_t*, int32_t*, float*,
                          csrspmm_b200_stream_t);
    size_t (*transpose_workspace_bytes)(int32_t, int64_t);
    int (*transpose)(int32_t, int32_t, int64_t, const int32_t*, const int32_t*, const float*, int32_t*, int32_t*, float*, void*, size_t,
                     csrspmm_b200_stream_t);
    int (*check_bounds)(int32_t, int32_t, int64_t, const int32_t*, const int32_t*, uint32_t*, csrspmm_b200_stream_t);
    int (*quantize)(int64_t, const float*, float*, uint8_t*, csrspmm_b200_stream_t);
};
Library g_lib = {};
PyObject* g_error = nullptr;  // _lib.SpmmError(status, where)

// A failed library call, turned into SpmmError at the Python boundary.
struct LibraryError {
    int status;
    const char* where;
};

void raise_library_error(const LibraryError& e)
{
    PyObject* exc = PyObject_CallFunction(g_error, "is", e.status, e.where);
    if (exc == nullptr) return;
    PyErr_SetObject(g_error, exc);
    Py_DECREF(exc);
}

void want(bool ok, const char* message)
{
    if (!ok) throw std::runtime_error(message);
}

const at::Tensor& tensor_of(PyObject* o, const char* name)
{
    if (!THPVariable_Check(o)) throw c10::TypeError({__func__, __FILE__, static_cast<uint32_t>(__LINE__)}, std::string(name) + " must be a tensor");
    return THPVariable_Unpack(o);
}

// The kernels take a leading dimension of at least the row's length.
bool rows_apart(const at::Tensor& t) { return t.size(0) <= 1 || t.stride(0) >= t.size(1); }

// The checks of the reference's wrappers, with its wording (torch_csrspmm/torch_csrspmm_naive.cpp:19-26).
void check_csr(const at::Tensor& rp, const at::Tensor& ci, const at::Tensor& va, const at::Tensor& B, bool packed)
{
    want(rp.is_cuda(), "A_row_ptr must be a CUDA tensor");
    want(ci.is_cuda(), "A_col_idx must be a CUDA tensor");
    want(va.is_cuda(), "A_values must be a CUDA tensor");
    want(B.is_cuda(), "B must be a CUDA tensor");
    want(rp.scalar_type() == at::kInt, "A_row_ptr must be int32");
    want(ci.scalar_type() == at::kInt, "A_col_idx must be int32");
    if (packed) want(va.scalar_type() == at::kByte, "packed A_values must be uint8");
    else want(va.scalar_type() == at::kFloat, "A_values must be float32");
    want(B.scalar_type() == at::kFloat, "B must be float32");
    want(B.dim() == 2 && rp.dim() == 1 && ci.dim() == 1 && va.dim() == 1 && rp.size(0) >= 1,
         "expected 1-D row_ptr/col_idx/values and 2-D B");
    want(rp.is_contiguous() && ci.is_contiguous() && va.is_contiguous(), "row_ptr, col_idx and values must be contiguous");
    want(B.stride(1) == 1 || B.size(1) <= 1, "B must be row-major (unit stride along its columns)");
    want(rows_apart(B), "B must be row-major (rows that do not overlap)");  // an expanded row: its storage ends after one
    const auto dev = B.device();
    want(rp.device() == dev && ci.device() == dev && va.device() == dev, "all tensors must be on the same device");
}

// Releases the GIL if this thread holds it (the registered operators run without it).
class WithoutGil {
public:
    WithoutGil() : state_(PyGILState_Check() ? PyEval_SaveThread() : nullptr) {}
    ~WithoutGil()
    {
        if (state_) PyEval_RestoreThread(state_);
    }
    WithoutGil(const WithoutGil&) = delete;
    WithoutGil& operator=(const WithoutGil&) = delete;

private:
    PyThreadState* state_;
};

template <class T>
T* address(const at::Tensor& t)
{
    return static_cast<T*>(t.data_ptr());
}

// Scratch of one call from torch's caching allocator, handed back when the call has been enqueued (the
// allocator keeps the block for the stream's next request).
class Scratch {
public:
    Scratch() = default;
    Scratch(const Scratch&) = delete;
    Scratch& operator=(const Scratch&) = delete;
    ~Scratch()
    {
        if (ptr_) c10::cuda::CUDACachingAllocator::raw_delete(ptr_);
    }
    void* get(size_t bytes, cudaStream_t stream)
    {
        ptr_ = c10::cuda::CUDACachingAllocator::raw_alloc_with_stream(std::max<size_t>(bytes, 256), stream);
        return ptr_;
    }
    // For scratch that only makes a call faster: null where memory has no room for it.
    void* get_if_room(size_t bytes, c10::cuda::CUDAStream stream)
    {
        namespace Allocator = c10::cuda::CUDACachingAllocator;
        const c10::DeviceIndex device = stream.device_index();
        int64_t active = -1;
        try {
            const auto stats = Allocator::getDeviceStats(device);
            active = stats.active_bytes[0].current;
            const int64_t reserved = stats.reserved_bytes[0].current;
            if (reserved - active < (int64_t)bytes) {  // not in torch's free blocks: what may it take, and what is there?
                if (Full::known(device, bytes, active)) return nullptr;
                constexpr int64_t kSegment = 2 << 20;  // what torch rounds larger allocations up to
                const int64_t want = ((int64_t)bytes + kSegment - 1) / kSegment * kSegment;
                const c10::cuda::CUDAStreamCaptureModeGuard relaxed{cudaStreamCaptureModeRelaxed};  // as torch does where it allocates
                size_t there = 0, total = 0;
                C10_CUDA_CHECK(cudaMemGetInfo(&there, &total));
                const int64_t allowed = (int64_t)(Allocator::getMemoryFraction(device) * (double)total) - reserved;
                if (reserved - active + std::min((int64_t)there, allowed) < want) {
                    Full::note(device, bytes, active);
                    return nullptr;
                }
            }
        } catch (const c10::Error&) {  // an allocator that does not tell
        }
        try {
            return get(bytes, stream);
        } catch (const c10::OutOfMemoryError&) {
            if (active >= 0) Full::note(device, bytes, active);
            return nullptr;
        }
    }

private:
    // Where there was no room for so many bytes a moment ago, with no more in use than now.  An allocation that fails makes torch
    // give all its free blocks back to the driver first, and asking the driver takes 200 us a time (200 000 rows of 24, 50 columns,
    // 101 us without the copy: 237 and 535 us a call), so a program that lives with full memory pays for one of them once a second.
    class Full {
    public:
        static bool known(c10::DeviceIndex device, size_t bytes, int64_t active)
        {
            if (device < 0 || device >= kDevices) return false;
            const std::lock_guard<std::mutex> lock(mutex_);
            const Full& f = full_[device];
            return bytes >= f.bytes_ && active >= f.active_ && Clock::now() < f.until_;
        }
        static void note(c10::DeviceIndex device, size_t bytes, int64_t active)
        {
            if (device < 0 || device >= kDevices) return;
            const std::lock_guard<std::mutex> lock(mutex_);
            Full& f = full_[device];
            const auto now = Clock::now();
            const bool fresh = now < f.until_;
            f.bytes_ = fresh ? std::min(f.bytes_, bytes) : bytes;
            f.active_ = fresh ? std::min(f.active_, active) : active;
            f.until_ = now + std::chrono::seconds(1);
        }

    private:
        using Clock = std::chrono::steady_clock;
        static constexpr int kDevices = 64;
        static inline std::mutex mutex_;
        static Full full_[kDevices];
        size_t bytes_ = 0;
        int64_t active_ = 0;
        Clock::time_point until_ = {};
    };

    void* ptr_ = nullptr;
};
Scratch::Full Scratch::Full::full_[kDevices];

struct Product {
    at::Tensor rp, ci, va, B, C;  // C undefined: allocate it
    at::Tensor workspace;         // undefined: take it from the allocator
    double alpha = 1.0, beta = 0.0;
    int entry = 0, kernel = 0;
    int max_row_nnz = 0;
    bool packed = false;
    double scale = 1.0;
    std::optional<int64_t> nnz;  // not given: col_idx's length
    int32_t* status_word = nullptr;
    const csrspmm_b200_schedule* schedule = nullptr;
    bool sync = false;
};

at::Tensor run_product(Product& q)
{
    check_csr(q.rp, q.ci, q.va, q.B, q.packed);
    const int64_t M = q.rp.size(0) - 1, Kd = q.B.size(0), Nd = q.B.size(1);
    const int64_t n = q.nnz.value_or(q.ci.size(0));
    if (q.packed) want(q.va.size(0) >= (n + 1) / 2, "packed values too short");
    else want(q.va.size(0) == n, "values and col_idx differ in length");
    want(q.ci.size(0) >= n, "col_idx too short");
    const c10::cuda::CUDAGuard guard(q.B.device());
    if (!q.C.defined()) {
        want(q.beta == 0.0, "beta != 0 needs C_out");
        q.C = at::detail::empty_cuda({M, Nd}, at::kFloat, q.B.device(), std::nullopt);
    } else {
        want(q.C.is_cuda() && q.C.scalar_type() == at::kFloat && q.C.dim() == 2 && q.C.size(0) == M && q.C.size(1) == Nd &&
                 q.C.device() == q.B.device(),
             "C_out must be a float32 CUDA tensor of shape (M, Nd) on B's device");
        want((q.C.stride(1) == 1 || Nd <= 1) && rows_apart(q.C), "C_out must be row-major");
    }
    csrspmm_b200_args a = {};
    a.struct_size = sizeof(a);
    a.M = static_cast<int32_t>(M);
    a.Kd = static_cast<int32_t>(Kd);
    a.Nd = static_cast<int32_t>(Nd);
    a.nnz = n;
    a.row_ptr = address<int32_t>(q.rp);
    a.col_idx = address<int32_t>(q.ci);
    a.values = q.va.data_ptr();
    a.value_format = q.packed ? CSRSPMM_B200_VALUES_E2M1 : CSRSPMM_B200_VALUES_F32;
    a.value_scale = q.packed ? static_cast<float>(q.scale) : 1.0f;
    a.B = address<float>(q.B);
    a.ldb = std::max(Kd > 1 ? q.B.stride(0) : Nd, Nd);
    a.C = address<float>(q.C);
    a.ldc = std::max(M > 1 ? q.C.stride(0) : Nd, Nd);
    a.alpha = static_cast<float>(q.alpha);
    a.beta = static_cast<float>(q.beta);
    a.entry = q.entry;
    a.kernel = q.kernel;
    a.max_row_nnz = q.max_row_nnz;
    a.status_word = q.status_word;
    a.schedule = q.schedule;

    const auto stream = c10::cuda::getCurrentCUDAStream(q.B.device().index());
    Scratch scratch;
    if (M > 0 && Nd > 0) {
        const int uses = g_lib.uses_workspace(&a);
        if (uses < 0) throw LibraryError{-uses, "csrspmm_b200_select_kernel"};
        if (uses > 0) {
            const size_t need = g_lib.workspace_bytes(&a);
            const size_t given = q.workspace.defined() ? q.workspace.nbytes() : 0;
            const auto use_given = [&] {
                a.workspace = q.workspace.data_ptr();
                a.workspace_bytes = given;
                if (q.workspace.is_cuda()) c10::cuda::CUDACachingAllocator::recordStream(q.workspace.storage().data_ptr(), stream);
            };
            const auto take = [&](void* memory, size_t bytes) {
                a.workspace = memory;
                a.workspace_bytes = std::max<size_t>(bytes, 256);
                return memory != nullptr;
            };
            const bool with_copy = Nd % 4 != 0 && need > (size_t)Kd * (size_t)Nd * 4;  // of B, which the product can do without
            try {
                if (q.workspace.defined() && given >= need) {
                    use_given();
                } else if (!with_copy) {
                    take(scratch.get(need, stream), need);
                } else if (!take(scratch.get_if_room(need, stream), need)) {
                    const size_t least = g_lib.least_workspace_bytes(&a);
                    if (given >= least && given > 0) use_given();
                    else if (least > 0) take(scratch.get(least, stream), least);
                }
            } catch (const c10::OutOfMemoryError&) {
                a.workspace = nullptr;  // the library's own pool may have it
            }
        }
    }
    int status;
    {
        // as under ctypes: a launch may wait for room in the stream's queue, and sync waits for the GPU
        const WithoutGil nogil;
        status = (q.sync ? g_lib.spmm_sync : g_lib.spmm)(&a, reinterpret_cast<csrspmm_b200_stream_t>(stream.stream()));
    }
    if (status != CSRSPMM_B200_OK) throw LibraryError{status, "csrspmm_b200_spmm"};
    return q.C;
}

// ---- the longest row behind a row_ptr tensor, measured once ----------------------------------------------
// One small kernel and a host read, remembered per (address, length, version, device) for the last 64
// matrices.  It only steers the kernel choice, so a stale entry -- another matrix later placed at the same
// address -- costs speed, never correctness.  The GIL guards the table.
struct LongestRow {
    const void* row_ptr;
    int64_t length;
    int64_t version;
    int device;
    int longest;
};
constexpr int kLongestRows = 64;
LongestRow g_longest[kLongestRows];
int g_longest_count = 0, g_longest_next = 0;

int longest_row(const at::Tensor& rp)
{
    if (!rp.is_cuda() || rp.scalar_type() != at::kInt || rp.dim() != 1 || rp.size(0) < 2 || !rp.is_contiguous()) return 0;
    const LongestRow key = {rp.data_ptr(), rp.size(0), rp.is_inference() ? 0 : (int64_t)rp._version(), rp.device().index(), 0};
    for (int k = 0; k < g_longest_count; ++k) {
        const LongestRow& e = g_longest[k];
        if (e.row_ptr == key.row_ptr && e.length == key.length && e.version == key.version && e.device == key.device) return e.longest;
    }
    const c10::cuda::CUDAGuard guard(rp.device());
    int64_t stats[4] = {0, 0, 0, 0};
    int status;
    {
        const auto stream = c10::cuda::getCurrentCUDAStream(rp.device().index());
        const WithoutGil nogil;
        status = g_lib.row_stats(static_cast<int32_t>(rp.size(0) - 1), address<int32_t>(rp), stats,
                                 reinterpret_cast<csrspmm_b200_stream_t>(stream.stream()));
    }
    if (status != CSRSPMM_B200_OK) throw LibraryError{status, "csrspmm_b200_row_stats_device"};
    LongestRow& e = g_longest[g_longest_next];
    e = key;
    e.longest = static_cast<int>(std::min<int64_t>(stats[0], INT32_MAX));
    g_longest_next = (g_longest_next + 1) % kLongestRows;
    g_longest_count = std::min(g_longest_count + 1, kLongestRows);
    return e.longest;
}

// ---- Python functions -----------------------------------------------------------------------------------

#define BEGIN_BINDING HANDLE_TH_ERRORS try {
#define END_BINDING                   \
    }                                 \
    catch (const LibraryError& e)     \
    {                                 \
        raise_library_error(e);       \
        return nullptr;               \
    }                                 \
    END_HANDLE_TH_ERRORS

double as_double(PyObject* o)
{
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return v;
}

long long as_integer(PyObject* o)
{
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}

// int(o): a whole number in any numeric type
long long as_int_of(PyObject* o)
{
    if (PyLong_Check(o)) return as_integer(o);
    const auto number = pybind11::reinterpret_steal<pybind11::object>(PyNumber_Long(o));
    if (!number) throw python_error();
    return as_integer(number.ptr());
}

void expect_args(Py_ssize_t got, Py_ssize_t wanted)
{
    if (got != wanted) throw std::runtime_error("csrspmm_b200 binding: wrong number of arguments");
}

// init(SpmmError, {name: address of csrspmm_b200_<name>})
PyObject* py_init(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    BEGIN_BINDING
    expect_args(nargs, 2);
    auto fill = [&](auto& fn, const char* name) {
        PyObject* o = PyDict_GetItemString(args[1], name);
        if (o == nullptr) throw std::runtime_error(std::string("csrspmm_b200 binding: no address for ") + name);
        fn = reinterpret_cast<std::decay_t<decltype(fn)>>(static_cast<uintptr_t>(as_integer(o)));
    };
    fill(g_lib.spmm, "spmm");
    fill(g_lib.spmm_sync, "spmm_sync");
    fill(g_lib.uses_workspace, "uses_workspace");
    fill(g_lib.workspace_bytes, "workspace_bytes");
    fill(g_lib.least_workspace_bytes, "least_workspace_bytes");
    fill(g_lib.row_stats, "row_stats_device");
    fill(g_lib.dense2csr_mask_bytes, "dense2csr_mask_bytes");
    fill(g_lib.dense2csr_count, "dense2csr_count_mask");
    fill(g_lib.dense2csr_fill, "dense2csr_fill_mask");
    fill(g_lib.quantize, "e2m1_quantize_device");
    fill(g_lib.transpose_workspace_bytes, "transpose_workspace_bytes");
    fill(g_lib.transpose, "transpose");
    fill(g_lib.check_bounds, "check_bounds_device");
    Py_INCREF(args[0]);
    Py_XSETREF(g_error, args[0]);
    Py_RETURN_NONE;
    END_BINDING
}

// spmm(row_ptr, col_idx, values, B, C|None, alpha, beta, entry, kernel, max_row_nnz, e2m1_scale|None, nnz|None,
//      workspace|None, status_word|None, sync, schedule handle) -> C
PyObject* py_spmm(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    BEGIN_BINDING
    expect_args(nargs, 16);
    Product q;
    q.rp = tensor_of(args[0], "A_row_ptr");
    q.ci = tensor_of(args[1], "A_col_idx");
    q.va = tensor_of(args[2], "A_values");
    q.B = tensor_of(args[3], "B");
    if (args[4] != Py_None) q.C = tensor_of(args[4], "C_out");
    q.alpha = as_double(args[5]);
    q.beta = as_double(args[6]);
    q.entry = static_cast<int>(as_int_of(args[7]));
    q.kernel = static_cast<int>(as_int_of(args[8]));
    q.max_row_nnz = static_cast<int>(as_int_of(args[9]));
    q.packed = args[10] != Py_None;
    if (q.packed) q.scale = as_double(args[10]);
    if (args[11] != Py_None) q.nnz = as_int_of(args[11]);
    if (args[12] != Py_None) q.workspace = tensor_of(args[12], "workspace");
    if (args[13] != Py_None) q.status_word = address<int32_t>(tensor_of(args[13], "status_word"));
    q.sync = PyObject_IsTrue(args[14]) == 1;
    q.schedule = reinterpret_cast<const csrspmm_b200_schedule*>(static_cast<uintptr_t>(as_integer(args[15])));
    return THPVariable_Wrap(run_product(q));
    END_BINDING
}

// op(entry, row_ptr, col_idx, values, B, alpha) -> new C: the reference's ops.  The longest row is measured, not
// believed: three of the reference's five ops carry no such argument, and a stale value passed to the other
// two would send a skewed matrix to the whole-row kernel.
PyObject* py_op(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    BEGIN_BINDING
    expect_args(nargs, 6);
    Product q;
    q.entry = static_cast<int>(as_integer(args[0]));
    q.rp = tensor_of(args[1], "A_row_ptr");
    q.ci = tensor_of(args[2], "A_col_idx");
    q.va = tensor_of(args[3], "A_values");
    q.B = tensor_of(args[4], "B");
    q.alpha = as_double(args[5]);
    q.max_row_nnz = longest_row(q.rp);
    return THPVariable_Wrap(run_product(q));
    END_BINDING
}

// enqueue(address of a csrspmm_b200_args, device index): a prepared product, on the device's current stream
PyObject* py_enqueue(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    BEGIN_BINDING
    expect_args(nargs, 2);
    const auto* a = reinterpret_cast<const csrspmm_b200_args*>(static_cast<uintptr_t>(as_integer(args[0])));
    const auto stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(as_integer(args[1])));
    int status;
    {
        const WithoutGil nogil;
        status = g_lib.spmm(a, reinterpret_cast<csrspmm_b200_stream_t>(stream.stream()));
    }
    if (status != CSRSPMM_B200_OK) throw LibraryError{status, "csrspmm_b200_spmm"};
    Py_RETURN_NONE;
    END_BINDING
}

at::Tensor new_array(int64_t n, at::ScalarType type, at::Device device)
{
    return at::detail::empty_cuda({n}, type, device, std::nullopt);
}

csrspmm_b200_stream_t current_stream(at::Device device)
{
    return reinterpret_cast<csrspmm_b200_stream_t>(c10::cuda::getCurrentCUDAStream(device.index()).stream());
}

void check(int status, const char* where)
{
    if (status != CSRSPMM_B200_OK) throw LibraryError{status, where};
}

// dense2csr(dense, tol) -> (row_ptr, col_idx, values, longest row)
PyObject* py_dense2csr(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    BEGIN_BINDING
    expect_args(nargs, 2);
    const at::Tensor dense = tensor_of(args[0], "dense");
    const float tol = static_cast<float>(as_double(args[1]));
    want(dense.is_cuda() && dense.scalar_type() == at::kFloat && dense.dim() == 2 && (dense.stride(1) == 1 || dense.size(1) <= 1) && rows_apart(dense),
         "dense must be a row-major float32 CUDA matrix");
    const int64_t H = dense.size(0), W = dense.size(1);
    const int64_t ld = std::max(H > 1 ? dense.stride(0) : W, W);
    const auto device = dense.device();
    const c10::cuda::CUDAGuard guard(device);
    at::Tensor rp = new_array(H + 1, at::kInt, device), ci, va;
    int64_t nnz = 0;
    int32_t longest = 0;
    {
        const WithoutGil nogil;
        const auto stream = current_stream(device);
        const float* data = address<float>(dense);
        Scratch scratch;
        const size_t mask_bytes = g_lib.dense2csr_mask_bytes((int32_t)H, (int32_t)W);  // a bit per element, or without
        uint32_t* const mask = static_cast<uint32_t*>(scratch.get_if_room(mask_bytes, c10::cuda::getCurrentCUDAStream(device.index())));
        check(g_lib.dense2csr_count((int32_t)H, (int32_t)W, data, ld, tol, address<int32_t>(rp), mask, &nnz, &longest, stream),
              "csrspmm_b200_dense2csr_count");
        ci = new_array(nnz, at::kInt, device);
        va = new_array(nnz, at::kFloat, device);
        if (nnz > 0)
            check(g_lib.dense2csr_fill((int32_t)H, (int32_t)W, data, ld, tol, mask, address<int32_t>(rp), address<int32_t>(ci),
                                       address<float>(va), stream),
                  "csrspmm_b200_dense2csr_fill");
    }
    return Py_BuildValue("(NNNi)", THPVariable_Wrap(rp), THPVariable_Wrap(ci), THPVariable_Wrap(va), (int)longest);
    END_BINDING
}

// quantize(values: contiguous float32 on the GPU) -> (packed, scale)
PyObject* py_quantize(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    BEGIN_BINDING
    expect_args(nargs, 1);
    const at::Tensor v = tensor_of(args[0], "values");
    want(v.is_cuda() && v.scalar_type() == at::kFloat && v.is_contiguous(), "values must be a contiguous float32 CUDA tensor");
    const int64_t n = v.numel();
    const c10::cuda::CUDAGuard guard(v.device());
    at::Tensor packed = new_array((n + 1) / 2, at::kByte, v.device());
    float scale = 1.0f;
    {
        const WithoutGil nogil;
        check(g_lib.quantize(n, address<float>(v), &scale, address<uint8_t>(packed), current_stream(v.device())),
              "csrspmm_b200_e2m1_quantize_device");
    }
    return Py_BuildValue("(Nd)", THPVariable_Wrap(packed), (double)scale);
    END_BINDING
}

// (row_ptr, col_idx, values) of A^T
std::tuple<at::Tensor, at::Tensor, at::Tensor> transpose(const at::Tensor& rp, const at::Tensor& ci, const at::Tensor& va, int64_t Kd)
{
    want(rp.is_cuda() && ci.is_cuda() && va.is_cuda() && ci.device() == rp.device() && va.device() == rp.device(),
         "row_ptr, col_idx and values must be CUDA tensors on one device");
    want(rp.scalar_type() == at::kInt && ci.scalar_type() == at::kInt && va.scalar_type() == at::kFloat,
         "row_ptr and col_idx must be int32, values float32");
    want(rp.dim() == 1 && ci.dim() == 1 && va.dim() == 1 && rp.size(0) >= 1 && ci.size(0) == va.size(0) && rp.is_contiguous() &&
             ci.is_contiguous() && va.is_contiguous(),
         "expected contiguous 1-D row_ptr, col_idx and values");
    want(Kd >= 0 && Kd < INT32_MAX && rp.size(0) <= INT32_MAX, "a matrix has fewer than 2^31 - 1 rows and columns");
    const auto device = rp.device();
    const c10::cuda::CUDAGuard guard(device);
    const int64_t nnz = ci.size(0);
    at::Tensor t_rp = new_array(Kd + 1, at::kInt, device), t_ci = new_array(nnz, at::kInt, device), t_va = new_array(nnz, at::kFloat, device);
    const auto stream = c10::cuda::getCurrentCUDAStream(device.index());
    const size_t need = g_lib.transpose_workspace_bytes((int32_t)Kd, nnz);
    Scratch scratch;
    void* ws = scratch.get(need, stream);
    int status;
    {
        const WithoutGil nogil;
        status = g_lib.transpose((int32_t)(rp.size(0) - 1), (int32_t)Kd, nnz, address<int32_t>(rp), address<int32_t>(ci), address<float>(va),
                                 address<int32_t>(t_rp), address<int32_t>(t_ci), address<float>(t_va), ws, std::max<size_t>(need, 256),
                                 reinterpret_cast<csrspmm_b200_stream_t>(stream.stream()));
    }
    check(status, "csrspmm_b200_transpose");
    return {t_rp, t_ci, t_va};
}

// transpose(row_ptr, col_idx, values, Kd) -> (row_ptr, col_idx, values) of A^T, waiting: the kernels clamp columns out of
// range, which transpose_csr's code for the host cannot place and refuses
PyObject* py_transpose(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    BEGIN_BINDING
    expect_args(nargs, 4);
    const at::Tensor rp = tensor_of(args[0], "row_ptr"), ci = tensor_of(args[1], "col_idx");
    const int64_t Kd = as_integer(args[3]), nnz = ci.numel();
    const auto t = transpose(rp, ci, tensor_of(args[2], "values"), Kd);
    {
        const WithoutGil nogil;
        const c10::cuda::CUDAGuard guard(rp.device());
        uint32_t problems = 0;
        check(g_lib.check_bounds((int32_t)(rp.size(0) - 1), (int32_t)Kd, nnz, address<int32_t>(rp), address<int32_t>(ci), &problems,
                                 current_stream(rp.device())),
              "csrspmm_b200_transpose");
    }
    return Py_BuildValue("(NNN)", THPVariable_Wrap(std::get<0>(t)), THPVariable_Wrap(std::get<1>(t)), THPVariable_Wrap(std::get<2>(t)));
    END_BINDING
}

// ---- torch.ops.csrspmm_b200 (schemas and fake implementations: csrspmm_b200/torch_library.py) ---------------
// Registered here and not through torch.library.custom_op, whose Python layers cost more per call than a
// product of a sampled subgraph takes on the GPU.

// A failed library call leaves an operator as SpmmError too.
template <class F>
auto as_operator(F&& body)
{
    try {
        return body();
    } catch (const LibraryError& e) {
        pybind11::gil_scoped_acquire gil;
        raise_library_error(e);
        throw pybind11::error_already_set();
    }
}

int kernel_id(c10::string_view name)
{
    if (name == "auto") return CSRSPMM_B200_KERNEL_AUTO;
    if (name == "row") return CSRSPMM_B200_KERNEL_ROW;
    if (name == "merge") return CSRSPMM_B200_KERNEL_MERGE;
    if (name == "tma") return CSRSPMM_B200_KERNEL_TMA;
    throw std::runtime_error("unknown kernel '" + std::string(name) + "' (auto, row, merge or tma)");
}

at::Tensor op_spmm(const at::Tensor& rp, const at::Tensor& ci, const at::Tensor& va, const at::Tensor& B, double alpha, c10::string_view kernel)
{
    return as_operator([&] {
        Product q;
        q.rp = rp, q.ci = ci, q.va = va, q.B = B.contiguous();
        q.alpha = alpha;
        q.kernel = kernel_id(kernel);
        return run_product(q);
    });
}

void op_spmm_inplace(const at::Tensor& rp, const at::Tensor& ci, const at::Tensor& va, const at::Tensor& B, const at::Tensor& C, double alpha,
                     double beta, c10::string_view kernel)
{
    as_operator([&] {
        Product q;
        q.rp = rp, q.ci = ci, q.va = va, q.B = B, q.C = C;
        q.alpha = alpha, q.beta = beta;
        q.kernel = kernel_id(kernel);
        return run_product(q);
    });
}

std::tuple<at::Tensor, at::Tensor, at::Tensor> op_transpose(const at::Tensor& rp, const at::Tensor& ci, const at::Tensor& va, c10::SymInt Kd)
{
    return as_operator([&] { return transpose(rp, ci, va, Kd.expect_int()); });
}

at::Tensor call_spmm(const at::Tensor& rp, const at::Tensor& ci, const at::Tensor& va, const at::Tensor& B, double alpha, c10::string_view kernel)
{
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("csrspmm_b200::spmm", "").typed<decltype(op_spmm)>();
    return op.call(rp, ci, va, B, alpha, kernel);
}

std::tuple<at::Tensor, at::Tensor, at::Tensor> call_transpose(const at::Tensor& rp, const at::Tensor& ci, const at::Tensor& va, c10::SymInt Kd)
{
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("csrspmm_b200::transpose", "").typed<decltype(op_transpose)>();
    return op.call(rp, ci, va, Kd);
}

// dB = alpha * A^T dC
struct SpmmWithGradient : torch::autograd::Function<SpmmWithGradient> {
    static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& rp, const at::Tensor& ci, const at::Tensor& va,
                              const at::Tensor& B, double alpha, std::string kernel)
    {
        ctx->save_for_backward({rp, ci, va});
        ctx->saved_data["Kd"] = B.sym_size(0);
        ctx->saved_data["alpha"] = alpha;
        ctx->saved_data["kernel"] = kernel;
        ctx->saved_data["values_need_grad"] = va.requires_grad();
        at::AutoDispatchBelowADInplaceOrView below;
        return call_spmm(rp, ci, va, B, alpha, kernel);
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads)
    {
        if (ctx->saved_data["values_need_grad"].toBool())
            throw std::runtime_error("csrspmm_b200::spmm has no gradient for the stored values of A");
        torch::autograd::variable_list out(6);
        if (ctx->needs_input_grad(3) && grads[0].defined()) {
            const auto saved = ctx->get_saved_variables();
            const auto t = call_transpose(saved[0], saved[1], saved[2], ctx->saved_data["Kd"].toSymInt());
            out[3] = call_spmm(std::get<0>(t), std::get<1>(t), std::get<2>(t), grads[0].contiguous(), ctx->saved_data["alpha"].toDouble(),
                               ctx->saved_data["kernel"].toStringRef());
        }
        return out;
    }
};

// ---- CsrMatrix @ B with a gradient for B ------------------------------------------------------------------
// A node of its own and not a Python autograd.Function: what the Python layers cost per step, forward and backward,
// is as much as the two products of a small graph (2466 rows of 8, 160 columns: 72 -> 50 us per step, about what torch
// takes for one multiplication and its gradient).  The backward product asks the matrix for its transpose, which it
// builds once and keeps.

class CsrMatmulBackward : public torch::autograd::Node {
public:
    CsrMatmulBackward(PyObject* matrix, double alpha, int kernel) : matrix_(matrix), alpha_(alpha), kernel_(kernel) { Py_INCREF(matrix_); }
    ~CsrMatmulBackward() override
    {
        if (!Py_IsInitialized()) return;
        pybind11::gil_scoped_acquire gil;
        Py_DECREF(matrix_);
    }
    std::string name() const override { return "CsrMatmulBackward"; }

    torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override
    {
        if (!grads[0].defined()) return {at::Tensor()};
        return as_operator([&]() -> torch::autograd::variable_list {
            const at::NoGradGuard no_grad;
            pybind11::gil_scoped_acquire gil;
            Product q;
            q.B = grads[0].contiguous();
            q.alpha = alpha_;
            q.kernel = kernel_;
            // (row_ptr, col_idx, values, longest row, schedule handle) of the transpose
            PyObject* parts = PyObject_CallMethod(matrix_, "_transpose_parts", "Li", (long long)q.B.size(1), kernel_);
            if (parts == nullptr) throw pybind11::error_already_set();
            const auto owned = pybind11::reinterpret_steal<pybind11::object>(parts);
            q.rp = tensor_of(PyTuple_GetItem(parts, 0), "row_ptr");
            q.ci = tensor_of(PyTuple_GetItem(parts, 1), "col_idx");
            q.va = tensor_of(PyTuple_GetItem(parts, 2), "values");
            q.max_row_nnz = static_cast<int>(as_integer(PyTuple_GetItem(parts, 3)));
            q.schedule = reinterpret_cast<const csrspmm_b200_schedule*>(static_cast<uintptr_t>(as_integer(PyTuple_GetItem(parts, 4))));
            return {run_product(q)};
        });
    }

private:
    PyObject* matrix_;
    double alpha_;
    int kernel_;
};

// matmul(matrix, row_ptr, col_idx, values, B, alpha, kernel, longest row, schedule handle) -> C
PyObject* py_matmul(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    BEGIN_BINDING
    expect_args(nargs, 9);
    const at::Tensor B = tensor_of(args[4], "B");
    // the product runs on an address and the node has no jvp: a tangent of B would be dropped without a word
    TORCH_CHECK_NOT_IMPLEMENTED(!torch::autograd::isFwGradDefined(B), "CsrMatrix @ B has no forward-mode derivative");
    Product q;
    q.rp = tensor_of(args[1], "A_row_ptr");
    q.ci = tensor_of(args[2], "A_col_idx");
    q.va = tensor_of(args[3], "A_values");
    q.alpha = as_double(args[5]);
    q.kernel = static_cast<int>(as_integer(args[6]));
    q.max_row_nnz = static_cast<int>(as_integer(args[7]));
    q.schedule = reinterpret_cast<const csrspmm_b200_schedule*>(static_cast<uintptr_t>(as_integer(args[8])));
    at::Tensor C;
    {
        const at::NoGradGuard no_grad;
        q.B = B.contiguous();
        C = run_product(q);
    }
    if (at::GradMode::is_enabled() && B.requires_grad()) {
        std::shared_ptr<CsrMatmulBackward> node(new CsrMatmulBackward(args[0], q.alpha, q.kernel), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(B));
        torch::autograd::set_history(C, node);
    }
    return THPVariable_Wrap(C);
    END_BINDING
}

at::Tensor autograd_spmm(const at::Tensor& rp, const at::Tensor& ci, const at::Tensor& va, const at::Tensor& B, double alpha,
                         c10::string_view kernel)
{
    return SpmmWithGradient::apply(rp, ci, va, B, alpha, std::string(kernel));
}

TORCH_LIBRARY_IMPL(csrspmm_b200, CUDA, m)
{
    m.impl("spmm", op_spmm);
    m.impl("spmm_", op_spmm_inplace);
    m.impl("transpose", op_transpose);
}

TORCH_LIBRARY_IMPL(csrspmm_b200, Autograd, m) { m.impl("spmm", autograd_spmm); }

// The dispatcher does not raise the version counter of a tensor that a schema names as written, and the kernel writes
// through an address: without this a C that a backward saved and spmm_ overwrote would give a wrong gradient.
void spmm_inplace_marking(const at::Tensor& rp, const at::Tensor& ci, const at::Tensor& va, const at::Tensor& B, const at::Tensor& C,
                          double alpha, double beta, c10::string_view kernel)
{
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("csrspmm_b200::spmm_", "").typed<decltype(op_spmm_inplace)>();
    if (!C.is_inference()) torch::autograd::increment_version(C);
    at::AutoDispatchBelowADInplaceOrView below;
    op.call(rp, ci, va, B, C, alpha, beta, kernel);
}

TORCH_LIBRARY_IMPL(csrspmm_b200, ADInplaceOrView, m) { m.impl("spmm_", spmm_inplace_marking); }

#define FASTCALL(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(f)), METH_FASTCALL
PyMethodDef g_methods[] = {
    {"init", FASTCALL(py_init), nullptr},
    {"spmm", FASTCALL(py_spmm), nullptr},
    {"op", FASTCALL(py_op), nullptr},
    {"enqueue", FASTCALL(py_enqueue), nullptr},
    {"dense2csr", FASTCALL(py_dense2csr), nullptr},
    {"quantize", FASTCALL(py_quantize), nullptr},
    {"transpose", FASTCALL(py_transpose), nullptr},
    {"matmul", FASTCALL(py_matmul), nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_torch_binding", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_binding() { return PyModule_Create(&g_module); }
