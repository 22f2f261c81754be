"""Every CUDA call of an entry point fails once (tests/cpp/fake_cudart.cpp stands in for the runtime: no GPU): the entry
point has to report it, free what it took exactly once, and leave nothing running that writes to host memory it lent out."""
import ctypes as C

import numpy as np
import pytest

from csrspmm_b200 import _lib, build


@pytest.fixture(scope="module")
def fake():
    L = C.CDLL(str(build.build_fake_runtime()))
    for name in ("fake_calls", "fake_live", "fake_bad_frees", "fake_busy", "fake_streams", "fake_settings", "fake_refused"):
        getattr(L, name).restype = C.c_long
    L.fake_reset.argtypes = [C.c_long]
    return L


def _csr(M, Kd, per_row):
    rng = np.random.default_rng(0)
    rp = (np.arange(M + 1) * per_row).astype(np.int32)
    return rp, np.sort(rng.integers(0, Kd, (M, per_row)), axis=1).astype(np.int32).ravel(), np.ones(M * per_row, np.float32)


def _schedule(L, keep):
    M, Kd, Nd = 600, 5000, 64
    rp, ci, _ = keep.setdefault("csr", _csr(M, Kd, 50))
    a = _lib.make_args(M, Kd, Nd, len(ci), rp.ctypes.data, ci.ctypes.data)
    opt = _lib.ScheduleOptions(C.sizeof(_lib.ScheduleOptions), 16, 1000, 32)
    handle = C.c_void_p()
    status = L.csrspmm_b200_schedule_create(C.byref(a), C.byref(opt), C.byref(handle), None)
    if status == 0:
        L.csrspmm_b200_schedule_destroy(handle)
    return status


def _operands(keep, M, Kd, Nd, per_row):
    if not keep:
        keep["csr"] = _csr(M, Kd, per_row)
        keep["B"], keep["C"] = np.zeros((Kd, Nd), np.float32), np.zeros((M, Nd), np.float32)
    rp, ci, va = keep["csr"]
    return _lib.make_args(M, Kd, Nd, len(ci), rp.ctypes.data, ci.ctypes.data, va.ctypes.data, keep["B"].ctypes.data, keep["C"].ctypes.data,
                          alpha=1.0, beta=0.5)


def _spmm(L, keep):  # split rows, scratch from the library
    return L.csrspmm_b200_spmm(C.byref(_operands(keep, 3000, 500, 64, 20)), None)


def _tiled(L, keep):
    return L.csrspmm_b200_spmm_tiled(C.byref(_operands(keep, 3000, 500, 64, 20)), 100, None)


def _host_blocks(L, keep):
    return L.csrspmm_b200_spmm_host(C.byref(_operands(keep, 5000, 16, 1024, 4)), None, C.c_size_t(0), None)


def _host_panels(L, keep):
    return L.csrspmm_b200_spmm_host(C.byref(_operands(keep, 4000, 4000, 1024, 4)), None, C.c_size_t(0), None)


def _row_stats(L, keep):
    rp = keep.setdefault("csr", _csr(700, 50, 3))[0]
    return L.csrspmm_b200_row_stats_device(700, C.c_void_p(rp.ctypes.data), (C.c_int64 * 4)(), None)


def _validate(L, keep):
    rp, ci, _ = keep.setdefault("csr", _csr(700, 50, 3))
    return L.csrspmm_b200_validate_csr_device(700, 50, C.c_int64(len(ci)), C.c_void_p(rp.ctypes.data), C.c_void_p(ci.ctypes.data), C.byref(C.c_uint32()), None)


def _bounds(L, keep):
    rp, ci, _ = keep.setdefault("csr", _csr(700, 50, 3))
    return L.csrspmm_b200_check_bounds_device(700, 50, C.c_int64(len(ci)), C.c_void_p(rp.ctypes.data), C.c_void_p(ci.ctypes.data), C.byref(C.c_uint32()), None)


def _dense2csr(L, keep):  # two launches of the scan
    dense, rp = keep.setdefault("d", (np.zeros((9000, 4), np.float32), np.zeros(9001, np.int32)))
    return L.csrspmm_b200_dense2csr_count(9000, 4, C.c_void_p(dense.ctypes.data), C.c_int64(4), C.c_float(0), C.c_void_p(rp.ctypes.data),
                                          C.byref(C.c_int64()), C.byref(C.c_int32()), None)


def _quantize(L, keep):
    v, packed = keep.setdefault("q", (np.ones(5000, np.float32), np.zeros(2500, np.uint8)))
    status = L.csrspmm_b200_e2m1_quantize_device(C.c_int64(5000), C.c_void_p(v.ctypes.data), C.byref(C.c_float()), C.c_void_p(packed.ctypes.data), None)
    return 0 if status == _lib.ERR_BAD_ARG else status  # no kernel has written a scale


def _scale(L, keep):
    v = keep.setdefault("q", np.ones(5000, np.float32))
    return L.csrspmm_b200_e2m1_scale_device(C.c_int64(5000), C.c_void_p(v.ctypes.data), C.byref(C.c_float()), None)


def _transpose(L, keep, Kd=70_000):  # through buckets
    M, n = 3000, 300_000
    if not keep:
        keep["csr"] = _csr(M, Kd, 100)
        keep["out"] = np.zeros(Kd + 1, np.int32), np.zeros(n, np.int32), np.zeros(n, np.float32)
        L.csrspmm_b200_transpose_workspace_bytes.restype = C.c_size_t
        keep["bytes"] = L.csrspmm_b200_transpose_workspace_bytes(Kd, C.c_int64(n))
        keep["ws"] = np.zeros(keep["bytes"] + 256, np.uint8)
    at = lambda x: C.c_void_p(x.ctypes.data)
    return L.csrspmm_b200_transpose(M, Kd, C.c_int64(n), *map(at, keep["csr"]), *map(at, keep["out"]), C.c_void_p((keep["ws"].ctypes.data + 255) // 256 * 256),
                                    C.c_size_t(keep["bytes"]), None)


def _transpose_digits(L, keep):
    return _transpose(L, keep, 600_000)  # three passes, with the scan


# the entry points that lend host memory to the GPU (the caller's operands, page-locked words that the next call gets), and
# the others, which read results back by copies to pageable memory, complete when the copy returns
LENDING = {"schedule": _schedule, "host_blocks": _host_blocks, "host_panels": _host_panels, "row_stats": _row_stats, "dense2csr": _dense2csr,
           "quantize": _quantize, "bounds": _bounds}
CALLS = dict(LENDING, spmm=_spmm, tiled=_tiled, transpose=_transpose, transpose_digits=_transpose_digits, validate=_validate, scale=_scale)


@pytest.mark.parametrize("name", sorted(CALLS))
def test_one_failed_call(fake, name):
    keep = {}
    run = lambda: CALLS[name](fake, keep)
    fake.fake_reset(0)
    assert run() == 0 and fake.fake_bad_frees() == 0
    fake.fake_reset(0)
    assert run() == 0
    calls, live = fake.fake_calls(), fake.fake_live()
    assert calls >= 2
    for k in range(1, calls + 1):
        fake.fake_reset(k)
        status = run()
        assert status in (0, _lib.ERR_CUDA), (k, status)  # 0: the call has another way to go on
        assert fake.fake_bad_frees() == 0, f"call {k} of {calls} fails: something is freed twice"
        assert fake.fake_live() == live, f"call {k} of {calls} fails: something is not freed"
        assert name not in LENDING or fake.fake_busy() == 0, f"call {k} of {calls} fails: work is still running"


def test_shared_memory_is_asked_for_once(fake):
    fake.fake_reset(0)
    keep, digits = {}, {}
    for _ in range(2):
        assert _transpose(fake, keep) == 0 and _transpose_digits(fake, digits) == 0
    before = fake.fake_settings()
    assert before > 0 and _transpose(fake, keep) == 0 and _transpose_digits(fake, digits) == 0 and fake.fake_settings() == before
    assert fake.fake_refused() == 0  # and no launch, in any test so far, took more than it had asked for


def test_kept_streams_are_bounded_and_given_back(fake):
    import threading
    fake.fake_reset(0)
    assert fake.csrspmm_b200_release_memory(None) == 0 and fake.fake_streams() == 0
    start = threading.Barrier(6)

    def work():
        keep = {}
        start.wait()
        for _ in range(3):
            assert _host_blocks(fake, keep) == 0

    threads = [threading.Thread(target=work) for _ in range(6)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert 2 <= fake.fake_streams() <= 4  # two sets of two
    assert fake.csrspmm_b200_release_memory(None) == 0 and fake.fake_streams() == 0
