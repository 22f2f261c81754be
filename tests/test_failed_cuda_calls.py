"""Every CUDA call of an entry point fails once (tests/cpp/fake_cudart.cpp stands in for the runtime: no GPU): the entry
point has to report it, free what it took exactly once, and leave nothing running that writes to host memory it lent out."""
import ctypes as C

import numpy as np
import pytest

from csrspmm_b200 import _lib, build


@pytest.fixture(scope="module")
def fake():
    L = C.CDLL(str(build.build_fake_runtime()))
    for name in ("fake_calls", "fake_live", "fake_bad_frees", "fake_busy"):
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


CALLS = {"schedule": _schedule}


@pytest.mark.parametrize("name", sorted(CALLS))
def test_one_failed_call(fake, name):
    keep = {}
    run = lambda: CALLS[name](fake, keep)
    fake.fake_reset(0)
    assert run() == 0 and fake.fake_bad_frees() == 0
    fake.fake_reset(0)
    assert run() == 0
    calls, live = fake.fake_calls(), fake.fake_live()
    assert calls > 3
    for k in range(1, calls + 1):
        fake.fake_reset(k)
        status = run()
        assert status in (0, _lib.ERR_CUDA), (k, status)  # 0: the call has another way to go on
        assert fake.fake_bad_frees() == 0, f"call {k} of {calls} fails: something is freed twice"
        assert fake.fake_live() == live, f"call {k} of {calls} fails: something is not freed"
