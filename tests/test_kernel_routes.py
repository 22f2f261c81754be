"""Which compiled kernels the entry points launch (tests/cpp/fake_cudart.cpp stands in for the runtime: no GPU)."""
import ctypes as C
import re

import pytest

from csrspmm_b200 import _lib, build


@pytest.fixture(scope="module")
def fake():
    L = C.CDLL(str(build.build_fake_runtime()))
    for name in ("fake_kernels", "fake_launched"):
        getattr(L, name).restype = C.c_size_t
    L.fake_reset.argtypes = [C.c_long]
    return L


def _names(function):
    text = C.create_string_buffer(function(None))
    function(text)
    return set(text.value.decode().split("\n")) - {""}


def _spmm(L, M, Kd, Nd, nnz, at=4096, **kw):  # nothing is read: no kernel runs
    a = _lib.make_args(M, Kd, Nd, nnz, 4096, 4096, 4096, at, at, workspace=4096, workspace_bytes=1 << 40, **kw)
    return L.csrspmm_b200_spmm(C.byref(a), None)


# rows of B in flight and CTAs per SM of the row kernel on long rows, by width and by the grid's CTAs per SM
@pytest.mark.parametrize("Nd,lanes,ctas,want", [
    (20, 8, 3, (8, 6)), (32, 8, 4, (16, 4)), (20, 8, 6, (8, 6)), (20, 8, 6.5, (4, 8)), (32, 8, 7, (8, 7)), (32, 8, 7.1, (4, 8)), (20, 8, 9, (8, 6)),
    (32, 8, 12.1, (4, 8)), (48, 16, 4, (16, 4)), (48, 16, 5, (4, 8)), (64, 16, 6, (8, 6)), (48, 16, 6.5, (4, 8)), (64, 16, 6.5, (8, 7)),
    (36, 16, 9, (8, 6)), (64, 16, 12, (8, 6)), (100, 32, 4, (16, 4)), (128, 32, 5, (4, 8)), (100, 32, 9, (8, 6)), (128, 32, 8, (4, 8)),
    (200, 32, 4, (6, 4)), (200, 32, 9, (6, 4)), (256, 32, 10.1, (2, 8)), (400, 32, 5, (4, 3)), (512, 32, 9, (4, 3)), (512, 32, 7, (3, 4))])
@pytest.mark.parametrize("fmt", [_lib.VALUES_F32, _lib.VALUES_E2M1])
def test_builds_of_the_row_kernel(fake, Nd, lanes, ctas, want, fmt):
    M = int(148 * ctas * 128 // lanes)
    fake.fake_reset(0)
    assert _spmm(fake, M, 2000, Nd, M * 70, kernel=_lib.KERNEL_ROW, value_format=fmt) == 0
    (name,) = _names(fake.fake_launched)
    G, NV, VW, U, FMT, FULL, MINB = re.search(r"spmm_row_kernel<(.*?)>", name).group(1).split(", ")
    assert (int(U), int(MINB)) == want and int(G) == lanes and int(VW) == 4 and int(FMT) == fmt and (FULL == "true") == (Nd // 4 == lanes * int(NV))
