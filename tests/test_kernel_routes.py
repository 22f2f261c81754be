"""Which compiled kernels the entry points launch (tests/cpp/fake_cudart.cpp stands in for the runtime: no GPU)."""
import ctypes as C
import itertools
import re

import pytest

from csrspmm_b200 import _lib, build
from test_failed_cuda_calls import CALLS
from test_gpu_transpose import BUCKETS, DIGITS, SIZES


@pytest.fixture(scope="module")
def fake():
    L = C.CDLL(str(build.build_fake_runtime()))
    for name in ("fake_kernels", "fake_launched", "csrspmm_b200_transpose_workspace_bytes"):
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


# products of every width class and alignment, on grids from a part of a wave to many, of short and long rows, with and without a
# longest row, few columns of A and many uses of a row of B among them
def _products():
    widths = (1, 2, 3, 4, 6, 7, 8, 10, 12, 13, 16, 20, 22, 25, 30, 32, 33, 48, 50, 63, 64, 90, 100, 127, 128, 131, 150, 200, 255, 256, 300, 501, 510, 512, 600, 1030)
    for Nd, waves, mean in itertools.product(widths, (0.1, 2, 5, 6.5, 8.5, 9.5, 11, 40), (4, 60, 125, 300)):
        lanes = 8 if Nd <= 32 else 16 if Nd <= 64 else 32
        M = int(148 * waves * 128 / lanes)
        for Kd, longest, at in itertools.product((60, 500, 2000, 1 << 20), (0, 2 * mean), (4096, 4104, 4100)):
            yield M, Kd, Nd, M * mean, longest, at
    yield 50_000, 2000, 30, 2_100_000, 0, 4096  # just over a wave of the largest tiles, on a copy of B


def _transpose(L, M, Kd, nnz):
    at = C.c_void_p(4096)  # nothing is read
    need = L.csrspmm_b200_transpose_workspace_bytes(Kd, C.c_int64(nnz))
    return L.csrspmm_b200_transpose(M, Kd, C.c_int64(nnz), at, at, at, at, at, at, at, C.c_size_t(need), None)


def test_nothing_is_compiled_that_no_call_launches(fake):
    """The builds of products without a schedule and of the transposition."""
    every = {k for k in _names(fake.fake_kernels) if re.search(r"spmm_(merge|row|resident|tma|fixup)_kernel|pad_rows|transpose_", k)}
    every = {k for k in every if not re.search(r"spmm_merge_kernel<.*, true, 0>", k)}  # launched beside the pieces of a schedule
    fake.fake_reset(0)
    for M, Kd, Nd, nnz, longest, at in _products():
        for kernel, fmt in itertools.product((_lib.KERNEL_ROW, _lib.KERNEL_MERGE, _lib.KERNEL_TMA), (_lib.VALUES_F32, _lib.VALUES_E2M1)):
            _spmm(fake, M, Kd, Nd, nnz, at, kernel=kernel, max_row_nnz=longest, value_format=fmt)
    for nnz, bits in itertools.product((1, 3000, 9000, 100_000, 1_000_000, 1_900_000, 6_000_000), range(1, 27)):
        assert _transpose(fake, 1000, 1 << bits, nnz) == 0
    assert sorted(every - _names(fake.fake_launched)) == []


def test_gpu_tests_run_every_kernel_of_the_transposition(fake):
    fake.fake_reset(0)
    for M, Kd, nnz, _ in (*SIZES, *BUCKETS, *DIGITS):
        assert _transpose(fake, M, Kd, nnz) == 0
    assert sorted({k for k in _names(fake.fake_kernels) if "transpose_" in k} - _names(fake.fake_launched)) == []


@pytest.mark.parametrize("size", DIGITS)
def test_sizes_of_the_digit_passes_take_them(fake, size):
    fake.fake_reset(0)
    assert _transpose(fake, *size[:3]) == 0
    launched = _names(fake.fake_launched)
    assert any("transpose_scatter_kernel" in k for k in launched) and not any("bucket" in k for k in launched)


def test_failed_calls_of_the_transposition_take_both_ways(fake):
    for name, kernels in (("transpose", ("bucket_count", "bucket_offsets", "bucket_scatter", "chunk_count", "bucket_sort")),
                          ("transpose_digits", ("transpose_count", "transpose_scatter", "scan_tiles", "scan_finish", "row_ptr"))):
        fake.fake_reset(0)
        assert CALLS[name](fake, {}) == 0
        launched = _names(fake.fake_launched)
        assert all(any(k in full for full in launched) for k in kernels), (name, launched)
