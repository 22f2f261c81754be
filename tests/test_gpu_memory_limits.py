"""Scratch that only makes a call faster (a padded copy of B, a bit per element of a matrix) where memory has no room for it: the
call does without.  The limit is torch's own, on what this process takes."""
import ctypes
import time

import numpy as np
import pytest
import torch

import oracle
from csrspmm_b200 import generators as G, ops

pytestmark = pytest.mark.gpu


@pytest.fixture
def limit_memory(cuda_lib):
    """limit(n): n bytes more than what torch holds now, and none of that free."""
    held = []

    def limit(more):
        set_limit = lambda n: torch.cuda.set_per_process_memory_fraction(n / torch.cuda.get_device_properties(0).total_memory)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        set_limit(torch.cuda.memory_reserved())
        for size in (16 << 20, 2 << 20):
            try:
                while True:
                    held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                pass
        set_limit(torch.cuda.memory_reserved() + more)
        time.sleep(1.1)  # the binding remembers for a second that there was no room
    yield limit
    held.clear()
    torch.cuda.set_per_process_memory_fraction(1.0)


def _problem(skew):
    M, Kd, Nd = 180_000, 150_000, 50  # a copy of B is 31 MB, more than what torch keeps free behind smaller tensors
    lens = np.random.default_rng(3).integers(20, 29, M)
    if skew:
        lens[7] = 30_000
    p = G.random_csr(M, Kd, Nd, 0.0, seed=3, lengths=lens)
    t = [torch.from_numpy(x).cuda() for x in (p.row_ptr, p.col_idx, p.values, p.B)]
    f64, mag = oracle.spmm_f64(p.row_ptr, p.col_idx, p.values, p.B, threads=4)
    longest = 0 if skew else int(lens.max())
    assert ops.plan_info(M, Kd, Nd, p.nnz, max_row_nnz=longest)["padded_copy"]
    return p, t, longest, lambda C: bool((np.abs(C.cpu().numpy() - f64) <= 1e-5 * mag + 1e-6).all())


@pytest.mark.parametrize("skew", [False, True])
@pytest.mark.parametrize("given", [0, 256, 8 << 20])
def test_prepared_call(limit_memory, skew, given):
    p, t, longest, right = _problem(skew)
    out = torch.empty((p.M, p.Nd), device="cuda")
    workspace = torch.empty(given, dtype=torch.uint8, device="cuda") if given else None
    limit_memory(6 << 20)
    call = ops.SpmmCall(*t, out, max_row_nnz=longest, workspace=workspace)
    want = ops.plan_info(p.M, p.Kd, p.Nd, p.nnz, max_row_nnz=longest, workspace=False)
    assert (call.kernel, call.launches) == (want["kernel"], want["launches"]) and want["kernel"] == ("merge" if skew else "row")
    assert right(call())


def _retries():
    return torch.cuda.memory_stats()["num_alloc_retries"]


@pytest.mark.parametrize("skew", [False, True])
@pytest.mark.parametrize("given", [0, 8 << 20])
def test_product_without_room(limit_memory, skew, given):
    """... and does not make torch give its free blocks back to find that out, call after call."""
    p, t, longest, right = _problem(skew)
    out = torch.empty((p.M, p.Nd), device="cuda")
    workspace = torch.empty(given, dtype=torch.uint8, device="cuda") if given else None
    limit_memory(6 << 20)
    before = _retries()
    for _ in range(5):
        out.zero_()
        ops.spmm(*t, out, max_row_nnz=longest, workspace=workspace)
        assert right(out)
    assert _retries() == before


def test_product_with_just_enough_room(limit_memory):
    p, t, longest, right = _problem(False)
    out = torch.empty((p.M, p.Nd), device="cuda")
    limit_memory(64 << 20)
    torch.cuda.reset_peak_memory_stats()
    held = torch.cuda.memory_allocated()
    ops.spmm(*t, out, max_row_nnz=longest)
    assert right(out) and torch.cuda.max_memory_allocated() >= held + p.Kd * 208  # the copy was made


@pytest.mark.parametrize("more,copied", [(256 << 20, True), (48 << 20, False)])
def test_captured_product(limit_memory, more, copied):
    """Into a graph whose pool has nothing yet: with room for the copy of B, and with room for C alone."""
    p, t, longest, right = _problem(False)
    ops.spmm(*t, max_row_nnz=longest)  # settings that a capture may not make
    limit_memory(more)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        out = ops.spmm(*t, max_row_nnz=longest)
    count = ctypes.c_size_t(0)  # every node of the captured call is a kernel
    assert ctypes.CDLL("libcudart.so.12").cudaGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), None, ctypes.byref(count)) == 0
    assert count.value == ops.plan_info(p.M, p.Kd, p.Nd, p.nnz, max_row_nnz=longest, workspace=copied)["launches"] == 1 + copied
    out.zero_()
    graph.replay()
    assert right(out)


def test_conversion_without_room(limit_memory):
    dense = torch.zeros((4096, 24_576), device="cuda")  # its bits: 12.6 MB
    dense.view(-1)[::1009] = 1.5
    want = ops.dense2csr(dense)
    limit_memory(6 << 20)
    before = _retries()
    for _ in range(3):
        got = ops.dense2csr(dense)
    assert _retries() == before and got[3] == want[3] and all(torch.equal(a, b) for a, b in zip(got[:3], want[:3]))
