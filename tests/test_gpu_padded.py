"""Products on a padded copy of B (widths that are no multiple of four), and the same without room for the copy."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from csrspmm_b200 import generators as G, ops

pytestmark = pytest.mark.gpu  # the test of the scratch size needs no GPU, but the library


@pytest.mark.parametrize("Nd", [19, 33, 57, 99, 130, 201, 255, 257, 510])
@pytest.mark.parametrize("kernel,skew,beta", [("row", False, 0.0), ("merge", False, 0.5), ("merge", True, -0.5)])
def test_padded_copy(cuda_lib, Nd, kernel, skew, beta):
    rng = np.random.default_rng(Nd)
    M, Kd = 9001, 2500
    lens = rng.integers(0, 2 * max(20, 9_000_000 // Nd // (M // 8)), M) % 1200
    if Nd % 2 == 0:
        lens = rng.integers(20, 120, M)
    if skew:
        lens[77] = Kd
    p = G.random_csr(M, Kd, Nd, 0.0, seed=3, lengths=lens)
    t = [torch.from_numpy(x).cuda() for x in (p.row_ptr, p.col_idx, p.values)]
    wide = torch.randn((Kd, Nd + 2), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    B = wide[:, 1:1 + Nd]  # rows that start anywhere, and do not follow each other
    C0 = rng.standard_normal((M, Nd), dtype=np.float32)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = ops.spmm(*t, B, torch.from_numpy(C0).cuda(), 1.5, beta, kernel=kernel, max_row_nnz=0 if skew else int(lens.max()),
                   status_word=status, sync=True).cpu().numpy()
    f64, mag = oracle.spmm_f64(p.row_ptr, p.col_idx, p.values, np.ascontiguousarray(B.cpu().numpy()), C0, 1.5, beta, threads=4)
    assert int(status) == 0 and (np.abs(got - f64) <= 1e-5 * mag + 1e-6).all()


# even widths: C in pairs, or (an odd leading dimension, a start off 8 bytes) float by float
@pytest.mark.parametrize("Nd", [18, 22, 30, 32 + 2, 66, 98, 130, 254])
@pytest.mark.parametrize("kernel,beta", [("row", 0.5), ("merge", 0.0)])
@pytest.mark.parametrize("ldc,start", [(0, 0), (2, 0), (1, 0), (0, 1)])
def test_padded_copy_of_even_widths(cuda_lib, Nd, kernel, beta, ldc, start):
    rng = np.random.default_rng(Nd)
    M, Kd = 6001, 2500
    mean = int(255e6 / 4 / Nd / M) + 2
    lens = rng.integers(mean - mean // 8, mean + mean // 4, M)
    lens[5] = 0
    p = G.random_csr(M, Kd, Nd, 0.0, seed=3, lengths=np.minimum(lens, Kd))
    # (254: 127 of 128 pairs at work, from 64 uses on)
    assert ops.plan_info(M, Kd, Nd, p.nnz, kernel=kernel, max_row_nnz=int(lens.max()), workspace=True)["padded_copy"]
    t = [torch.from_numpy(x).cuda() for x in (p.row_ptr, p.col_idx, p.values, p.B)]
    C0 = rng.standard_normal((M, Nd + ldc), dtype=np.float32)
    C = torch.full((M * (Nd + ldc) + start,), 7.0, device="cuda")[start:].view(M, Nd + ldc)
    C.copy_(torch.from_numpy(C0))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.spmm(*t, C[:, :Nd], 1.5, beta, kernel=kernel, max_row_nnz=int(lens.max()), status_word=status, sync=True)
    got = C.cpu().numpy()
    f64, mag = oracle.spmm_f64(p.row_ptr, p.col_idx, p.values, p.B, C0[:, :Nd], 1.5, beta, threads=4)
    assert int(status) == 0 and (np.abs(got[:, :Nd] - f64) <= 1e-5 * mag + 1e-6).all()
    assert np.array_equal(got[:, Nd:], C0[:, Nd:])  # nothing beyond the rows


def test_the_copy_is_counted_as_scratch():
    assert ops.workspace_bytes(200000, 200000, 57, 1_600_000) >= ops.workspace_bytes(200000, 200000, 60, 1_600_000) + 200000 * 240 - 256


@pytest.mark.parametrize("M,Kd,Nd,mean,longest", [(5000, 5000, 57, 300, 350), (60_000, 20_000, 57, 16, 40), (20_000, 20_000, 201, 24, 0), (9000, 9000, 64, 8, 20),
                                                  (9000, 256, 2048, 25, 60)])
def test_call_says_what_it_launches(cuda_lib, M, Kd, Nd, mean, longest):
    lens = np.random.default_rng(M).integers(mean - mean // 8, mean + mean // 8 + 1, M)
    p = G.random_csr(M, Kd, Nd, 0.0, seed=3, lengths=lens)
    t = [torch.from_numpy(x).cuda() for x in (p.row_ptr, p.col_idx, p.values, p.B)]
    call = ops.SpmmCall(*t, torch.empty((M, Nd), device="cuda"), max_row_nnz=longest)
    assert call.kernel == ops.selected_kernel(M, Kd, Nd, p.nnz, max_row_nnz=longest)
    call()  # the first call makes the settings that a capture may not
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        call()
    count = ctypes.c_size_t(0)  # every node of the captured call is a kernel
    assert ctypes.CDLL("libcudart.so.12").cudaGraphGetNodes(ctypes.c_void_p(g.raw_cuda_graph()), None, ctypes.byref(count)) == 0
    assert count.value == call.launches
