"""Dense -> CSR and quantisation at the sizes where the work is cut: warps per row, chunks, scan tiles, odd strides."""
import numpy as np
import pytest
import torch

from csrspmm_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,pad", [(1, 1, 0), (3, 511, 1), (9, 512, 0), (5, 513, 3), (7, 1024, 0), (2, 1025, 0), (3, 2047, 1), (3, 2049, 0),
                                     (2, 4097, 3), (2, 9001, 0), (8193, 7, 0), (20000, 3, 1)])
@pytest.mark.parametrize("tol", [0.0, 0.6])
def test_dense2csr(cuda_lib, H, W, pad, tol):
    rng = np.random.default_rng(H * 10007 + W)
    dense = (rng.standard_normal((H, W)) * (rng.random((H, W)) < 0.3)).astype(np.float32)
    wide = torch.zeros((H, W + pad), device="cuda")
    wide[:, :W] = torch.from_numpy(dense).cuda()
    rp, ci, va, longest = ops.dense2csr(wide[:, :W], tol)
    keep = np.abs(dense) > tol
    assert np.array_equal(rp.cpu().numpy(), np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32))
    assert np.array_equal(ci.cpu().numpy(), np.nonzero(keep)[1].astype(np.int32))
    assert np.array_equal(va.cpu().numpy(), dense[keep]) and longest == int(keep.sum(1).max())


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 4095, 4097, 148 * 4 * 4096 + 5])
@pytest.mark.parametrize("offset", [0, 1])
def test_quantize_equals_the_host_codec(cuda_lib, n, offset):
    v = np.random.default_rng(n).standard_normal(n + offset, dtype=np.float32)
    packed, scale = ops.e2m1_quantize(torch.from_numpy(v).cuda()[offset:])
    want, want_scale = ops.e2m1_quantize(torch.from_numpy(v[offset:].copy()))
    assert scale == want_scale and torch.equal(packed.cpu(), want)


def test_kept_memory_is_given_back(cuda_lib):
    dense = torch.ones(3_000_000, 2, device="cuda")  # its row counts: some 12 MB of scratch
    ops.dense2csr(dense)
    torch.cuda.synchronize()
    assert ops.release_memory() >= 12_000_000
    assert ops.release_memory() == 0
    rp, _, _, longest = ops.dense2csr(dense)  # and calls go on
    assert int(rp[-1]) == 6_000_000 and longest == 2
