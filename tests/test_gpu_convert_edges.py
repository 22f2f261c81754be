"""Dense -> CSR and quantisation at the sizes where the work is cut: warps per row, chunks, scan tiles, odd strides."""
import numpy as np
import pytest
import torch

from csrspmm_b200 import _lib, ops

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


# the magnitudes between two codes and their neighbours, at scales over the whole range: limits per scale from 1.2e-38 to 4e37, a
# division per value beyond
@pytest.mark.parametrize("largest", [6.0, 1.0, 0.0471, 3.3e38, 2.5e38, 2.3e38, 7.1e-38, 7.0e-38, 1e-41, 123456.789])
def test_codes_at_their_limits(cuda_lib, largest):
    scale = np.float32(largest) / np.float32(6.0)
    v = [np.float32(largest), np.float32(0.0), np.float32(-0.0), np.float32("nan")]
    for middle in (0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 6.0):
        with np.errstate(over="ignore", invalid="ignore"):
            at = np.float32(middle) * scale
        if not np.isfinite(at):
            at = np.float32(3e38)
        around = (np.array(at).view(np.int32) + np.arange(-6, 7, dtype=np.int32)).clip(0, 0x7F7FFFFF).astype(np.int32).view(np.float32)
        around = around[around <= np.float32(largest)]
        v += [*around, *-around]
    v = torch.from_numpy(np.array(v, dtype=np.float32))
    packed, got = ops.e2m1_quantize(v.cuda())
    want, want_scale = ops.e2m1_quantize(v)
    assert got == want_scale and torch.equal(packed.cpu(), want)


# more columns than a warp's span and than all warps' spans, every density, through the bits and without them
@pytest.mark.parametrize("H,W,pad", [(3, 1023, 0), (5, 1024, 4), (2, 1025, 3), (3, 4100, 0), (2, 8192 + 33, 0)])
@pytest.mark.parametrize("share", [0.0, 0.002, 1.0])
def test_dense2csr_spans(cuda_lib, H, W, pad, share):
    rng = np.random.default_rng(W)
    dense = np.where(rng.random((H, W)) < share, rng.standard_normal((H, W)), 0.0).astype(np.float32)
    dense[0, -1] = np.nan  # never kept
    wide = torch.zeros((H, W + pad), device="cuda")
    wide[:, :W] = torch.from_numpy(dense).cuda()
    with np.errstate(invalid="ignore"):
        keep = np.abs(dense) > 0
    rp, ci, va, longest = ops.dense2csr(wide[:, :W])
    assert np.array_equal(rp.cpu().numpy(), np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32))
    assert np.array_equal(ci.cpu().numpy(), np.nonzero(keep)[1].astype(np.int32)) and np.array_equal(va.cpu().numpy(), dense[keep])
    L, n = _lib.lib(), int(rp[-1])
    ci2, va2 = torch.full_like(ci, -1), torch.full_like(va, 7.0)
    if n > 0:
        stream = torch.cuda.current_stream().cuda_stream
        assert L.csrspmm_b200_dense2csr_fill(H, W, wide.data_ptr(), W + pad, 0.0, rp.data_ptr(), ci2.data_ptr(), va2.data_ptr(), stream) == 0
    assert torch.equal(ci2, ci) and torch.equal(va2, va) and longest == int(keep.sum(1).max())


def test_kept_memory_is_given_back(cuda_lib):
    dense = torch.ones(3_000_000, 2, device="cuda")  # its row counts: some 12 MB of scratch
    ops.dense2csr(dense)
    torch.cuda.synchronize()
    assert ops.release_memory() >= 12_000_000
    assert ops.release_memory() == 0
    rp, _, _, longest = ops.dense2csr(dense)  # and calls go on
    assert int(rp[-1]) == 6_000_000 and longest == 2
