"""What the CPython binding takes and refuses."""
import pytest
import torch

from csrspmm_b200 import ops

pytestmark = pytest.mark.gpu


def _matrix():
    rp, ci = torch.tensor([0, 2, 3, 5], dtype=torch.int32), torch.tensor([0, 3, 1, 2, 4], dtype=torch.int32)
    return rp.cuda(), ci.cuda(), torch.tensor([1.0, 2, 3, 4, 5]).cuda(), torch.arange(20.0).reshape(5, 4).cuda()


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("nnz", [-1, -5])
def test_a_negative_number_of_entries_is_refused(cuda_lib, packed, nnz):
    rp, ci, va, B = _matrix()
    kw = {}
    if packed:
        va, kw["e2m1_scale"] = ops.e2m1_quantize(va)
    with pytest.raises(RuntimeError, match="differ in length|nnz=-"):
        ops.spmm(rp, ci, va, B, nnz=nnz, **kw)


def test_whole_numbers_of_any_type_are_taken(cuda_lib):
    rp, ci, va, B = _matrix()
    want = ops.spmm(rp, ci, va, B)
    assert torch.equal(ops.spmm(rp, ci, va, B, nnz=5.0, max_row_nnz=2.0), want)
    assert torch.equal(ops.spmm(rp, ci, va, B, nnz=torch.tensor(5), max_row_nnz=torch.tensor(2)), want)


def _products(rp, ci, va, B, C=None, **kw):
    """The three ways to a product that take strided operands."""
    yield lambda: ops.spmm(rp, ci, va, B, C, **kw)
    yield lambda: ops.SpmmCall(rp, ci, va, B, torch.empty(3, B.size(1), device="cuda") if C is None else C, **kw)
    yield lambda: ops.spmm_tiled(rp, ci, va, B, C, **kw)


def test_operands_that_end_before_their_last_row_are_refused(cuda_lib):
    rp, ci, va, B = _matrix()
    for run in _products(rp, ci, va, B[:1].expand(5, 4)):
        with pytest.raises(RuntimeError, match="overlap"):
            run()
    for C in (torch.zeros(1, 4, device="cuda").expand(3, 4), torch.zeros(4, 3, device="cuda").t()):
        for run in _products(rp, ci, va, B, C):
            with pytest.raises(RuntimeError, match="C_out must be row-major"):
                run()
    for run in _products(rp, ci[:4], va, B, nnz=5):
        with pytest.raises(RuntimeError, match="col_idx too short"):
            run()
    with pytest.raises(RuntimeError, match="row-major"):
        ops.dense2csr(B[:1].expand(5, 4))
    packed, scale = ops.e2m1_quantize(va)
    for p in (packed, packed.cpu()):
        with pytest.raises(RuntimeError, match="too short"):
            ops.e2m1_dequantize(p, 7, scale)
    narrow = torch.ones(5, 3, device="cuda")[:, :1]  # one column of a wider matrix, and one row with any stride, are fine
    assert torch.equal(ops.spmm(rp, ci, va, torch.ones(5, 1, device="cuda")), ops.spmm(rp, ci, va, narrow))
    assert ops.dense2csr(torch.ones(4, device="cuda").as_strided((1, 4), (0, 1)))[3] == 4
