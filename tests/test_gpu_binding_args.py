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
