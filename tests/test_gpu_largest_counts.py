"""2^31 - 1 entries, 2^31 - 1 columns: positions a chunk beyond the last one do not fit an int.  The row and resident
kernels end 64 entries earlier; above, whole rows run on the panel kernel."""
import pytest
import torch

from csrspmm_b200 import ops

pytestmark = pytest.mark.gpu
LARGEST = (1 << 31) - 1
ROWS = 1 << 20


@pytest.fixture(scope="module")
def entries():
    ci = torch.zeros(LARGEST, dtype=torch.int32, device="cuda")
    packed = torch.full((1 << 30,), 0x22, dtype=torch.uint8, device="cuda")  # every value is 1.0 * scale
    yield ci, packed
    del ci, packed
    torch.cuda.empty_cache()


@pytest.mark.parametrize("nnz", [LARGEST - 64, LARGEST])
@pytest.mark.parametrize("kernel,Nd,longest", [("row", 32, 0), ("row", 30, 0), ("row", 128, 0), ("row", 128, 2048), ("merge", 32, 0), ("tiled", 32, 0)])
def test_entries(cuda_lib, entries, kernel, Nd, longest, nnz):
    rp = (torch.arange(ROWS + 1, device="cuda") * 2048).clamp_(max=nnz).to(torch.int32)  # the last row is a shorter one
    ci, packed = entries
    Kd = 300
    B = (torch.arange(Kd * Nd, device="cuda") % 7).float().view(Kd, Nd)
    if kernel == "tiled":
        got = ops.spmm_tiled(rp, ci[:nnz], packed, B, panel_rows=100, e2m1_scale=0.5, nnz=nnz)
    else:
        resident = ops.plan_info(ROWS, Kd, Nd, nnz, kernel=kernel, max_row_nnz=longest)["resident_lanes"]
        assert resident == (32 if longest and nnz < LARGEST else 0)
        got = ops.spmm(rp, ci[:nnz], packed, B, kernel=kernel, max_row_nnz=longest, e2m1_scale=0.5, sync=True)
    lens = (rp[1:] - rp[:-1]).float()
    assert torch.equal(got, 0.5 * lens[:, None] * B[0])  # exact: small whole numbers, halved


@pytest.mark.parametrize("pad", [1, 0])  # rows on 16 bytes and not
def test_columns(cuda_lib, pad):
    wide = torch.zeros(2, LARGEST + pad, device="cuda")
    dense = wide[:, :LARGEST]
    at = torch.tensor([0, 511, LARGEST - 4097, LARGEST - 2], device="cuda")
    dense[0, at], dense[1, LARGEST - 1] = torch.arange(1.0, 5.0, device="cuda"), 9.0
    rp, ci, va, longest = ops.dense2csr(dense)
    assert rp.tolist() == [0, 4, 5] and longest == 4 and va.tolist() == [1, 2, 3, 4, 9]
    assert torch.equal(ci[:4].long(), at) and int(ci[4]) == LARGEST - 1
    del wide, dense
    torch.cuda.empty_cache()
