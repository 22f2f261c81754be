"""The device transposition against the host one: tile edges, one to three digit passes, repeats, hub columns."""
import numpy as np
import pytest
import torch

from csrspmm_b200 import _lib, torch_library as TL

pytestmark = pytest.mark.gpu


SIZES = [(1, 1, 1, False), (5, 1, 1023, False), (300, 2, 1024, False), (300, 1024, 1025, False), (70, 1025, 5000, True), (4000, 70001, 30000, False),
         (900, 3000, 131072, False), (900, 3000, 131073, True), (17, (1 << 20) + 1, 2000, False), (50000, 2048, 1300000, True),
         (60000, (1 << 22) + 3, 1250000, False)]


@pytest.mark.parametrize("M,Kd,nnz,hub", SIZES)
def test_transpose(cuda_lib, M, Kd, nnz, hub):
    rng = np.random.default_rng(nnz)
    rows = np.sort(rng.integers(0, M, nnz))  # many rows stay empty
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=M))]).astype(np.int32)
    ci = rng.integers(0, Kd, nnz).astype(np.int32)  # unsorted, with repeats
    if hub:
        ci[rng.random(nnz) < 0.4] = Kd - 1
    t = [torch.from_numpy(x) for x in (rp, ci, rng.standard_normal(nnz, dtype=np.float32))]
    want = TL.transpose_csr(*t, Kd)
    got = TL.transpose_csr(*(x.cuda() for x in t), Kd)
    assert all(torch.equal(g.cpu(), w) for g, w in zip(got, want))


# one tile and two, tiles of one and two entries per thread, one wave and two; columns per bucket 1 to 512 and the first width
# beyond; buckets of one chunk and of many, all entries in one column, chunks of 8192
BUCKETS = [(300, 512, 8192, 0.0), (300, 513, 8193, 0.4), (7, 3, 4097, 1.0), (2, 1, 4096, 1.0), (400, 64, 100000, 0.0), (5000, 1 << 19, 151552, 0.3),
           (5000, (1 << 19) + 1, 151553, 0.3), (3000, 40000, 151553, 0.9), (20000, 65536, 1212416, 1.0), (20000, 65535, 1212417, 0.05),
           (60000, 1 << 18, 2200000, 0.2)]
# what buckets have no room for, by digits: one pass (few columns) whose CTAs add the counts up themselves, with the scan, and with
# sixteen entries per thread; two passes of five and of eight bits; three at the last size of eight entries per thread and the
# first of sixteen; four, with fewer entries than columns and with the scan
DIGITS = [(9, 2, 9000, 0.4), (400, 64, 1000000, 0.0), (4000, 256, 1900000, 0.3), (5000, 512, 2200000, 0.1), (70000, 65536, 4900000, 0.05),
          (50000, (1 << 19) + 1, 1818623, 0.2), (50000, (1 << 19) + 1, 1818624, 0.2), (3000, (1 << 24) + 1, 3000, 0.1),
          (3000, (1 << 24) + 1, 200000, 0.3)]


def _check(M, Kd, nnz, share):
    rng = np.random.default_rng(Kd)
    rp = np.concatenate([[0], np.sort(rng.integers(0, nnz + 1, M - 1)), [nnz]]).astype(np.int32)
    ci = rng.integers(0, Kd, nnz).astype(np.int32)
    ci[rng.random(nnz) < share] = Kd // 3
    t = [torch.from_numpy(x) for x in (rp, ci, rng.standard_normal(nnz, dtype=np.float32))]
    want = TL.transpose_csr(*t, Kd)
    got = TL.transpose_csr(*(x.cuda() for x in t), Kd)
    assert all(torch.equal(g.cpu(), w) for g, w in zip(got, want))


@pytest.mark.parametrize("M,Kd,nnz,share", BUCKETS)
def test_transpose_through_buckets(cuda_lib, M, Kd, nnz, share):
    _check(M, Kd, nnz, share)


@pytest.mark.parametrize("M,Kd,nnz,share", DIGITS)
def test_transpose_by_digits(cuda_lib, M, Kd, nnz, share):
    _check(M, Kd, nnz, share)


def test_transpose_of_nothing(cuda_lib):
    rp, ci, va = torch.zeros(4, dtype=torch.int32).cuda(), torch.zeros(0, dtype=torch.int32).cuda(), torch.zeros(0).cuda()
    t_rp, t_ci, t_va = TL.transpose_csr(rp, ci, va, 9)
    assert t_rp.tolist() == [0] * 10 and t_ci.numel() == t_va.numel() == 0


@pytest.mark.parametrize("rp,ci", [([0, 2], [0, 9]), ([0, 2], [-1, 3]), ([0, 1], [0, 3])])
def test_a_matrix_that_is_none_is_refused(cuda_lib, rp, ci):
    t = torch.tensor(rp, dtype=torch.int32), torch.tensor(ci, dtype=torch.int32), torch.ones(2)
    for arrays in (t, [x.cuda() for x in t]):
        with pytest.raises((RuntimeError, IndexError)):
            TL.transpose_csr(*arrays, 9)


def test_operator_errors_keep_their_type(cuda_lib):
    rp, ci, va = torch.tensor([0, 1], dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32).cuda(), torch.ones(1).cuda()
    with pytest.raises(_lib.SpmmError):  # the bulk-copy kernel needs whole vectors
        torch.ops.csrspmm_b200.spmm(rp, ci, va, torch.ones(1, 3).cuda(), 1.0, "tma")
