"""Merge-path tiles cut at row starts (longest row known) against the ordinary ones: tile edges, empty rows, a longest
row that was given too small, packed values and every width class."""
import numpy as np
import pytest
import torch

import oracle
from csrspmm_b200 import generators as G, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nd", [1, 3, 4, 8, 16, 30, 32, 64, 100, 128, 256, 512, 600])
@pytest.mark.parametrize("hint", ["right", "too small"])
def test_row_aligned_tiles(cuda_lib, Nd, hint):
    rng = np.random.default_rng(Nd)
    lens = rng.integers(0, 12, 9000)
    lens[:700] = 0
    lens[4000:4300] = 0
    lens[-1] = 0
    lens[5000] = 900 if hint == "right" else 7000  # the second does not fit a tile
    p = G.random_csr(len(lens), 8000, Nd, 0.0, seed=9, lengths=lens)
    t = [torch.from_numpy(x).cuda() for x in (p.row_ptr, p.col_idx, p.values, p.B)]
    C0 = rng.standard_normal((p.M, Nd), dtype=np.float32)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = ops.spmm(*t, torch.from_numpy(C0).cuda(), 1.5, -0.5, kernel="merge", max_row_nnz=900 if hint == "right" else 11,
                   status_word=status, sync=True).cpu().numpy()
    f64, mag = oracle.spmm_f64(p.row_ptr, p.col_idx, p.values, p.B, C0, 1.5, -0.5, threads=4)
    assert int(status) == 0 and (np.abs(got - f64) <= 1e-5 * mag + 1e-6).all()


# long grids of the largest tiles, whose lane groups find their shares by votes: one entry more or less than whole tiles of 3072 (and
# 1536) items, runs of empty rows longer than a tile, a row of several tiles; whole widths, guarded ones and padded copies
@pytest.mark.parametrize("Nd", [2, 8, 20, 32, 36, 57, 64, 128, 256])
@pytest.mark.parametrize("over", [-1, 0, 1])
def test_long_grids_of_tiles(cuda_lib, Nd, over):
    rng = np.random.default_rng(Nd)
    M, tiles = 60_000, 700
    lens = rng.integers(0, 60, M)
    lens[1000:8000] = 0
    lens[20_000] = 9000
    lens[-1] = 0
    short = 3072 * tiles + over - M - int(lens.sum())
    lens[30_000:50_000] += short // 20_000
    lens[30_000] += short - short // 20_000 * 20_000
    assert M + int(lens.sum()) == 3072 * tiles + over and lens.min() >= 0
    p = G.random_csr(M, 70_000, Nd, 0.0, seed=3, lengths=lens)
    t = [torch.from_numpy(x).cuda() for x in (p.row_ptr, p.col_idx, p.values, p.B)]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = ops.spmm(*t, None, 1.0, 0.0, kernel="merge", status_word=status, sync=True).cpu().numpy()
    f64, mag = oracle.spmm_f64(p.row_ptr, p.col_idx, p.values, p.B, np.zeros((M, Nd), np.float32), 1.0, 0.0, threads=4)
    # rows of several tiles are sums of partial sums in fp32: the bound of the tests above, a rounding per term of its magnitude
    assert int(status) == 0 and (np.abs(got - f64) <= 1e-5 * mag + 1e-6).all()
