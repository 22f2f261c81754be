"""The row kernel's builds for grids of a wave or two, at the grid sizes where the choice changes, bit for bit against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from csrspmm_b200 import generators as G, ops

pytestmark = pytest.mark.gpu

EDGES = [4, 6, 7, 8, 9, 10, 12]  # CTAs per SM


@pytest.mark.parametrize("Nd,rows_per_cta", [(32, 16), (20, 16), (64, 8), (128, 4), (100, 4), (256, 4), (200, 4), (512, 4), (520, 4)])
@pytest.mark.parametrize("waves", EDGES)
@pytest.mark.parametrize("packed", [False, True])
def test_grids_at_the_edges(cuda_lib, Nd, rows_per_cta, waves, packed):
    for over in (0, 1):
        M, Kd = 148 * waves * rows_per_cta + over, 300
        rng = np.random.default_rng(M)
        lens = np.minimum(rng.poisson(70, M), 110)
        lens[::97] = 0
        p = G.random_csr(M, Kd, Nd, 0.0, seed=2, lengths=lens)
        t = [torch.from_numpy(x).cuda() for x in (p.row_ptr, p.col_idx, p.values, p.B)]
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        kw = dict(max_row_nnz=0, kernel="row", status_word=status, sync=True)  # (0: no resident kernel)
        values = p.values
        if packed:
            t[2], scale = ops.e2m1_quantize(t[2])
            values = oracle.e2m1_decode(t[2].cpu().numpy(), p.nnz, scale)
            kw.update(e2m1_scale=scale, nnz=p.nnz)
        got = ops.spmm(*t, None, 1.0, 0.0, **kw).cpu().numpy()
        assert int(status) == 0
        assert np.array_equal(got, oracle.spmm(p.row_ptr, p.col_idx, values, p.B, np.zeros((M, Nd), np.float32), 1.0, 0.0))
