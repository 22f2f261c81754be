"""The resident kernel (a panel of B in shared memory) at the edges of its range, bit for bit against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from csrspmm_b200 import generators as G, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,Kd,Nd,mean,lanes", [(3, 1, 128, 1, 0), (700, 64, 132, 6, 0), (150, 97, 1024, 33, 32), (1000, 400, 388, 40, 32), (900, 401, 200, 40, 16),
                                                (517, 800, 68, 90, 0), (200, 256, 4096, 64, 32), (40, 30, 2496, 29, 32), (700, 64, 132, 14, 32), (1700, 800, 68, 90, 16),
                                                (5000, 8, 132, 8, 32)])
@pytest.mark.parametrize("beta,packed", [(0.0, False), (0.5, False), (0.0, True)])
def test_resident_panels(cuda_lib, M, Kd, Nd, mean, lanes, beta, packed):
    rng = np.random.default_rng(M + Kd)
    lens = np.minimum(rng.poisson(mean, M), Kd)
    lens[:: max(M // 7, 1)] = 0  # empty rows among them, the first one too
    lens[M // 2] = min(Kd, 4 * mean)
    p = G.random_csr(M, Kd, Nd, 0.0, seed=5, lengths=lens)
    # `lanes` says which of the sizes reach it (0: too little re-use of B, the ordinary build sums whole rows)
    assert ops.plan_info(M, Kd, Nd, p.nnz, kernel="row", max_row_nnz=max(int(lens.max()), 1))["resident_lanes"] == lanes
    t = [torch.from_numpy(x).cuda() for x in (p.row_ptr, p.col_idx, p.values, p.B)]
    C0 = rng.standard_normal((M, Nd), dtype=np.float32)
    C = torch.from_numpy(C0).cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    kw = dict(max_row_nnz=max(int(lens.max()), 1), kernel="row", status_word=status, sync=True)
    values = p.values
    if packed:
        t[2], scale = ops.e2m1_quantize(t[2])
        values = oracle.e2m1_decode(t[2].cpu().numpy(), p.nnz, scale)
        kw.update(e2m1_scale=scale, nnz=p.nnz)
    got = ops.spmm(*t, C, 1.25, beta, **kw)
    assert np.array_equal(got.cpu().numpy(), oracle.spmm(p.row_ptr, p.col_idx, values, p.B, C0, 1.25, beta)) and int(status) == 0
