"""The lines of the kernel choice for even rows (host logic)."""
import pytest

from csrspmm_b200 import ops


@pytest.mark.parametrize("M,Kd,Nd,mean,want", [
    (12000, 12000, 32, 64, "merge"), (12001, 12001, 32, 64, "row"), (512, 4096, 32, 63, "row"),     # few long rows, eight lanes each
    (12000, 12000, 64, 150, "merge"), (512, 4096, 64, 149, "row"),                                  # sixteen
    (591, 4096, 512, 200, "merge"), (592, 4096, 512, 200, "row"), (591, 4096, 512, 199, "row"),     # a warp
    (2400, 4096, 30, 80, "merge"), (2401, 4096, 30, 80, "row"), (591, 4096, 50, 80, "merge"), (592, 4096, 50, 80, "row"),
    (1 << 20, 1 << 20, 64, 16, "merge"), (1 << 20, 1 << 20, 64, 65, "row"), (180000, 180000, 64, 16, "row")])  # B beyond 48 MB
def test_even_rows(M, Kd, Nd, mean, want):
    assert ops.selected_kernel(M, Kd, Nd, M * mean, max_row_nnz=max(60, mean + mean // 2)) == want
