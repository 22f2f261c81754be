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


@pytest.mark.parametrize("sizes,longest,with_room,without", [
    ((5000, 5000, 57, 1_500_000), 350, dict(kernel="merge", launches=2, padded_copy=True, row_aligned=True), dict(kernel="row")),
    ((200_000, 200_000, 57, 1_600_000), 40, dict(kernel="row", launches=2, padded_copy=True), dict(kernel="row")),
    ((20_000, 20_000, 201, 480_000), 0, dict(kernel="merge", launches=3, padded_copy=True), dict(kernel="merge", launches=2)),
    ((16_384, 16_384, 64, 262_144), 40, dict(kernel="row"), dict(kernel="row")),
    ((8192, 256, 4096, 209_715), 60, dict(kernel="row", resident_lanes=32), dict(kernel="row", resident_lanes=32)),
    ((512, 4096, 64, 102_400), 300, dict(kernel="merge", row_aligned=True), dict(kernel="merge", row_aligned=True))])
def test_plan_info_says_what_runs(sizes, longest, with_room, without):
    for room, want in ((True, with_room), (False, without)):
        got = ops.plan_info(*sizes, max_row_nnz=longest, workspace=room)
        assert got == dict(dict(launches=1, padded_copy=False, resident_lanes=0, row_aligned=False), **want)
    assert ops.selected_kernel(*sizes, max_row_nnz=longest) == with_room["kernel"]
    assert ops.plan_info(0, 5, 64, 0)["launches"] == 0


# even widths: a padded copy of B only where it was measured to pay
@pytest.mark.parametrize("M,Kd,Nd,mean,want", [
    (80_910, 56_130, 30, 157, True), (308_165, 350_025, 30, 15, False), (100_000, 60_000, 26, 29, True), (100_000, 60_500, 26, 29, False),
    (18_944, 10_000, 22, 370, True), (18_945, 58_783, 22, 370, False), (28_416, 58_783, 22, 370, False), (28_417, 58_783, 22, 370, True),  # waves
    (60_000, 26_000, 22, 64, True), (150_000, 75_000, 50, 12, True), (253_847, 293_193, 54, 22, False),
    (489_723, 1_227_653, 50, 37, False), (200_000, 100_000, 66, 12, True), (200_000, 101_000, 66, 12, False), (60_773, 4886, 138, 15, True),
    (100_000, 100_000, 150, 12, True), (200_000, 200_000, 150, 10, False), (170_295, 18_568, 254, 20, True), (7911, 8319, 370, 130, True),
    (100_000, 40_000, 62, 100, False), (100_000, 40_000, 118, 20, False)])
def test_copies_of_even_widths(M, Kd, Nd, mean, want):
    assert ops.plan_info(M, Kd, Nd, M * mean, max_row_nnz=0)["padded_copy"] == want


@pytest.mark.parametrize("Nd,mean,longest,want", [(50, 10, 60, True), (50, 10, 0, False), (50, 10, 65, False), (34, 10, 60, True), (50, 7, 60, False),
                                                  (54, 15, 64, True), (58, 15, 64, False), (66, 15, 64, False)])
def test_copies_for_even_rows(Nd, mean, longest, want):
    assert ops.plan_info(300_000, 200_000, Nd, 300_000 * mean, max_row_nnz=longest)["padded_copy"] == want
