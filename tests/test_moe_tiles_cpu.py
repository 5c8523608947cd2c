"""Rows per expert tile where a rank holds some of the experts, and of FP8 experts."""
import pytest

from uniserve_v1_b200.ops import functional as F


@pytest.mark.parametrize("T,E_local,E_total,top,fp8,rows", [
    (256, 16, 128, 8, False, 32),             # 16 routes to an expert, not 128
    (1536, 16, 128, 8, False, 256), (1535, 16, 128, 8, False, 32), (32, 8, 128, 8, False, 16),
    (160, 128, 128, 8, True, 16), (161, 128, 128, 8, True, 32), (320, 64, 64, 4, True, 16), (321, 64, 64, 4, True, 32),
    (1280, 16, 128, 8, True, 16), (8192, 128, 128, 8, True, 32)])
def test_rows_per_tile_of_a_share(T, E_local, E_total, top, fp8, rows):
    """A rank's share of the experts sees its share of the routes."""
    ws = F.MoeWorkspace.create(T, top, E_local, 64, 64, "cpu", E_total=E_total, fp8=fp8)
    assert ws.block_n == rows and ws.max_tiles >= E_local + T * top // rows
