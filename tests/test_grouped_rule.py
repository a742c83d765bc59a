"""Rows per tile of the grouped products (``ops.grouped_tile_rows``): a decision of the host alone."""
import pytest


@pytest.mark.parametrize("experts,inner,hidden,rows,want", [
    (32, 1024, 2048, 1, 64), (32, 1024, 2048, 2, 64), (32, 1024, 2048, 4, 128), (32, 1024, 2048, 256, 128),
    (32, 1024, 1536, 8, 64), (32, 1024, 1536, 16, 128), (16, 1024, 2048, 32, 64), (16, 1024, 2048, 64, 128),
    (8, 768, 1536, 2, 64), (8, 768, 1536, 96, 64), (8, 768, 1536, 256, 128), (8, 512, 1024, 64, 64), (8, 512, 1024, 1024, 128)])
def test_lines(experts, inner, hidden, rows, want):
    """Small experts stay on tiles of 64 rows: the other kernel takes as long for a few rows as for many."""
    from llm_rs_b200 import ops
    assert ops.grouped_tile_rows(rows * experts, experts, experts * inner * hidden) == want
