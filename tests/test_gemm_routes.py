"""Routing rules of the native GEMM kernels (host code, no GPU)."""
from __future__ import annotations

import pytest

from gemm_routes import CLUSTER_64, TMA_128, WS_64, dgemm_route

MAX_GRID_Y = 65535
TILE_COLS = {TMA_128: 128, WS_64: 64, CLUSTER_64: 64}


@pytest.mark.parametrize("m", [33, 64, 192, 320, 640, 704, 1000])
@pytest.mark.parametrize("k", [256, 512, 4096])
@pytest.mark.parametrize("n", [64 * MAX_GRID_Y, 64 * MAX_GRID_Y + 1, 4_300_000, 5_000_000, 128 * MAX_GRID_Y])
def test_column_tiles_fit_the_grid(m, n, k):
    """Every n the 128 x 128 tiles can launch stays on a kernel that can launch it."""
    r = dgemm_route(m, n, k)
    assert (n + TILE_COLS[r.kernel] - 1) // TILE_COLS[r.kernel] <= MAX_GRID_Y


def test_last_column_count_of_the_64_wide_tiles():
    assert dgemm_route(64, 64 * MAX_GRID_Y, 256).kernel == WS_64
    assert dgemm_route(64, 64 * MAX_GRID_Y + 1, 256).kernel == TMA_128
