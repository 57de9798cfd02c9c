"""Routing rules of the native GEMM kernels (host code, no GPU)."""
from __future__ import annotations

import itertools

import pytest

from gemm_routes import CLUSTER_64, TILES, TMA_128, WS_64, dgemm_route, sgemm_route

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


@pytest.mark.parametrize("tma", [True, False])
@pytest.mark.parametrize("tri", [0, 1])
def test_clusters_keep_the_planned_k_ranges(tma, tri):
    """A cluster adds up K ranges no longer than those the plan would sum through the
    workspace: longer ones round worse, and leave SMs idle (576 x 576 x 1024)."""
    sizes = [17, 64, 65, 128, 250, 320, 384, 512, 576, 640, 704, 770, 1000, 1024]
    for m, n, k in itertools.product(sizes, sizes, [64, 128, 200, 256, 300, 512, 777, 1024, 1025, 2000, 4096]):
        if tri and m != n:
            continue
        r, planned = dgemm_route(m, n, k, tri, tma), dgemm_route(m, n, k, tri, tma, automatic=False)
        chunk = r.k_chunk
        if r.kernel in (WS_64, CLUSTER_64):
            chunk = ((k + r.cluster - 1) // r.cluster + 15) // 16 * 16
        assert min(k, chunk) <= min(k, planned.k_chunk), (m, n, k, r, planned)


def test_cluster_of_two_range():
    assert dgemm_route(576, 576, 1024).kernel == TILES  # 81 tiles, three ranges
    assert dgemm_route(576, 704, 1024)[2:4] == (WS_64, 2)  # 99 tiles, two ranges
    assert dgemm_route(1024, 512, 512)[2:4] == (WS_64, 2)
    assert dgemm_route(768, 768, 512)[2:4] == (WS_64, 2)  # 144 tiles


def test_sgemm_clusters_keep_the_planned_k_ranges():
    """As above for FP32: 128 x 64 cluster tiles (16-deep slices) against the plan's 128 x 128
    tiles, whose ranges are multiples of 32."""
    up = lambda x, q: (x + q - 1) // q * q  # noqa: E731
    sizes = [17, 64, 128, 129, 256, 300, 384, 512, 600, 640, 900, 1024, 2000, 4096]
    clusters = set()
    for m, n, k in itertools.product(sizes, sizes, [16, 100, 256, 511, 512, 801, 1000, 1300, 2048, 2310, 2560, 4000]):
        r = sgemm_route(m, n, k)
        if not r.cluster:
            continue
        chunk = up(up(k, r.cluster) // r.cluster, 16)
        if r.halves:
            chunk = (chunk // 16 + 1) // 2 * 16
        assert min(k, chunk) <= min(k, up(up(k, r.splits) // r.splits, 32)), (m, n, k, r)
        clusters.add(r[1:])
    assert clusters == {(8, 0), (4, 0), (2, 0), (1, 0), (8, 1), (4, 1), (2, 1)}


def test_cluster_routes_need_no_workspace():
    for shape, route in (((256, 256, 256), (CLUSTER_64, 4)), ((1024, 512, 512), (WS_64, 2)),
                         ((2048, 2048, 2048), (WS_64, 1)), ((2048, 512, 2048), (TMA_128, 2))):
        r = dgemm_route(*shape)
        assert r[2:4] == route and r.ranges == 1, (shape, r)
    assert dgemm_route(256, 256, 4096).ranges == dgemm_route(256, 256, 4096, tma=False).ranges == 16
    # a split count that the caller asked for keeps the workspace
    assert dgemm_route(2048, 512, 2048, automatic=False).ranges == 2


def test_rules_follow_the_sm_count():
    """The routing rules use the SM count that the plan was made for (a partitioned GPU has fewer)."""
    # up to two CTAs per SM: 56 tiles in clusters of four are 224 CTAs
    assert dgemm_route(448, 512, 200, sms=148).kernel == CLUSTER_64
    assert dgemm_route(448, 512, 200, sms=74).kernel == TILES
    # rounds of tiles: 121 tiles of 128 x 128 are one round on 148 SMs, two on 74 (484 of 64 x 64: seven)
    assert dgemm_route(1400, 1400, 512, sms=148).kernel == TMA_128
    assert dgemm_route(1400, 1400, 512, sms=74).kernel == WS_64
    # one CTA per SM: 24 tiles of 128 x 64
    assert sgemm_route(300, 500, 300, sms=148).cluster == 4
    assert sgemm_route(300, 500, 300, sms=74).cluster == 2


@pytest.mark.parametrize("m,n,k,kernel", [
    (256, 256, 256, CLUSTER_64), (128, 1024, 300, CLUSTER_64),       # up to 33 tiles: an SM for each CTA
    (384, 384, 160, CLUSTER_64), (384, 384, 256, TILES),             # 36 tiles: 144 CTAs of the plan fit, clusters do not
    (448, 448, 192, TILES), (448, 448, 256, CLUSTER_64), (448, 448, 300, TILES),  # 49 tiles, three and four ranges
    (512, 512, 512, CLUSTER_64), (512, 512, 768, CLUSTER_64), (512, 512, 1024, TILES),
    (448, 640, 512, CLUSTER_64), (520, 500, 512, TILES), (520, 500, 128, TILES),  # 70 and 72 tiles
])
def test_small_dgemm_clusters(m, n, k, kernel):
    assert dgemm_route(m, n, k, tma=False).kernel == kernel


@pytest.mark.parametrize("m,n,k,cluster", [
    (128, 960, 4000, 8), (128, 1024, 1500, 8), (128, 1152, 2048, 0), (160, 558, 3017, 0),  # 15, 16, 18 tiles
    (128, 2112, 1500, 4), (128, 2304, 511, 4), (128, 2304, 1500, 0), (128, 2368, 4000, 0),  # 33, 36, 37 tiles
    (1024, 576, 4000, 2),  # 72 tiles
])
def test_sgemm_clusters_that_share_sms(m, n, k, cluster):
    assert sgemm_route(m, n, k).cluster == cluster


@pytest.mark.parametrize("n,kernel", [(1300, WS_64), (1500, WS_64), (1700, TMA_128), (2048, TMA_128), (2200, WS_64),
                                      (2400, WS_64), (2700, TMA_128), (2876, TMA_128), (2950, WS_64), (3600, TMA_128)])
def test_triangle_tiles(n, kernel):
    assert dgemm_route(n, n, 1335, tri=1).kernel == kernel
