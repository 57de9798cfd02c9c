"""Each TMA route of the native DGEMM against the CPU oracle, the route asserted (GPU).

The 128 x 128 tiles unsplit (the route of large products), split in two over a
cluster and in more ranges through the workspace, with ragged tails, every
transpose pair and beta != 0, and the triangle mode of the first two.  A launch
count does not tell the 64 x 64 from the 128 x 128 kernel, so the planner is asked
which one the shape takes.  Bound: |C - C_oracle| <= 4 k u (|alpha| |op(A)| |op(B)|
+ |beta| |C0|); padding rows of C stay bit-exact.
"""
from __future__ import annotations

import numpy as np
import pytest

from gemm_routes import TILES, TMA_128, WS_64, dgemm_route
from test_dgemm_tiles_gpu import TRANS, U64, _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", TRANS)
@pytest.mark.parametrize("shape,route", [
    ((1497, 1410, 301), (TMA_128, 1, 1)),  # one round of 144 tiles, ragged in all three
    ((1536, 1500, 96), (TMA_128, 1, 1)),   # whole K slices
    ((1001, 903, 1499), (TMA_128, 2, 1)),  # two K ranges in a cluster
    ((640, 514, 1057), (TMA_128, 1, 4)),   # more ranges: the workspace
    ((2050, 1930, 259), (WS_64, 1, 1)),
], ids=lambda s: "x".join(map(str, s)) if len(s) == 3 and s[0] > 16 else None)
@pytest.mark.parametrize("beta", [0.0, -0.5])
def test_routes(blas, oracle, ta, tb, shape, route, beta):
    m, n, k = shape
    assert dgemm_route(m, n, k)[2:5] == route
    even = lambda x: x % 2  # noqa: E731
    _case(blas, oracle, ta, tb, m, n, k, even(m if ta == "N" else k), even(k if tb == "N" else n), 3, 1.25, beta, True, 9)


@pytest.mark.parametrize("uplo", ["U", "L"])
@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("n,k,route", [
    (1990, 300, (TMA_128, 1, 1)),  # 136 live tiles of 128 x 128: one round
    (1000, 1500, (TMA_128, 2, 1)),
    (900, 1025, (TMA_128, 2, 1)),
    (1200, 1300, (WS_64, 1, 1)),
    (2200, 260, (WS_64, 1, 1)),
    (576, 1000, (TILES, 1, 3)),
])
def test_triangle_routes(blas, uplo, trans, n, k, route):
    import torch
    assert dgemm_route(n, n, k, tri=1)[2:5] == route
    rng = np.random.default_rng(n)
    a, c0 = rng.uniform(-1, 1, (n, k)), rng.uniform(-1, 1, (n, n))
    ta = torch.from_numpy(np.ascontiguousarray(a.T if trans == "N" else a)).cuda()
    tc = torch.from_numpy(np.ascontiguousarray(c0.T)).cuda()
    blas.dsyrk_device(uplo, trans, n, k, 1.5, ta, n if trans == "N" else k, 0.5, tc, n)
    c = tc.cpu().numpy().T
    # 4 k u for the library and k u for the float64 reference
    bound = 5 * k * U64 * (1.5 * (np.abs(a) @ np.abs(a).T) + 0.5 * np.abs(c0))
    keep = np.triu(np.ones((n, n), bool)) if uplo == "U" else np.tril(np.ones((n, n), bool))
    assert np.all(np.abs(c - (1.5 * (a @ a.T) + 0.5 * c0))[keep] <= bound[keep])
    assert np.array_equal(c[~keep], c0[~keep])


def test_more_columns_than_64_wide_tiles_reach(blas):
    """64 x 4,194,304 x 256 (11 GB): 65,536 column tiles of 64, one more than grid.y has."""
    import torch
    m, n, k = 64, 64 * 65536, 256
    assert dgemm_route(m, n, k).kernel == TMA_128
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.rand((k, m), generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    b = torch.rand((n, k), generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    c = torch.full((n, m), 7.0, device="cuda", dtype=torch.float64)
    blas.dgemm_device("N", "N", m, n, k, 1.0, a, m, b, k, 0.0, c, m)
    for at in (slice(0, 300), slice(n // 2 - 150, n // 2 + 150), slice(n - 300, n)):
        ref, scale = b[at] @ a, b[at].abs() @ a.abs()
        assert bool(((c[at] - ref).abs() <= 5 * k * U64 * scale).all())
