"""Native DGEMM on the 64 x 64 warp-specialised tiles against the CPU oracle (GPU).

Shapes the planner sends there: about one tile per SM with K split over a
cluster of two CTAs (one launch, where the split-K workspace route takes two),
several waves whose 128 x 128 tiles would fill the last one badly, ragged M / N / K
tails, every transpose pair, and the triangle mode.  Bound:
|C - C_oracle| <= 4 k u (|alpha| |op(A)| |op(B)| + |beta| |C0|); padding rows
of C stay bit-exact.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_dgemm_tiles_gpu import TRANS, U64, _case

pytestmark = pytest.mark.gpu


def _launches(lib):
    return lib.zynum_blas_gpu_launch_count()


@pytest.mark.parametrize("ta,tb", TRANS)
@pytest.mark.parametrize("shape", [
    (1024, 512, 512),   # 128 tiles: cluster of 2, whole tiles and slices
    (1001, 450, 301),   # cluster of 2, ragged, the last rank's K range shorter
    (770, 449, 1023),   # cluster of 2, two full K tails
    (641, 514, 256),    # cluster of 2, one row and two columns past the last whole tile
    (1200, 1100, 257),  # no split, 342 tiles, K tail of 1
])
def test_ws_tiles_match_oracle(blas, oracle, lib, ta, tb, shape):
    m, n, k = shape
    # even leading dimensions (TMA-describable) whatever the size
    even = lambda x: x % 2  # noqa: E731
    ar, br = (m if ta == "N" else k), (k if tb == "N" else n)
    before = _launches(lib)
    _case(blas, oracle, ta, tb, m, n, k, even(ar), even(br), 3, -1.25, 0.75, True, 7)
    assert _launches(lib) - before == 1


def test_ws_tiles_beta_zero_overwrites_nan(blas, lib):
    import torch
    m, n, k = 1024, 512, 512
    a = torch.rand((k, m), dtype=torch.float64, device="cuda")
    b = torch.rand((n, k), dtype=torch.float64, device="cuda")
    c = torch.full((n, m), float("nan"), dtype=torch.float64, device="cuda")
    blas.dgemm_device("N", "N", m, n, k, 1.0, a, m, b, k, 0.0, c, m)
    assert torch.isfinite(c).all()


@pytest.mark.parametrize("uplo", ["U", "L"])
@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("n,k", [(1700, 300), (700, 600)])  # no split; cluster of two
def test_ws_tiles_triangle(blas, uplo, trans, n, k):
    import torch
    rng = np.random.default_rng(3)
    a = rng.uniform(-1, 1, (n, k))
    c0 = rng.uniform(-1, 1, (n, n))
    ta = torch.from_numpy(np.ascontiguousarray(a.T if trans == "N" else a)).cuda()
    tc = torch.from_numpy(np.ascontiguousarray(c0.T)).cuda()
    blas.dsyrk_device(uplo, trans, n, k, 1.5, ta, n if trans == "N" else k, 0.5, tc, n)
    c = tc.cpu().numpy().T
    ref = 1.5 * (a @ a.T) + 0.5 * c0
    # 4 k u for the library and k u for the float64 reference
    bound = 5 * k * U64 * (1.5 * (np.abs(a) @ np.abs(a).T) + 0.5 * np.abs(c0))
    keep = np.triu(np.ones((n, n), bool)) if uplo == "U" else np.tril(np.ones((n, n), bool))
    assert np.all(np.abs(c - ref)[keep] <= bound[keep])
    assert np.array_equal(c[~keep], c0[~keep])
