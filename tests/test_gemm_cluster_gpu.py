"""Small GEMMs on cluster tiles against the CPU oracle (GPU).

DGEMM on 64 x 64 tiles with K split over a cluster of four, SGEMM on 128 x 64
tiles over clusters of 1 to 8: edges of the tiles, remainders, K ranges that
leave the last ranks of a cluster little or nothing to do, every transpose pair,
odd and padded leading dimensions, one launch per product.  Bound:
|C - C_oracle| <= 4 k u (|alpha| |op(A)| |op(B)| + |beta| |C0|); padding rows
of C stay bit-exact.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_dgemm_tiles_gpu import TRANS, _case

pytestmark = pytest.mark.gpu

F64_SHAPES = [(128, 128, 128), (65, 63, 129), (64, 64, 255), (20, 400, 130), (256, 256, 256), (500, 512, 512)]
F32_SHAPES = [(128, 64, 1), (17, 33, 15), (129, 65, 127), (256, 256, 129),  # clusters of 1 and 8
              (300, 500, 33), (512, 512, 512), (900, 450, 100), (1024, 1024, 65)]  # 4, 4, 2, 1


@pytest.mark.parametrize("ta,tb", TRANS)
@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("shape", F64_SHAPES)
def test_small_dgemm(blas, oracle, lib, ta, tb, pad, shape):
    m, n, k = shape
    before = lib.zynum_blas_gpu_launch_count()
    _case(blas, oracle, ta, tb, m, n, k, pad, 2 * pad, 3 * pad, 1.5, -0.5, True, 3)
    assert lib.zynum_blas_gpu_launch_count() - before == 1


@pytest.mark.parametrize("ta,tb", TRANS)
@pytest.mark.parametrize("pad", [0, 3])
@pytest.mark.parametrize("shape", F32_SHAPES)
def test_small_sgemm(blas, oracle, lib, ta, tb, pad, shape):
    m, n, k = shape
    _case(blas, oracle, ta, tb, m, n, k, pad, pad, 2 * pad, 1.5, -0.5, True, 4, dtype=np.float32)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("uplo", ["U", "L"])
@pytest.mark.parametrize("n,k", [(300, 200), (130, 520)])
def test_small_triangle(blas, lib, dtype, uplo, n, k):
    import torch
    rng = np.random.default_rng(6)
    a = rng.uniform(-1, 1, (n, k)).astype(dtype)
    c0 = rng.uniform(-1, 1, (n, n)).astype(dtype)
    t_a, t_c = torch.from_numpy(np.ascontiguousarray(a.T)).cuda(), torch.from_numpy(np.ascontiguousarray(c0.T)).cuda()
    if dtype == np.float64:
        blas.dsyrk_device(uplo, "N", n, k, 1.5, t_a, n, 0.5, t_c, n)
    else:
        st = lib.zynum_blas_gpu_ssyrk_device(uplo.encode(), b"N", n, k, 1.5, t_a.data_ptr(), n, 0.5, t_c.data_ptr(), n,
                                             torch.cuda.current_stream().cuda_stream)
        assert st == 0
    c = t_c.cpu().numpy().T
    a64, c64 = a.astype(np.float64), c0.astype(np.float64)
    u = 2.0 ** -53 if dtype == np.float64 else 2.0 ** -24
    # 4 k u for the library and k 2^-53 for the float64 reference
    bound = (4 * k * u + k * 2.0 ** -53) * (1.5 * np.abs(a64) @ np.abs(a64).T + 0.5 * np.abs(c64))
    keep = np.triu(np.ones((n, n), bool)) if uplo == "U" else np.tril(np.ones((n, n), bool))
    assert np.all(np.abs(c - (1.5 * a64 @ a64.T + 0.5 * c64))[keep] <= bound[keep])
    assert np.array_equal(c[~keep], c0[~keep])
