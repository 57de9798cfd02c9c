"""SGEMM cluster tiles whose CTAs sum their K range in two halves, against the CPU oracle (GPU).

Products planned with more K ranges than a cluster has CTAs: clusters of 8, 4
and 2, tile edges, K remainders, every transpose pair, odd leading dimensions.
Bound: |C - C_oracle| <= 4 k u (|alpha| |op(A)| |op(B)| + |beta| |C0|).
"""
from __future__ import annotations

import numpy as np
import pytest

from gemm_routes import sgemm_route
from test_dgemm_tiles_gpu import TRANS, _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", TRANS)
@pytest.mark.parametrize("pad", [0, 3])
@pytest.mark.parametrize("shape,cluster", [
    ((256, 256, 2560), 8), ((129, 65, 2310), 8), ((300, 300, 4000), 8),
    ((512, 512, 1300), 4), ((600, 600, 801), 2),
], ids=lambda s: "x".join(map(str, s)) if isinstance(s, tuple) else None)
def test_sgemm_halves(blas, oracle, lib, ta, tb, pad, shape, cluster):
    m, n, k = shape
    assert sgemm_route(m, n, k)[1:] == (cluster, 1)
    before = lib.zynum_blas_gpu_launch_count()
    _case(blas, oracle, ta, tb, m, n, k, pad, pad, 2 * pad, 1.5, -0.5, True, 4, dtype=np.float32)
    assert lib.zynum_blas_gpu_launch_count() - before == 1
