"""Batched FP64 TRSM around the number of CTAs that hold its work items (GPU).

The CTAs claim items from a counter: batches of fewer items than CTAs, as many,
and a few more, of one and of several blocks.  alpha != 1 shows an item solved
twice, or never.  |X - X_oracle| <= 1e-11 (1 + |X_oracle|).
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("uplo,trans", [("L", "N"), ("U", "T"), ("U", "N")])
@pytest.mark.parametrize("count", [1, 2, 147, 149, 443, 444, 445, 900])
@pytest.mark.parametrize("n,r", [(5, 3), (65, 33), (130, 8)])
def test_every_item_once(blas, oracle, uplo, trans, count, n, r):
    import torch
    rng = np.random.default_rng(count)
    a = np.tril(rng.standard_normal((n, n)) * 0.5 / np.sqrt(n), -1) + np.diag(2.0 + rng.uniform(0, 1, n))
    a = np.asfortranarray(a if uplo == "L" else a.T)
    b = rng.standard_normal((count, r, n))  # problem, column, row
    ta, tb = torch.from_numpy(np.ascontiguousarray(a.T)).cuda(), torch.from_numpy(b).cuda()
    batch = blas.TrsmBatch([n] * count, [r] * count, uplo=uplo, transa=trans)
    pa = torch.full((count,), ta.data_ptr(), dtype=torch.int64, device="cuda")
    pb = torch.tensor([tb[q].data_ptr() for q in range(count)], dtype=torch.int64, device="cuda")
    ld = torch.full((count,), n, dtype=torch.int32, device="cuda")
    batch.run(-0.75, pa, ld, pb, ld)
    batch.run(2.0, pa, ld, pb, ld)  # the counter starts again
    ref = np.asfortranarray(b.reshape(count * r, n).T)
    oracle.trsm("L", uplo, trans, "N", n, count * r, -0.75, a, n, ref, n)
    oracle.trsm("L", uplo, trans, "N", n, count * r, 2.0, a, n, ref, n)
    got = tb.cpu().numpy().reshape(count * r, n).T
    assert np.all(np.abs(got - ref) <= 1e-11 * (1 + np.abs(ref)))
