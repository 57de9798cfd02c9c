"""Batched FP64 TRSM at the edges of its blocks, chunks and column groups (GPU).

Orders around the 64-row blocks and 16-deep chunks (a ragged block is solved
first for an upper triangle, last for a lower one), right-hand sides around the
8-column tiles and the 32 columns of a work item, odd and padded leading
dimensions, every triangle / transpose / diagonal, alpha != 1, against the CPU
oracle: |X - X_oracle| <= 1e-11 (1 + |X_oracle|) for the well-conditioned
triangles used; padding rows of B stay bit-exact.
"""
from __future__ import annotations

import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORDERS = [1, 15, 31, 33, 63, 64, 65, 80, 127, 128, 133, 192, 195, 257]
RHS = [1, 8, 9, 31, 32, 33, 64]


@pytest.mark.parametrize("uplo,trans,diag", list(itertools.product("UL", "NT", "NU")))
def test_trsm_batch_edges(blas, oracle, uplo, trans, diag):
    import torch
    rng = np.random.default_rng(12)
    sizes = list(itertools.product(ORDERS, RHS))
    host, dev = [], []
    for i, (n, r) in enumerate(sizes):
        lda, ldb = n + i % 3, n + i % 2
        a = rng.standard_normal((lda, n)) * 0.5 / np.sqrt(n)
        a[np.arange(n), np.arange(n)] = 2.0 + np.abs(rng.standard_normal(n))
        a[n:] = -999.0
        b = rng.standard_normal((ldb, r))
        b[n:] = -999.0
        host.append((np.asfortranarray(a), np.asfortranarray(b), lda, ldb))
        dev.append((torch.from_numpy(np.ascontiguousarray(a.T)).cuda(), torch.from_numpy(np.ascontiguousarray(b.T)).cuda()))
    batch = blas.TrsmBatch([n for n, _ in sizes], [r for _, r in sizes], uplo=uplo, transa=trans, diag=diag)
    assert batch.info()["items"] == len(sizes)
    ptr = [torch.tensor([d[j].data_ptr() for d in dev], dtype=torch.int64, device="cuda") for j in (0, 1)]
    ld = [torch.tensor([h[j] for h in host], dtype=torch.int32, device="cuda") for j in (2, 3)]
    batch.run(-0.75, ptr[0], ld[0], ptr[1], ld[1])
    torch.cuda.synchronize()
    for (n, r), (a, b, lda, ldb), (_, x) in zip(sizes, host, dev):
        ref = b.copy(order="F")
        oracle.trsm("L", uplo, trans, diag, n, r, -0.75, a, lda, ref, ldb)
        got = x.cpu().numpy().T
        assert np.all(np.abs(got[:n] - ref[:n]) <= 1e-11 * (1 + np.abs(ref[:n]))), (n, r)
        assert np.array_equal(got[n:], b[n:]), (n, r)
