"""Staged transfers of the host entry points: pageable matrices copied by several threads (GPU).

Sizes around what decides the route and the chunking (2 MB per transfer, 512 KB
slots): transfers just under and over the threshold, columns longer than a slot,
padded leading dimensions, column panels, both transposes, page-locked arrays.
The result must equal, bit for bit, the device entry point's on the same inputs,
and rows outside C's window must stay untouched.
"""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(blas, ta, tb, m, n, k, pad, beta, seed, dtype=np.float64, pinned=False):
    import torch
    rng = np.random.default_rng(seed)
    (ra, ca), (rb, cb) = ((m, k) if ta == "N" else (k, m)), ((k, n) if tb == "N" else (n, k))
    host = {}
    for x, r, c in (("a", ra, ca), ("b", rb, cb), ("c", m, n)):
        t = torch.from_numpy(rng.uniform(-1, 1, (c, r + pad)).astype(dtype))
        host[x] = t.pin_memory() if pinned else t
    c0 = host["c"].numpy().copy()
    fn = blas.dgemm if dtype == np.float64 else blas.sgemm
    fn(ta, tb, m, n, k, 1.25, host["a"].numpy().T, ra + pad, host["b"].numpy().T, rb + pad, beta, host["c"].numpy().T,
       m + pad)
    # the host entry point packs its device copies, so compare with packed device operands
    dev = {x: torch.from_numpy(np.ascontiguousarray(host[x].numpy()[:, :r])).cuda() for x, r in (("a", ra), ("b", rb))}
    dc = torch.from_numpy(np.ascontiguousarray(c0[:, :m])).cuda()
    return host["c"].numpy(), c0, dev, dc


@pytest.mark.parametrize("ta,tb,m,n,k,pad,beta", [
    ("N", "N", 512, 512, 511, 0, 0.0),       # every transfer just under 2 MB
    ("N", "T", 513, 512, 513, 3, 0.5),       # just over, several columns per slot
    ("T", "N", 700, 650, 900, 0, 1.0),
    ("N", "N", 140000, 24, 16, 5, 0.5),      # columns longer than a slot: pieces
    ("T", "N", 16, 24, 140000, 0, 0.0),
])
@pytest.mark.parametrize("pinned", [False, True])
def test_host_gemm_equals_device(blas, ta, tb, m, n, k, pad, beta, pinned):
    c, c0, dev, dc = _run(blas, ta, tb, m, n, k, pad, beta, 11, pinned=pinned)
    blas.dgemm_device(ta, tb, m, n, k, 1.25, dev["a"], dev["a"].shape[1], dev["b"], dev["b"].shape[1], beta, dc, m)
    assert np.array_equal(c[:, :m], dc.cpu().numpy())
    assert np.array_equal(c[:, m:], c0[:, m:])


@pytest.mark.parametrize("tb", ["N", "T"])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_host_gemm_panels(blas, tb, beta):
    # 2100 x 2300 x 1100: column panels; the panels' products may be split differently from
    # the whole one's, so bound the difference: each within 4 k u (|alpha| |A||B| + |beta| |C0|)
    m, n, k = 2100, 2300, 1100
    c, c0, dev, dc = _run(blas, "N", tb, m, n, k, 2, beta, 5)
    a, b = dev["a"].cpu().numpy().T, dev["b"].cpu().numpy().T
    blas.dgemm_device("N", tb, m, n, k, 1.25, dev["a"], m, dev["b"], dev["b"].shape[1], beta, dc, m)
    bound = 8 * k * 2.0 ** -53 * (1.25 * np.abs(a) @ np.abs(b if tb == "N" else b.T) + beta * np.abs(c0[:, :m]).T)
    assert np.all(np.abs(c[:, :m].T - dc.cpu().numpy().T) <= bound)
    assert np.array_equal(c[:, m:], c0[:, m:])


def test_host_gemm_from_several_threads_and_after_shutdown(blas):
    out, errors = {}, []

    def call(i):
        try:
            c, c0, dev, dc = _run(blas, "N", "N", 600, 601, 602, 1, 0.5, i)
            blas.dgemm_device("N", "N", 600, 601, 602, 1.25, dev["a"], 600, dev["b"], 602, 0.5, dc, 600)
            out[i] = np.array_equal(c[:, :600], dc.cpu().numpy()) and np.array_equal(c[:, 600:], c0[:, 600:])
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    for _ in range(2):
        threads = [threading.Thread(target=call, args=(i,)) for i in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors and all(out[i] for i in range(4))
        blas.shutdown()  # the slots are given back; the next call takes new ones
