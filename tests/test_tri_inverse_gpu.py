"""Inverses of diagonal blocks of badly conditioned triangles (GPU).

TRSM multiplies by the inverses of 64 x 64 diagonal blocks.  Each column of such
an inverse is a substitution, so that |L X - I| <= c u |L| |X| whatever the
conditioning, with c = 68 for 64 rows (at most 64 roundings in a sum, 4 more for
the difference, the reciprocal diagonal and its product); a complex product
rounds like 2 sqrt(2) real ones, a complex quotient like 8: c = 4 (64 + 12).
"""
from __future__ import annotations

import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = 64


def _triangle(rng, family, dtype):
    def normal(*shape):
        x = rng.standard_normal(shape)
        return x + 1j * rng.standard_normal(shape) if np.issubdtype(dtype, np.complexfloating) else x

    low = np.tril(normal(N, N), -1)
    if family == "gaussian":
        d = normal(N)
    elif family == "graded":
        d = 10.0 ** rng.uniform(-4, 4, N)
    else:
        low, d = np.clip(low.real, -2, 2) + (low - low.real), np.ones(N)
    low[np.arange(N), np.arange(N)] = d
    return low.astype(dtype)


def _check(op, x, constant):
    wide = np.clongdouble if np.iscomplexobj(op) else np.longdouble
    res = np.abs(op.astype(wide) @ x.astype(wide) - np.eye(N))
    u = np.finfo(op.dtype).eps / 2
    assert np.isfinite(x).all()
    scale = np.abs(op).astype(np.longdouble) @ np.abs(x).astype(np.longdouble)
    assert np.all(res <= constant * u * scale), float((res[scale > 0] / scale[scale > 0]).max() / u)


@pytest.mark.parametrize("family", ["gaussian", "graded", "unit"])
@pytest.mark.parametrize("uplo", ["U", "L"])
def test_leaf_inverses(blas, family, uplo):
    import torch
    rng = np.random.default_rng(2)
    blocks = 32
    n = N * blocks
    a = np.zeros((n, n))
    for q in range(blocks):
        low = _triangle(rng, family, np.float64)
        a[q * N:(q + 1) * N, q * N:(q + 1) * N] = low if uplo == "L" else low[::-1, ::-1]
    ta = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    inv = torch.zeros(blas.dtrsm_inverse_bytes(n) // 8, dtype=torch.float64, device="cuda")
    blas.dtrsm_inverse_device(uplo, "N", n, ta, n, inv)
    leaves = inv.cpu().numpy()[:n * 256].reshape(n // 256, 256, 256)  # [leaf][column][row]
    for q in range(blocks):
        o = q % 4 * N
        _check(a[q * N:(q + 1) * N, q * N:(q + 1) * N], leaves[q // 4, o:o + N, o:o + N].T, 68)


@pytest.mark.parametrize("dtype,family", [
    (d, f) for d in (np.float64, np.float32, np.complex128, np.complex64) for f in ("gaussian", "graded", "unit")
    if not (f == "graded" and d in (np.float32, np.complex64))])  # those inverses are beyond FP32's range
@pytest.mark.parametrize("uplo,trans", list(itertools.product("UL", "NT")))
def test_solve_for_the_identity(blas, lib, family, uplo, trans, dtype):
    """op(A) X = I with one block: X is the inverse itself."""
    import torch
    rng = np.random.default_rng(3)
    for _ in range(8):
        low = _triangle(rng, family, dtype)
        op = low if (uplo == "L") == (trans == "N") else low[::-1, ::-1]
        a = op if trans == "N" else op.T
        ta = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
        x = torch.eye(N, dtype=ta.dtype, device="cuda")
        if dtype == np.float64:
            blas.dtrsm_device("L", uplo, trans, "N", N, N, 1.0, ta, N, x, N)
        elif dtype == np.float32:
            st = lib.zynum_blas_gpu_strsm_device(b"L", uplo.encode(), trans.encode(), b"N", N, N, 1.0, ta.data_ptr(), N,
                                                 x.data_ptr(), N, torch.cuda.current_stream().cuda_stream)
            assert st == 0
        else:
            blas.trsm_device_c("L", uplo, trans, "N", N, N, 1.0, ta, N, x, N)
        _check(op, x.cpu().numpy().T, 4 * (N + 12) if np.iscomplexobj(op) else 68)
