"""Triangles with extreme entries, non-finite entries and bad conditioning (GPU).

Batched FP64 TRSM: entries whose ratio to the diagonal leaves the range of a
double although the solution does not, zero right-hand sides, Inf and NaN,
against the CPU oracle, and the residual of badly conditioned triangles.  The
solver substitutes like the oracle, so what is finite there is finite here.
"""
from __future__ import annotations

import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U64 = 2.0 ** -53
FORMS = list(itertools.product("UL", "NT"))
SIZES = list(itertools.product([2, 33, 64, 65, 130], [1, 9, 33]))


def _stored(lower, uplo, trans):
    """A whose op(A) is `lower`, turned around (row and column i become n - 1 - i) where op(A) is upper."""
    op_upper = (uplo == "U") == (trans == "N")
    op = lower[::-1, ::-1] if op_upper else lower
    return np.asfortranarray(op.T if trans == "T" else op), op_upper


def _solve(blas, uplo, trans, problems, diag="N"):
    """problems: (a, b); returns the solutions of one batch."""
    import torch
    dev = [[torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in p] for p in problems]
    batch = blas.TrsmBatch([b.shape[0] for _, b in problems], [b.shape[1] for _, b in problems], uplo=uplo, transa=trans,
                           diag=diag)
    ptr = [torch.tensor([d[j].data_ptr() for d in dev], dtype=torch.int64, device="cuda") for j in (0, 1)]
    ld = torch.tensor([b.shape[0] for _, b in problems], dtype=torch.int32, device="cuda")
    batch.run(1.0, ptr[0], ld, ptr[1], ld)
    torch.cuda.synchronize()
    return [d[1].cpu().numpy().T for d in dev]


def _oracle(oracle, uplo, trans, a, b, diag="N"):
    ref = np.asfortranarray(b)
    n, r = b.shape
    with np.errstate(all="ignore"):
        oracle.trsm("L", uplo, trans, diag, n, r, 1.0, np.asfortranarray(a), n, ref, n)
    return ref


def _lower(rng, n):
    low = np.tril(rng.standard_normal((n, n)) * 0.5 / np.sqrt(n), -1)
    low[np.arange(n), np.arange(n)] = 2.0 + np.abs(rng.standard_normal(n))
    return low


# column j of the triangle and row j of the right-hand side: the entries' ratio to the diagonal
# is beyond the largest double, or so small that it is subnormal; x_j and its products are neither
@pytest.mark.parametrize("diagonal,entry,rhs,others", [
    (1e-160, 1e160, 1e-300, 1.0), (1e-160, 1e160, 0.0, 1.0), (1e160, 1e-160, 1e300, 1e-20)])
@pytest.mark.parametrize("uplo,trans", FORMS)
def test_ratio_to_the_diagonal_outside_the_range(blas, oracle, uplo, trans, diagonal, entry, rhs, others):
    rng = np.random.default_rng(5)
    problems, j_of = [], []
    for n, r in SIZES:
        j = n // 3
        low = np.diag(1.0 + rng.uniform(0, 1, n))
        low[j, j] = diagonal
        low[j + 1:, j] = entry * rng.uniform(0.5, 1, n - j - 1)
        b = others * rng.uniform(0.5, 1, (n, r))
        b[j] = -rhs * rng.uniform(0.5, 1, r)  # negative: no cancellation in the rows below
        a, turned = _stored(low, uplo, trans)
        problems.append((a, np.asfortranarray(b[::-1] if turned else b)))
        j_of.append(j)
    for (a, b), x in zip(problems, _solve(blas, uplo, trans, problems)):
        ref = _oracle(oracle, uplo, trans, a, b)
        assert np.isfinite(ref).all()
        # x_j and then x_p: at most 6 roundings here (1 / diagonal is one of its own), 4 in the oracle
        assert np.all(np.abs(x - ref) <= 16 * U64 * np.abs(ref)), b.shape


@pytest.mark.parametrize("uplo,trans", FORMS)
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("where", ["a", "b"])
def test_non_finite_entries(blas, oracle, uplo, trans, value, where):
    rng = np.random.default_rng(6)
    problems = []
    for n, r in SIZES:
        low, b = _lower(rng, n), rng.standard_normal((n, r))
        i = 2 * n // 3
        if where == "a":
            low[i, i // 2] = value
        else:
            b[i, r // 2] = value
        a, turned = _stored(low, uplo, trans)
        problems.append((a, np.asfortranarray(b[::-1] if turned else b)))
    for (a, b), x in zip(problems, _solve(blas, uplo, trans, problems)):
        ref = _oracle(oracle, uplo, trans, a, b)
        finite = np.isfinite(ref)
        assert np.array_equal(np.isnan(x), np.isnan(ref)) and np.array_equal(np.isinf(x), np.isinf(ref)), b.shape
        assert np.array_equal(x[np.isinf(ref)], ref[np.isinf(ref)])
        assert np.all(np.abs(x[finite] - ref[finite]) <= 1e-11 * (1 + np.abs(ref[finite])))


@pytest.mark.parametrize("uplo,trans", FORMS)
@pytest.mark.parametrize("diag", ["N", "U"])
def test_only_the_stored_triangle_is_read(blas, uplo, trans, diag):
    rng = np.random.default_rng(7)
    clean, dirty = [], []
    for n, r in SIZES:
        a, _ = _stored(_lower(rng, n), uplo, trans)
        b = np.asfortranarray(rng.standard_normal((n, r)))
        bad = a.copy(order="F")
        bad[np.tril_indices(n, -1) if uplo == "U" else np.triu_indices(n, 1)] = np.nan
        if diag == "U":
            bad[np.arange(n), np.arange(n)] = np.nan
        clean.append((a, b))
        dirty.append((bad, b))
    for x, y in zip(_solve(blas, uplo, trans, clean, diag), _solve(blas, uplo, trans, dirty, diag)):
        assert np.array_equal(x, y)


def _ill_conditioned(rng, n, family):
    low = np.tril(rng.standard_normal((n, n)), -1)
    if family == "gaussian":
        d = rng.standard_normal(n)
    elif family == "graded":
        d = 10.0 ** rng.uniform(-4, 4, n)
    else:  # unit diagonal, entries up to 2
        low, d = np.tril(rng.uniform(-2, 2, (n, n)), -1), np.ones(n)
    low[np.arange(n), np.arange(n)] = d
    return low


@pytest.mark.parametrize("uplo,trans", FORMS)
@pytest.mark.parametrize("family", ["gaussian", "graded", "unit"])
def test_residual_of_ill_conditioned_triangles(blas, uplo, trans, family):
    """|b - op(A) x| <= (n + 4) u (|op(A)| |x| + |b|): substitution's bound, whatever the conditioning."""
    rng = np.random.default_rng(8)
    problems = []
    for n, r in SIZES:
        a, _ = _stored(_ill_conditioned(rng, n, family), uplo, trans)
        problems.append((a, np.asfortranarray(rng.uniform(-1, 1, (n, r)))))
    for (a, b), x in zip(problems, _solve(blas, uplo, trans, problems)):
        op = (a.T if trans == "T" else a).astype(np.longdouble)
        res = np.abs(b - op @ x)
        assert np.all(res <= (b.shape[0] + 4) * U64 * (np.abs(op) @ np.abs(x) + np.abs(b))), b.shape
