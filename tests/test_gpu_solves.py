"""Triangular solves with few right-hand sides (scaled diagonal blocks, the
chained solve), and the row permutation of the LU solves, at block edges and
for scalings where the scaled form must step aside.  Bound: the componentwise
backward error of substitution, c * n * 2^-53 * |M||x| (c = 4: prescaled rows,
the reciprocal, and the residual is taken in extended precision)."""
from __future__ import annotations

import numpy as np
import pytest

import flens_gb300 as fg
import oracle

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _residual_ok(M, X, B):
    L = np.longdouble
    n = M.shape[0]
    with np.errstate(all="ignore"):
        R = np.abs(M.astype(L) @ X.astype(L) - B.astype(L))
        bound = 4 * n * U * (np.abs(M).astype(L) @ np.abs(X).astype(L)) + L(1e-300)
    assert np.all(R <= bound)


def _tri(n, uplo, kind, seed):
    A = oracle.uniform(seed, n, n) / n
    A[np.arange(n), np.arange(n)] = 1.0 + oracle.uniform(seed + 1, n, 1)[:, 0] / 4
    if kind == "rows":                       # rows over 2^+-400: still scaled
        A = A * 2.0 ** np.random.default_rng(seed).integers(-400, 401, (n, 1))
    elif kind == "wide":                     # reciprocals beyond 2^900: unscaled
        A = A * 2.0 ** np.where(np.arange(n) % 5 == 0, -930, 0)[:, None]
    return np.asfortranarray(np.tril(A) if uplo == "L" else np.triu(A))


@pytest.mark.parametrize("n", [1, 31, 33, 64, 65, 130, 200])
@pytest.mark.parametrize("nvec", [1, 3, 4, 5, 33])
@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("kind", ["plain", "rows", "wide"])
def test_trsm_few(cuda, n, nvec, uplo, kind):
    for trans in "NT":
        A = _tri(n, uplo, kind, n)
        B = oracle.uniform(n + 9, n, nvec)
        X = fg.dtrsm("L", uplo, trans, "N", 1.0, A, B.copy(order="F"))
        _residual_ok(A if trans == "N" else A.T, X, B)


@pytest.mark.parametrize("n", [65, 130, 200])
@pytest.mark.parametrize("nvec", [1, 4])
@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("other", [np.nan, 5e-324, 2.0 ** -950, -2.0 ** 1000])
def test_other_triangle_decides_nothing(cuda, n, nvec, uplo, other):
    for trans in "NT":
        A = _tri(n, uplo, "plain", n)
        B = oracle.uniform(n + 9, n, nvec)
        want = fg.dtrsm("L", uplo, trans, "N", 1.0, A, B.copy(order="F"))
        low = np.tril(np.ones((n, n), dtype=bool))
        A[~low if uplo == "L" else ~low.T] = other
        assert np.array_equal(fg.dtrsm("L", uplo, trans, "N", 1.0, A, B.copy(order="F")), want)


def test_large_right_hand_side_that_cancels(cuda):
    """b / diagonal overflows, the solution does not."""
    n = 100
    A = _tri(n, "L", "plain", 4)
    A[:, 0] = 1e-5
    A[0, 0] = 1.0
    A[50, :] *= 2.0 ** -60
    A[50, 0] = 1.0
    A = np.asfortranarray(A)
    B = np.zeros((n, 2))
    B[0, 0] = 2.0 ** 1000
    B[:, 0] = A[:, 0] * B[0, 0]
    B[0, 1] = 1.0
    X = fg.dtrsm("L", "L", "N", "N", 1.0, A, B.copy(order="F"))
    assert np.all(np.isfinite(X))
    _residual_ok(A, X, B)


@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("at", [0, 40, 64, 100])
def test_small_entries_beside_a_large_quotient(cuda, uplo, at):
    """Diagonal matrix, exact quotients: one of 2^1010, the others near 2^-900."""
    n = 130
    d, x = np.ones(n), np.full(n, 2.0 ** -900)
    d[at], x[at] = 2.0 ** -500, 2.0 ** 1010
    x *= 1.0 + np.arange(n) / 1024.0
    X = fg.dtrsm("L", uplo, "N", "N", 1.0, np.asfortranarray(np.diag(d)), (d * x)[:, None].copy(order="F"))
    assert np.array_equal(X[:, 0], x)


@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("row,cols", [(20, (3, 7)), (50, (3, 7)), (50, (7, 40)), (90, (66, 70)), (127, (66, 120))])
def test_terms_that_cancel_beyond_the_scaled_range(cuda, uplo, row, cols):
    """2^250 (2^200 - 2^200) + 2^-600 x = 2^399, exact in FP64 in any order: no sum
    overflows but in the rows over their diagonal (2^1050)."""
    n = 130
    A, B, want = np.eye(n), np.ones((n, 2)), np.ones((n, 2))
    A[row, row] = 2.0 ** -600
    A[row, cols[0]], A[row, cols[1]] = 2.0 ** 250, -2.0 ** 250
    B[list(cols)] = want[list(cols)] = 2.0 ** 200
    B[row] = 2.0 ** 399
    want[row] = 2.0 ** 999
    if uplo == "U":
        A, B, want = A[::-1, ::-1], B[::-1], want[::-1]
    X = fg.dtrsm("L", uplo, "N", "N", 1.0, np.asfortranarray(A), np.asfortranarray(B))
    assert np.array_equal(X, want)


def test_infinite_right_hand_side(cuda):
    n = 96
    A = _tri(n, "L", "plain", 5)
    B = np.zeros((n, 1))
    B[40] = np.inf
    X = fg.dtrsm("L", "L", "N", "N", 1.0, A, B.copy(order="F"))
    assert np.all(X[:40] == 0) and np.isinf(X[40, 0]) and not np.any(np.isfinite(X[41:]))


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 129, 700, 2111])
@pytest.mark.parametrize("trans", "NT")
@pytest.mark.parametrize("nrhs", [1, 4, 16, 40])
def test_solve_with_interchanges(cuda, n, trans, nrhs):
    import torch
    A0 = fg.to_colmajor(torch.from_numpy(oracle.uniform(n, n, n)).to(cuda))
    B0 = fg.to_colmajor(torch.from_numpy(oracle.uniform(n + 1, n, nrhs)).to(cuda))
    A, X = fg.to_colmajor(A0.clone()), fg.to_colmajor(B0.clone())
    piv = torch.zeros(n, dtype=torch.int32, device=cuda)
    info = torch.zeros(1, dtype=torch.int32, device=cuda)
    fg.dgetrf_dev(A, piv, info)
    fg.dgetrs_dev(trans, A, piv, X)
    fg.sync()
    L = torch.tril(A, -1).abs()
    L.diagonal().add_(1.0)
    LU = L @ torch.triu(A).abs()
    p = piv.cpu().numpy() - 1
    perm = np.arange(n)
    for i in range(n):
        perm[[i, p[i]]] = perm[[p[i], i]]
    LU = LU[torch.from_numpy(np.argsort(perm)).to(cuda)]          # |P^T| |L| |U|
    op = (lambda M: M) if trans == "N" else (lambda M: M.t())  # noqa: E731
    R = (op(A0) @ X - B0).abs()
    assert bool((R <= 12 * n * U * (op(LU) @ X.abs()) + 4 * n * U * (op(A0).abs() @ X.abs())).all())


@pytest.mark.parametrize("side,uplo,trans,diag", [("L", "L", "N", "N"), ("L", "U", "N", "U"), ("L", "L", "T", "U"),
                                                  ("R", "U", "N", "N"), ("R", "L", "T", "N"), ("R", "L", "N", "U")])
@pytest.mark.parametrize("k", [1, 7, 8, 9, 33, 57, 64])
def test_many_vectors_both_row_layouts(cuda, side, uplo, trans, diag, k):
    """2561 vectors (cyclic rows) and the same among 6000 (consecutive rows): equal
    bits, and the substitution's own bound."""
    import torch
    g = torch.Generator(device=cuda)
    g.manual_seed(k)
    T0 = torch.rand((k, k), generator=g, dtype=torch.float64, device=cuda) - 0.5 + 2 * torch.eye(k, dtype=torch.float64, device=cuda)
    if k > 1:
        T0[0, k - 1] = 0.0                             # (off the diagonal)
    M = fg.to_colmajor(T0)
    B = torch.rand((6000, k), generator=g, dtype=torch.float64, device=cuda) - 0.5
    B = B if side == "R" else B.t()
    few = B[37:2598] if side == "R" else B[:, 37:2598]
    X, Y = fg.to_colmajor(B.clone()), fg.to_colmajor(few.clone())
    fg.dtrsm_dev(side, uplo, trans, diag, 1.0, M, X)
    fg.dtrsm_dev(side, uplo, trans, diag, 1.0, M, Y)
    fg.sync()
    assert torch.equal(Y, X[37:2598] if side == "R" else X[:, 37:2598])
    T = torch.tril(T0) if uplo == "L" else torch.triu(T0)
    if diag == "U":
        T = T - torch.diag(torch.diagonal(T)) + torch.eye(k, dtype=torch.float64, device=cuda)
    T = T.t() if trans == "T" else T
    P, Q = (Y @ T, Y.abs() @ T.abs()) if side == "R" else (T @ Y, T.abs() @ Y.abs())
    assert bool(((P - few).abs() <= 4 * (k + 1) * 2.0 ** -53 * (Q + few.abs())).all())
