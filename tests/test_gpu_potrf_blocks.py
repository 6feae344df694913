"""Cholesky at the edges of its blocks (64-column steps, 256-column blocks, the
look-ahead above), the other triangle untouched, and INFO at every kind of
position.  Bound of the backward error: 4 * n * 2^-53 * |L||L^T|."""
from __future__ import annotations

import numpy as np
import pytest

import flens_gb300 as fg
import oracle

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _spd(n, seed):
    G = oracle.uniform(seed, n, n)
    return G @ G.T / n + np.eye(n)


def _potrf(cuda, uplo, A0):
    import torch
    A = fg.to_colmajor(torch.from_numpy(A0).to(cuda))
    info = torch.full((1,), -7, dtype=torch.int32, device=cuda)
    fg.dpotrf_dev(uplo, A, info)
    fg.sync()
    return A, int(info.item())


@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("n", [1, 2, 33, 63, 64, 65, 127, 256, 257, 320, 513, 900, 2100])
def test_factor(cuda, uplo, n):
    import torch
    A0 = _spd(n, n)
    low = np.tril(np.ones((n, n), dtype=bool))
    keep = ~low if uplo == "L" else ~low.T
    A0[keep] = np.nan                                  # never read
    A, info = _potrf(cuda, uplo, A0)
    assert info == 0
    got = A.cpu().numpy()
    assert np.all(np.isnan(got[keep]))
    S = torch.from_numpy(np.where(keep, 0.0, A0)).to(cuda)
    S = S + (S.t() if uplo == "L" else S.t()) - torch.diag(torch.diagonal(S))
    L = torch.from_numpy(np.where(keep, 0.0, got)).to(cuda)
    L = L if uplo == "L" else L.t()
    assert bool(((L @ L.t() - S).abs() <= 4 * n * U * (L.abs() @ L.t().abs())).all())


@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("f", [0, 1, 31, 32, 62, 63, 64, 100, 255, 256, 300, 511, 699])
@pytest.mark.parametrize("bad", [-1.0, np.nan])
def test_info_and_leading_part(cuda, uplo, f, bad):
    n = 700
    A0 = _spd(n, 5)
    want, info = _potrf(cuda, uplo, A0)
    assert info == 0
    A0[f, f] = bad
    A, info = _potrf(cuda, uplo, A0)
    assert info == f + 1
    tri = np.tril if uplo == "L" else np.triu
    a, w = A.cpu().numpy(), want.cpu().numpy()
    assert np.array_equal(tri(a[:f, :f]), tri(w[:f, :f]))
    other = np.triu(np.ones((n, n), dtype=bool), 1) if uplo == "L" else np.tril(np.ones((n, n), dtype=bool), -1)
    assert np.array_equal(a[other], A0[other])


def test_failure_in_the_last_block_stays_with_its_call(cuda):
    """Calls on two streams by one thread share the host's INFO word: a failure in one
    call's last block does not stop the other."""
    import torch
    n = 700
    good = _spd(n, 5)
    bad = good.copy()
    bad[n - 3, n - 3] = -1.0
    want, _ = _potrf(cuda, "L", good)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(20):
        A = [fg.to_colmajor(torch.from_numpy(x).to(cuda)) for x in (bad, good)]
        info = [torch.zeros(1, dtype=torch.int32, device=cuda) for _ in A]
        torch.cuda.synchronize()
        for s, a, i in zip(streams, A, info):
            with torch.cuda.stream(s):
                fg.dpotrf_dev("L", a, i)
        torch.cuda.synchronize()
        assert [int(i.item()) for i in info] == [n - 2, 0]
        assert torch.equal(torch.tril(A[1]), torch.tril(want))


@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("n", [2, 64, 130])
@pytest.mark.parametrize("e", [-1064, -1020, 0, 1016])
def test_pivots_at_the_ends_of_the_range(cuda, uplo, n, e):
    """2^e M, M of small integers: pivots whose reciprocal overflows (e = -1064) or
    is subnormal (e = 1016).  Same bound, plus n units of the last subnormal."""
    r = np.random.default_rng(n)
    M = r.integers(-1, 2, (n, n)) * (r.random((n, n)) < 0.2)
    M = (np.tril(M, -1) + np.tril(M, -1).T + np.diag(r.integers(100, 127, n))).astype(np.float64)
    A, info = _potrf(cuda, uplo, np.ldexp(M, e))
    assert info == 0
    L = A.cpu().numpy()
    L = np.ldexp(np.tril(L) if uplo == "L" else np.triu(L).T, -(e // 2))
    tol = 4 * n * U * (np.abs(L) @ np.abs(L).T) + n * 2.0 ** (-1074 - e)
    assert np.all(np.abs(L @ L.T - M) <= tol)


@pytest.mark.parametrize("uplo", "LU")
def test_reciprocal_of_the_pivot(cuda, uplo):
    """Blocks [d 1; 1 c] with c a little above 1/d: L22^2 = c - 1/d shows the
    reciprocal's own error, bounded by its rounding plus the root's 2^-52 L22^2."""
    from fractions import Fraction
    n = 128
    d = np.random.default_rng(3).uniform(1.0, 4.0, n // 2)
    c = (1.0 / d) * (1.0 + 2.0 ** -20)
    A0 = np.zeros((n, n))
    A0[0::2, 0::2] = np.diag(d)
    A0[1::2, 1::2] = np.diag(c)
    A0[0::2, 1::2] = A0[1::2, 0::2] = np.eye(n // 2)
    A, info = _potrf(cuda, uplo, A0)
    assert info == 0
    L22 = np.diagonal(A.cpu().numpy())[1::2]
    for di, ci, li in zip(d, c, L22):
        want = 1 / Fraction(float(di))
        got = Fraction(float(ci)) - Fraction(float(li)) ** 2
        assert abs(got - want) <= want * Fraction(1, 2 ** 53) + Fraction(float(li)) ** 2 / 2 ** 51


@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("n,first", [(64, 0), (64, 1), (64, 33), (40, 39), (150, 70), (700, 300)])
@pytest.mark.parametrize("e", [-200, 124, 126, 300])
def test_pivots_that_cross_the_range(cuda, uplo, n, first, e):
    """D A D with D = 2^e from row `first` on: the bound is that of A, entry by entry."""
    d = np.where(np.arange(n) < first, 0, e)
    A0 = np.ldexp(_spd(n, n), d[:, None] + d[None, :])
    A, info = _potrf(cuda, uplo, A0)
    assert info == 0
    L = A.cpu().numpy()
    L = np.ldexp(np.tril(L) if uplo == "L" else np.triu(L).T, -d[:, None])
    assert np.all(np.abs(L @ L.T - np.ldexp(A0, -(d[:, None] + d[None, :]))) <= 4 * n * U * (np.abs(L) @ np.abs(L).T))


@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("n,first", [(2, 1), (64, 1), (64, 33), (130, 20), (130, 64), (700, 300)])
def test_rows_whose_products_overflow(cuda, uplo, n, first):
    """D A D with D = 2^100, from row `first` on 2^500: the pivots before it are in the
    middle of the range, the product of two entries below them is not.  The bound is
    that of A, entry by entry."""
    d = np.where(np.arange(n) < first, 100, 500)
    A0 = np.ldexp(_spd(n, n), d[:, None] + d[None, :])
    A, info = _potrf(cuda, uplo, A0)
    assert info == 0
    L = A.cpu().numpy()
    L = np.ldexp(np.tril(L) if uplo == "L" else np.triu(L).T, -d[:, None])
    assert np.all(np.abs(L @ L.T - np.ldexp(A0, -(d[:, None] + d[None, :]))) <= 4 * n * U * (np.abs(L) @ np.abs(L).T))


@pytest.mark.parametrize("uplo", "LU")
def test_overflow_is_not_a_failed_pivot(cuda, uplo):
    """[2^200 2^600; 2^600 c]: positive definite for c = 2^1001, not for c = 2^999, whose
    pivot -2^999 is stored."""
    for c, want in ((2.0 ** 1001, 0), (2.0 ** 999, 2)):
        A, info = _potrf(cuda, uplo, np.array([[2.0 ** 200, 2.0 ** 600], [2.0 ** 600, c]]))
        got = A.cpu().numpy()
        assert info == want
        assert got[1, 1] == (2.0 ** 500 if want == 0 else -2.0 ** 999)
        assert got[0, 0] == 2.0 ** 100 and (got[1, 0] if uplo == "L" else got[0, 1]) == 2.0 ** 500


@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("n,f", [(64, 10), (200, 0), (200, 70), (256, 255), (300, 130), (500, 200), (513, 300),
                                 (700, 63), (700, 64), (700, 250), (700, 400), (700, 699)])
def test_what_a_failed_pivot_leaves(cuda, uplo, n, f):
    """A(f, f) = -2: rows and columns behind the failing 64-column step hold A minus the
    updates of the whole steps before it, its own block's columns behind f are as they
    were, and no quotient by the failing pivot is anywhere.  Each entry is one sum of at
    most n products: 2 n 2^-53 (|A| + |L||L^T|)."""
    A0 = _spd(n, 7)
    A0[f, f] = -2.0
    A, info = _potrf(cuda, uplo, A0)
    assert info == f + 1
    got = A.cpu().numpy()
    got = np.tril(got) if uplo == "L" else np.triu(got).T
    c = f // 64 * 64
    b = min(c + 64, n)                                 # the failing step's block: rows and columns c .. b - 1
    L = got[:, :c]
    want = np.tril(A0 - L @ L.T)
    want[:, :c] = 0.0
    tol = 2 * n * U * (np.abs(A0) + np.abs(L) @ np.abs(L).T)
    rest = np.tril(np.ones((n, n), dtype=bool))
    rest[:, :c] = False
    rest[c:b, c:f + 1] = False                         # written by the step itself
    assert np.all(np.abs(got - want)[rest] <= tol[rest])
    # the leading columns: L L^T = A in all rows before the step's, and below
    lead = np.tril(np.ones((n, n), dtype=bool))[:, :c]
    assert np.all((np.abs(L @ L.T - A0)[:, :c] <= tol[:, :c])[lead])


@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("at", [0, 1, 29, 30, 40, 60])
@pytest.mark.parametrize("a,b", [(-540, -540), (-500, -520), (-560, -480)])
def test_products_below_the_range(cuda, uplo, at, a, b):
    """A pivot 2^-240 at `at`, 2^a and 2^b beside it, ones and zeros otherwise: the fill-in
    -2^(a + b + 240) is a normal number, the product of the two entries is not."""
    n = 64
    A0 = np.eye(n)
    A0[at, at] = 2.0 ** -240
    A0[at + 1, at] = A0[at, at + 1] = 2.0 ** a
    A0[at + 2, at] = A0[at, at + 2] = 2.0 ** b
    A, info = _potrf(cuda, uplo, A0)
    assert info == 0
    L = A.cpu().numpy()
    L = np.tril(L) if uplo == "L" else np.triu(L).T
    want = np.eye(n)
    want[at, at], want[at + 1, at], want[at + 2, at] = 2.0 ** -120, 2.0 ** (a + 120), 2.0 ** (b + 120)
    want[at + 2, at + 1] = -2.0 ** (a + b + 240)
    assert np.array_equal(L, want)
