"""The FP64 product by exact residues on the tensor cores (mod_gemm.cu), as
dgemm and dsyrk take it for large products.

Exactness: integer operands give the integer product itself.  Accuracy: sampled
elements against rational arithmetic, with the route's own bound (rounding of
the operands below 4 * 2^-53 * |A||B|, one rounding of the sum, one or two of C).
Tiles the data check refuses (graded rows, non-finite entries, extreme
exponents) come from the FP64 kernel and meet its bound k * 2^-53 * |A||B|.
"""
from __future__ import annotations

import ctypes
from fractions import Fraction

import numpy as np
import pytest

import flens_gb300 as fg

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _dev(cuda, X, pad=0):
    import torch
    r, c = X.shape
    t = torch.zeros((c, r + pad), dtype=torch.float64, device=cuda).t()[:r]
    t.copy_(torch.from_numpy(np.ascontiguousarray(X)))
    return t


def _gemm(cuda, ta, tb, alpha, A, B, beta, C, pad=0):
    """The product and the number of kernels it took (1: the FP64 kernel alone)."""
    dA, dB, dC = _dev(cuda, A, pad), _dev(cuda, B, pad), _dev(cuda, C, pad)
    before = fg.lib().flens_gb300_launch_count()
    fg.dgemm_dev(ta, tb, alpha, dA, dB, beta, dC)
    used = fg.lib().flens_gb300_launch_count() - before
    fg.sync()
    return dC.cpu().numpy(), used


def _op(X, t):
    return X if t == "N" else X.T


# tile edges (128 x 256), one and several 1024-deep chunks, two k blocks (4097)
SHAPES = [(300, 300, 300), (128, 256, 1024), (129, 257, 1025), (513, 255, 640), (257, 1100, 100),
          (200, 100, 4097), (2000, 40, 2050)]


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("ta,tb", ["NN", "NT", "TN", "TT"])
def test_integer_products_exact(cuda, m, n, k, ta, tb):
    r = np.random.default_rng(m + n + k)
    lim = 1 << 19
    A = r.integers(-lim, lim + 1, (m, k) if ta == "N" else (k, m)).astype(np.float64)
    B = r.integers(-lim, lim + 1, (k, n) if tb == "N" else (n, k)).astype(np.float64)
    C = r.integers(-lim, lim + 1, (m, n)).astype(np.float64)
    got, used = _gemm(cuda, ta, tb, -1.0, A, B, 2.0, C, pad=3)
    assert used >= 5, "the FP64 kernel alone"
    want = 2 * C.astype(np.int64) - _op(A, ta).astype(np.int64) @ _op(B, tb).astype(np.int64)
    assert np.array_equal(got.astype(np.int64), want)


@pytest.mark.parametrize("m,n,k,spread", [(400, 500, 300, 0), (300, 300, 3000, 2), (1500, 600, 64, 1)])
def test_accuracy_sampled(cuda, m, n, k, spread):
    r = np.random.default_rng(k)
    A = r.uniform(-1, 1, (m, k)) * 2.0 ** r.integers(-40, 41, (m, 1)) * 2.0 ** r.integers(-spread, spread + 1, (m, k))
    B = r.uniform(-1, 1, (k, n)) * 2.0 ** r.integers(-40, 41, (1, n))
    C = np.zeros((m, n))
    got, used = _gemm(cuda, "N", "N", 1.0, A, B, 0.0, C)
    assert used >= 5
    for i, j in zip(r.integers(0, m, 60), r.integers(0, n, 60)):
        ex = sum(Fraction(a) * Fraction(b) for a, b in zip(A[i].tolist(), B[:, j].tolist()))
        mag = float(np.abs(A[i]) @ np.abs(B[:, j]))
        assert abs(Fraction(got[i, j]) - ex) <= Fraction(4 * U * mag + U * abs(float(ex)))


@pytest.mark.parametrize("E", [4, 8, 12, 16, 24])
def test_wide_entries(cuda, E):
    """Entries u 2^e, e uniform in [-E, E]: accurate whether a tile is accepted or
    refused (the bound of the FP64 sum, with 4 for the operands' rounding)."""
    r = np.random.default_rng(E)
    m, n, k = 300, 520, 1500
    A = np.ldexp(r.uniform(-1, 1, (m, k)), r.integers(-E, E + 1, (m, k)))
    B = np.ldexp(r.uniform(-1, 1, (k, n)), r.integers(-E, E + 1, (k, n)))
    got, used = _gemm(cuda, "N", "N", 1.0, A, B, 0.0, np.zeros((m, n)))
    assert used >= 5
    L = np.longdouble
    for i in r.integers(0, m, 12):
        ex = A[i].astype(L) @ B.astype(L)
        mag = np.abs(A[i]) @ np.abs(B)
        err = np.abs(got[i].astype(L) - ex).astype(np.float64) / (U * mag)
        assert err.max() <= (4.5 if E <= 8 else np.sqrt(k) + 4.5)


@pytest.mark.parametrize("m,n,k", [(300, 300, 1024), (300, 300, 513), (257, 300, 1025), (200, 270, 2048), (150, 300, 3072)])
def test_sums_at_the_edge_of_fp32(cuda, m, n, k):
    """Rows and columns constant but for their last entry, with odd significands of as
    many bits (53, from k = 1025 on 52) as make every residue modulo 256 one of 128: a
    full chunk's sum is 2^24 in magnitude.  The operands are exact, the result is the
    sum rounded once."""
    r = np.random.default_rng(k)
    bits = 53 if k <= 1024 else 52

    def odd(size):
        v = (r.integers(1 << (bits - 2), 1 << (bits - 1), size) * 2 + 1).astype(np.float64)
        return v * 2.0 ** -bits * np.where(r.random(size) < 0.5, -1.0, 1.0)

    A, B = np.repeat(odd((m, 1)), k, 1), np.repeat(odd((1, n)), k, 0)
    A[:, -1], B[-1] = odd(m), odd(n)
    got, used = _gemm(cuda, "N", "N", 1.0, A, B, 0.0, np.zeros((m, n)))
    assert used >= 5
    a, a1, b, b1 = ([Fraction(x) for x in v.tolist()] for v in (A[:, 0], A[:, -1], B[0], B[-1]))
    for i in range(m):
        assert got[i].tolist() == [float((k - 1) * a[i] * b[j] + a1[i] * b1[j]) for j in range(n)]


@pytest.mark.parametrize("k", [200, 300, 1000, 1500])
@pytest.mark.parametrize("e", [-13, -11, -10, -9, -8, -7, -6, -5, -1])
@pytest.mark.parametrize("swap", [False, True])
def test_products_of_one_term_are_exact(cuda, k, e, swap):
    """A I and I A for A bidiagonal, 1 on the diagonal and 53-bit entries in [2^e,
    2^(e+1)) beside it: the FP64 sum is A itself."""
    r = np.random.default_rng(k - e)
    A = np.eye(k)
    A[np.arange(k - 1), np.arange(1, k)] = np.ldexp(1.0 + r.integers(0, 1 << 52, k - 1) * 2.0 ** -52, e)
    A, B = (np.eye(k), A) if swap else (A, np.eye(k))
    got, used = _gemm(cuda, "N", "N", 1.0, A, B, 0.0, np.zeros((k, k)))
    assert used >= 5 or k < 300
    assert np.array_equal(got, B if swap else A)


@pytest.mark.parametrize("beta", [1.0, -0.5])
def test_c_is_rounded_once_whatever_the_depth(cuda, beta):
    """k = 8200 is summed in parts; C is 2^30 times the product: one rounding of
    the result, one of beta*C (exact here), and 8 * 2^-53 |A||B|."""
    r = np.random.default_rng(13)
    m, n, k = 130, 140, 8200
    A, B = r.uniform(-1, 1, (m, k)), r.uniform(-1, 1, (k, n))
    C = r.uniform(-1, 1, (m, n)) * 2.0 ** 30
    got, used = _gemm(cuda, "N", "N", 1.0, A, B, beta, C)
    assert used >= 10
    for i, j in zip(r.integers(0, m, 60), r.integers(0, n, 60)):
        ex = Fraction(beta) * Fraction(float(C[i, j])) + sum(
            Fraction(a) * Fraction(b) for a, b in zip(A[i].tolist(), B[:, j].tolist()))
        mag = float(np.abs(A[i]) @ np.abs(B[:, j]))
        assert abs(Fraction(float(got[i, j])) - ex) <= Fraction(U) * abs(ex) + Fraction(8 * U * mag)


@pytest.mark.parametrize("uplo", "LU")
def test_deep_triangle(cuda, uplo):
    """syrk with k in two parts and C in four blocks: integers, the other triangle kept."""
    import torch
    n, k = 4200, 5000
    g = torch.Generator(device=cuda)
    g.manual_seed(2)
    A = torch.randint(-9, 10, (k, n), generator=g, device=cuda).double().t()
    C0 = torch.randint(-9, 10, (n, n), generator=g, device=cuda).double().t()
    C = fg.to_colmajor(C0.clone())
    fg.dsyrk_dev(uplo, "N", 2.0, A, -1.0, C)
    fg.sync()
    want = 2 * (A @ A.t()) - C0
    tri = torch.tril if uplo == "L" else torch.triu
    assert torch.equal(tri(C), tri(want))
    other = torch.triu(C0, 1) if uplo == "L" else torch.tril(C0, -1)
    assert torch.equal(torch.triu(C, 1) if uplo == "L" else torch.tril(C, -1), other)


def test_few_terms_keep_the_fp64_bound(cuda):
    """Rows of A with 1 to 6 nonzeros in a 300^3 product: n nonzero terms, n * 2^-53 *
    |A||B| in each element."""
    r = np.random.default_rng(11)
    m = n = k = 300
    B = r.uniform(0.25, 1.0, (k, n))
    A = np.zeros((m, k))
    for i in range(m):
        at = r.choice(k, 1 + i % 6, replace=False)
        A[i, at] = r.uniform(0.5, 1.0, at.size) * 2.0 ** -r.integers(0, 10, at.size)
    got, used = _gemm(cuda, "N", "N", 1.0, A, B, 0.0, np.zeros((m, n)))
    assert used >= 5
    for i in range(m):
        at = np.flatnonzero(A[i])
        for j in range(0, n, 7):
            terms = [Fraction(float(A[i, x])) * Fraction(float(B[x, j])) for x in at]
            assert abs(Fraction(float(got[i, j])) - sum(terms)) <= at.size * Fraction(1, 1 << 53) * sum(terms)


def _refused(cuda, A, B, C, alpha=1.0, beta=1.0):
    k = A.shape[1]
    got, used = _gemm(cuda, "N", "N", alpha, A, B, beta, C)
    assert used >= 5
    with np.errstate(all="ignore"):
        want = beta * C + alpha * (A @ B)
        mag = abs(beta) * np.abs(C) + np.abs(alpha) * (np.abs(A) @ np.abs(B))
    fin = np.isfinite(want)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[~fin & ~np.isnan(want)], want[~fin & ~np.isnan(want)])
    with np.errstate(all="ignore"):
        assert np.all(np.abs(got - want)[fin] <= (2 * (k + 2) * U * mag)[fin])


def test_graded_rows_keep_fp64_accuracy(cuda):
    """One large entry per row where B is tiny: fixed point would lose the rest."""
    r = np.random.default_rng(5)
    A, B, C = r.uniform(-1, 1, (400, 300)), r.uniform(-1, 1, (300, 600)), np.zeros((400, 600))
    A[:200, 0] *= 1e25
    B[0, :300] *= 1e-25
    _refused(cuda, A, B, C)


def test_special_values(cuda):
    r = np.random.default_rng(6)
    A, B, C = r.uniform(-1, 1, (400, 300)), r.uniform(-1, 1, (300, 600)), r.uniform(-1, 1, (400, 600))
    A[3, 7], A[200, 5], B[11, 400], C[390, 590] = np.nan, np.inf, -np.inf, np.nan
    A[250], B[:, 20] = 0.0, 0.0                       # exact zeros, and 0 * Inf
    _refused(cuda, A, B, C, alpha=1.5, beta=0.0)


@pytest.mark.parametrize("ea,eb", [(900, -900), (-1000, 40), (500, 300), (-1060, 1000)])
def test_extreme_exponents(cuda, ea, eb):
    r = np.random.default_rng(7)
    A, B = np.ldexp(r.uniform(-1, 1, (300, 300)), ea), np.ldexp(r.uniform(-1, 1, (300, 300)), eb)
    _refused(cuda, A, B, np.zeros((300, 300)))


def test_zero_and_sparse_operands(cuda):
    """Columns that meet no nonzero give exact zeros; sparse rows stay accurate."""
    r = np.random.default_rng(8)
    A, B = r.uniform(-1, 1, (400, 512)), r.uniform(-1, 1, (512, 600))
    A[:, 256:] = 0.0
    B[:256, 300:] = 0.0
    A[5] = 0.0
    A[7, :] = 0.0
    A[7, 9] = 0.3
    _refused(cuda, A, B, np.zeros((400, 600)))
    got, _ = _gemm(cuda, "N", "N", 1.0, A, B, 0.0, np.zeros((400, 600)))
    assert np.all(got[:, 300:] == 0.0) and np.all(got[5] == 0.0)


@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("trans", "NT")
@pytest.mark.parametrize("n,k", [(700, 200), (257, 1100), (4400, 70)])
def test_triangle_products(cuda, uplo, trans, n, k):
    import torch
    r = np.random.default_rng(n)
    A = r.integers(-9, 10, (n, k) if trans == "N" else (k, n)).astype(np.float64)
    C = r.integers(-9, 10, (n, n)).astype(np.float64)
    dA, dC = _dev(cuda, A), _dev(cuda, C, 1)
    before = fg.lib().flens_gb300_launch_count()
    fg.dsyrk_dev(uplo, trans, -1.0, dA, 1.0, dC)
    assert fg.lib().flens_gb300_launch_count() - before >= 5
    fg.sync()
    X = torch.from_numpy(_op(A, trans)).to(cuda)
    want = C - (X @ X.t()).cpu().numpy()
    keep = np.tril(np.ones((n, n)), -1) if uplo == "U" else np.triu(np.ones((n, n)), 1)
    assert np.array_equal(dC.cpu().numpy(), np.where(keep > 0, C, want))


def test_capture_and_no_memory_take_the_fp64_kernel(cuda):
    import torch
    r = np.random.default_rng(9)
    A, B = (_dev(cuda, r.uniform(-1, 1, (500, 500))) for _ in range(2))
    C = [_dev(cuda, np.zeros((500, 500))) for _ in range(3)]
    fg.dgemm_dev("N", "N", 1.0, A, B, 0.0, C[0])
    fg.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        fg.dgemm_dev("N", "N", 1.0, A, B, 0.0, C[1])
    g.replay()
    fail = fg.lib().flens_gb300_test_fail_device_allocs
    fail.argtypes = [ctypes.c_int]
    fail(1)
    try:
        before = fg.lib().flens_gb300_launch_count()
        fg.dgemm_dev("N", "N", 1.0, A, B, 0.0, C[2])
        assert fg.lib().flens_gb300_launch_count() - before == 1
    finally:
        fail(0)
    fg.sync()
    c = [x.cpu().numpy() for x in C]
    assert np.array_equal(c[1], c[2])
    assert np.abs(c[0] - c[1]).max() <= 500 * U * 500


def test_threads_on_one_stream(cuda):
    """Calls of several threads on one stream have their own scratch."""
    import threading

    import torch
    r = np.random.default_rng(10)
    ops = [(r.integers(-99, 100, (400, 300)).astype(float), r.integers(-99, 100, (300, 500)).astype(float))
           for _ in range(8)]
    dev = [(_dev(cuda, a), _dev(cuda, b), _dev(cuda, np.zeros((400, 500)))) for a, b in ops]
    s = torch.cuda.Stream()
    torch.cuda.synchronize()

    def work(i):
        with torch.cuda.stream(s):
            for _ in range(10):
                fg.dgemm_dev("N", "N", 1.0, dev[i][0], dev[i][1], 0.0, dev[i][2])

    ts = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    s.synchronize()
    for (a, b), (_, _, c) in zip(ops, dev):
        assert np.array_equal(c.cpu().numpy(), a @ b)


def test_scratch_given_back(cuda):
    """After a synchronisation the pool keeps the scratch of a product (512 MB and more
    at 3000^3); trimmed, that is free again, and the next call takes it anew."""
    import torch
    r = np.random.default_rng(12)
    A, B = (_dev(cuda, r.integers(-9, 10, (3000, 3000)).astype(float)) for _ in range(2))
    C = [_dev(cuda, np.zeros((3000, 3000))) for _ in range(2)]
    fg.dgemm_dev("N", "N", 1.0, A, B, 0.0, C[0])
    fg.sync()
    kept = torch.cuda.mem_get_info()[0]
    fg.scratch_trim()
    assert torch.cuda.mem_get_info()[0] - kept >= 500 << 20
    fg.dgemm_dev("N", "N", 1.0, A, B, 0.0, C[1])
    fg.scratch_trim()                                 # the running call keeps its own
    fg.sync()
    assert torch.equal(C[0], C[1])
