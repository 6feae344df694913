"""The orders that hand large products to the tensor cores: the recursive LU
and the halved triangular solve, over their shapes and variants, by residuals
in FP64 (bound: the backward error c * n * 2^-53 * |factors| of a blocked
algorithm, c = 4 for the factors or the solve and the residual's own rounding)."""
from __future__ import annotations

import numpy as np
import pytest

import flens_gb300 as fg
import oracle

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _dev(cuda, X):
    import torch
    return fg.to_colmajor(torch.from_numpy(X).to(cuda))


@pytest.mark.parametrize("m,n", [(2048, 2048), (2111, 2500), (2500, 2111), (2049, 2113)])
@pytest.mark.parametrize("shift", [0.0, 0.25])
def test_recursive_lu(cuda, m, n, shift):
    import torch
    A0 = oracle.uniform(m, m, n)
    k = min(m, n)
    A0[np.arange(k), np.arange(k)] += shift * n
    A, dA0 = _dev(cuda, A0), _dev(cuda, A0)
    piv = torch.zeros(k, dtype=torch.int32, device=cuda)
    info = torch.zeros(1, dtype=torch.int32, device=cuda)
    fg.dgetrf_dev(A, piv, info)
    fg.sync()
    assert int(info.item()) == 0
    p = piv.cpu().numpy() - 1
    perm = np.arange(m)
    for i in range(k):
        assert i <= p[i] < m
        perm[[i, p[i]]] = perm[[p[i], i]]
    L = torch.tril(A[:, :k], -1)
    assert float(L.abs().max()) <= 1.0
    L.diagonal().add_(1.0)
    Up = torch.triu(A[:k])
    R = (dA0[torch.from_numpy(perm).to(cuda)] - L @ Up).abs()
    assert bool((R <= 4 * k * U * (L.abs() @ Up.abs())).all())


def test_recursive_lu_singular_column(cuda):
    """INFO is the first exactly zero pivot; the factorisation goes on."""
    import torch
    n = 2100
    A0 = oracle.uniform(3, n, n)
    A0[:, 1500] = 0.0
    A = _dev(cuda, A0)
    piv = torch.zeros(n, dtype=torch.int32, device=cuda)
    info = torch.zeros(1, dtype=torch.int32, device=cuda)
    fg.dgetrf_dev(A, piv, info)
    fg.sync()
    assert int(info.item()) == 1501
    assert bool(torch.isfinite(A).all())


@pytest.mark.parametrize("side", "LR")
@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("trans", "NT")
@pytest.mark.parametrize("diag", "NU")
@pytest.mark.parametrize("ka", [513, 777])
def test_halved_trsm(cuda, side, uplo, trans, diag, ka):
    import torch
    nvec = 700
    A = oracle.uniform(ka, ka, ka) / ka
    A[np.arange(ka), np.arange(ka)] = 1.5
    B = oracle.uniform(1, *((ka, nvec) if side == "L" else (nvec, ka)))
    dA, X, dB = _dev(cuda, A), _dev(cuda, B), _dev(cuda, B)
    before = fg.lib().flens_gb300_launch_count()
    fg.dtrsm_dev(side, uplo, trans, diag, -0.5, dA, X)
    assert fg.lib().flens_gb300_launch_count() - before > 2 * ((ka + 63) // 64)
    fg.sync()
    T = torch.tril(dA) if uplo == "L" else torch.triu(dA)
    if diag == "U":
        T.diagonal().fill_(1.0)
    T = T if trans == "N" else T.t()
    R, M = ((T @ X, T.abs() @ X.abs()) if side == "L" else (X @ T, X.abs() @ T.abs()))
    assert bool(((R + 0.5 * dB).abs() <= 4 * ka * U * M).all())


@pytest.mark.parametrize("m,n", [(1024, 1024), (1100, 3000), (3000, 1100), (4600, 4600), (6600, 6700), (8300, 1100),
                                 (12600, 1024), (13000, 1200), (21000, 1100)])
def test_lookahead_lu(cuda, m, n):
    """Outer blocks of 64, 128 and 256 columns, wide and tall, 32-column and grid
    panels: factors that multiply back, twice the same bits (nothing depends on how
    the two streams interleave)."""
    import torch
    k = min(m, n)
    g = torch.Generator(device="cuda").manual_seed(m)
    A0 = (torch.rand((n, m), generator=g, dtype=torch.float64, device=cuda) * 2 - 1).t()
    runs = []
    for _ in range(2):
        A = fg.to_colmajor(A0.clone())
        piv = torch.zeros(k, dtype=torch.int32, device=cuda)
        info = torch.zeros(1, dtype=torch.int32, device=cuda)
        fg.dgetrf_dev(A, piv, info)
        runs.append((A, piv))
    fg.sync()
    (A, piv), (A2, piv2) = runs
    assert int(info.item()) == 0
    assert torch.equal(A, A2) and torch.equal(piv, piv2)
    p = piv.cpu().numpy() - 1
    perm = np.arange(m)
    for i in range(k):
        assert i <= p[i] < m
        perm[[i, p[i]]] = perm[[p[i], i]]
    L = torch.tril(A[:, :k], -1)
    assert float(L.abs().max()) <= 1.0
    L.diagonal().add_(1.0)
    Up = torch.triu(A[:k])
    R = (A0[torch.from_numpy(perm).to(cuda)] - L @ Up).abs()
    assert bool((R <= 4 * k * U * (L.abs() @ Up.abs())).all())


def test_lookahead_on_two_streams_at_once(cuda):
    """Two factorisations on two streams share no scratch or side stream."""
    import torch
    n = 1500
    A0 = [_dev(cuda, oracle.uniform(s, n, n)) for s in (1, 2)]
    want = []
    for a in A0:
        A, piv = fg.to_colmajor(a.clone()), torch.zeros(n, dtype=torch.int32, device=cuda)
        fg.dgetrf_dev(A, piv, torch.zeros(1, dtype=torch.int32, device=cuda))
        want.append((A, piv))
    fg.sync()
    streams = [torch.cuda.Stream() for _ in A0]
    got = [(fg.to_colmajor(a.clone()), torch.zeros(n, dtype=torch.int32, device=cuda),
            torch.zeros(1, dtype=torch.int32, device=cuda)) for a in A0]
    torch.cuda.synchronize()
    for _ in range(1):
        for s, (A, piv, info) in zip(streams, got):
            with torch.cuda.stream(s):
                fg.dgetrf_dev(A, piv, info)
    torch.cuda.synchronize()
    for (A, piv), (B, p2, _) in zip(want, got):
        assert torch.equal(A, B) and torch.equal(piv, p2)


@pytest.mark.parametrize("m,n", [(2048, 2048), (2500, 2100), (13300, 2100), (14000, 2048), (16384, 2048), (16500, 2100)])
@pytest.mark.parametrize("precision", [1, 3, 6])
def test_lookahead_lu_fp32(cuda, m, n, precision):
    """The FP32 LU: 64- and 32-column cluster panels and the grid panel beyond them;
    the same bits twice, and (3xTF32) factors that multiply back."""
    import ctypes

    import torch
    f = fg.lib().flens_gb300_sgetrf_tc
    v, i = ctypes.c_void_p, ctypes.c_int
    f.argtypes = [i, i, i, v, i, v, v, v]
    g = torch.Generator(device="cuda").manual_seed(m)
    A0 = (torch.rand((n, m), generator=g, device=cuda) * 2 - 1).t()
    runs = []
    for _ in range(2):
        A = fg.to_colmajor(A0.clone())
        piv = torch.zeros(n, dtype=torch.int32, device=cuda)
        info = torch.zeros(1, dtype=torch.int32, device=cuda)
        st = f(precision, m, n, A.data_ptr(), m, piv.data_ptr(), info.data_ptr(),
               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == 0, fg.last_error()
        runs.append((A, piv))
    torch.cuda.synchronize()
    (A, piv), (A2, piv2) = runs
    assert int(info.item()) == 0
    assert torch.equal(A, A2) and torch.equal(piv, piv2)
    if precision != 3:
        return
    p = piv.cpu().numpy() - 1
    perm = np.arange(m)
    for c in range(n):
        perm[[c, p[c]]] = perm[[p[c], c]]
    X = A.double()
    L = torch.tril(X, -1)
    L.diagonal().add_(1.0)
    Up = torch.triu(X[:n])
    R = (A0.double()[torch.from_numpy(perm).to(cuda)] - L @ Up).abs()
    assert bool((R <= 4 * n * 2.0 ** -24 * (L.abs() @ Up.abs())).all())
