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
