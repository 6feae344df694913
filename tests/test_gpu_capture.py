"""Solves and factorisations recorded in a CUDA graph and replayed on other inputs:
under capture every product takes the FP64 kernel, solves keep their order (by halves
where the products are deep), the LU its right-looking steps.  Bounds: 4 n 2^-53
|T||X| for a triangle, 8 n 2^-53 |L||U| for the LU, and both with it for a solve."""
from __future__ import annotations

import pytest

import flens_gb300 as fg

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _uniform(g, m, n):
    import torch
    return torch.rand((n, m), generator=g, dtype=torch.float64, device="cuda").mul_(2).sub_(1).t()


def _replayed(call, inputs, buffers):
    """call() recorded once on `buffers`, then replayed for each set of inputs."""
    import torch
    for b, x in zip(buffers, inputs[0]):
        b.copy_(x)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        call()                                        # workspaces
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        call()
    for xs in inputs:
        for b, x in zip(buffers, xs):
            b.copy_(x)
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        yield xs


@pytest.mark.parametrize("n,nrhs", [(130, 3), (300, 100), (600, 300), (1100, 2700)])
@pytest.mark.parametrize("side,uplo,trans,diag", [("L", "L", "N", "N"), ("L", "U", "T", "N"), ("R", "U", "N", "U")])
def test_trsm(cuda, n, nrhs, side, uplo, trans, diag):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    B = fg.colmajor_empty(*((n, nrhs) if side == "L" else (nrhs, n)))
    A = fg.colmajor_empty(n, n)
    ins = [(_uniform(g, n, n) / n + 2 * torch.eye(n, dtype=torch.float64, device="cuda"), _uniform(g, *B.shape))
           for _ in range(2)]
    for A0, B0 in _replayed(lambda: fg.dtrsm_dev(side, uplo, trans, diag, 1.0, A, B), ins, (A, B)):
        T = torch.tril(A0) if uplo == "L" else torch.triu(A0)
        if diag == "U":
            T = T - torch.diag(torch.diagonal(T)) + torch.eye(n, dtype=torch.float64, device="cuda")
        T = T.t() if trans == "T" else T
        R, Q = ((T @ B, T.abs() @ B.abs()) if side == "L" else (B @ T, B.abs() @ T.abs()))
        assert bool(((R - B0).abs() <= 4 * n * U * (Q + B0.abs())).all())


@pytest.mark.parametrize("n,nrhs", [(200, 1), (700, 40), (1100, 300)])
def test_lu_and_solve(cuda, n, nrhs):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    A, B = fg.colmajor_empty(n, n), fg.colmajor_empty(n, nrhs)
    piv = torch.zeros(n, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")

    def call():
        fg.dgetrf_dev(A, piv, info)
        fg.dgetrs_dev("N", A, piv, B)

    ins = [(_uniform(g, n, n), _uniform(g, n, nrhs)) for _ in range(2)]
    for A0, B0 in _replayed(call, ins, (A, B)):
        assert int(info.item()) == 0
        perm = list(range(n))
        for i, p in enumerate(piv.tolist()):
            perm[i], perm[p - 1] = perm[p - 1], perm[i]
        L = torch.tril(A, -1) + torch.eye(n, dtype=torch.float64, device="cuda")
        R = torch.triu(A)
        LU = L.abs() @ R.abs()
        assert bool(((L @ R - A0[perm]).abs() <= 8 * n * U * LU).all())
        assert bool(((A0 @ B - B0)[perm].abs() <= 16 * n * U * (LU @ B.abs() + B0[perm].abs())).all())
