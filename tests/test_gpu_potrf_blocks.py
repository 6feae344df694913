"""Cholesky at the edges of its blocks (64-column steps, 256-column bases, the
halving above), the other triangle untouched, and INFO at every kind of
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
