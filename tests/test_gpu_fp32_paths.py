"""FP32 paths at their edges: the thread-per-vector block solve of the FP32 LU's
U12 (64-row blocks, ragged last block, both storage orders come from the LU's
shapes), and the tensor-core operands at sizes off every tile and line (bitwise
equal to products of operands rounded by torch, within the FP32 sum's bound)."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import flens_gb300 as fg
import oracle

pytestmark = pytest.mark.gpu


def _lib():
    L = fg.lib()
    i, v, c, x = ctypes.c_int, ctypes.c_void_p, ctypes.c_char, ctypes.c_float
    L.flens_gb300_sgetrf_tc.argtypes = [i, i, i, v, i, v, v, v]
    L.flens_gb300_sgemm_tc.argtypes = [i, c, c, i, i, i, x, v, i, v, i, x, v, i, v]
    return L


@pytest.mark.parametrize("m,n", [(300, 3000), (257, 2700), (65, 2625), (1000, 4000)])
def test_wide_fp32_lu(cuda, m, n):
    """Many columns to the right of each block: U12 by thread per vector."""
    import torch
    A0 = torch.from_numpy(oracle.uniform(m, m, n)).to(cuda).float()
    A0[torch.arange(m), torch.arange(m)] += m / 4.0
    A0 = fg.to_colmajor(A0)
    A = fg.to_colmajor(A0.clone())
    piv = torch.zeros(m, dtype=torch.int32, device=cuda)
    info = torch.zeros(1, dtype=torch.int32, device=cuda)
    st = _lib().flens_gb300_sgetrf_tc(3, m, n, A.data_ptr(), m, piv.data_ptr(), info.data_ptr(), None)
    assert st == 0, fg.last_error()
    fg.sync()
    torch.cuda.synchronize()
    p = piv.cpu().numpy() - 1
    perm = np.arange(m)
    for i in range(m):
        perm[[i, p[i]]] = perm[[p[i], i]]
    X = A.double()
    L = torch.tril(X[:, :m], -1)
    L.diagonal().add_(1.0)
    U = torch.triu(X)
    R = (A0.double()[torch.from_numpy(perm).to(cuda)] - L @ U).abs()
    assert bool((R <= 4 * m * 2.0 ** -24 * (L.abs() @ U.abs())).all())


@pytest.mark.parametrize("ta,tb", ["NN", "TN", "NT", "TT"])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (33, 257, 65), (130, 70, 3), (300, 513, 129), (129, 31, 1000)])
@pytest.mark.parametrize("precision", [0, 1, 2, 3, 5, 6])
def test_tc_operands(cuda, ta, tb, m, n, k, precision):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    A = torch.rand((k, m) if ta == "N" else (m, k), generator=g, device=cuda) * 2 - 1     # column-major op storage
    B = torch.rand((n, k) if tb == "N" else (k, n), generator=g, device=cuda) * 2 - 1
    C = torch.zeros((n, m), device=cuda)
    st = _lib().flens_gb300_sgemm_tc(precision, ta.encode(), tb.encode(), m, n, k, 1.0, A.data_ptr(), A.shape[1],
                                     B.data_ptr(), B.shape[1], 0.0, C.data_ptr(), m, None)
    assert st == 0, fg.last_error()
    torch.cuda.synchronize()
    opA = (A.t() if ta == "N" else A).double()
    opB = (B.t() if tb == "N" else B).double()
    mag = opA.abs() @ opB.abs()
    want = opA @ opB
    if precision == 1:
        want = (opA.bfloat16().double()) @ (opB.bfloat16().double())
    # relative error per product of each operand form (TF32 and e4m3 half steps, e4m3
    # with the row scale's own rounding; terms dropped), and the FP32 sum
    per = {0: 2.0 ** -10, 1: 0.0, 2: 2.0 ** -3, 3: 2.0 ** -20, 5: 2.0 ** -6, 6: 2.0 ** -9}[precision]
    big = opA.abs().amax(1, keepdim=True) * opB.abs().amax(0, keepdim=True) * k
    sub = {2: 2.0 ** -14, 5: 2.0 ** -14, 6: 2.0 ** -14}.get(precision, 0.0)      # e4m3's subnormal step
    bound = per * mag + sub * big + (k + 8) * 2.0 ** -23 * mag
    assert bool(((C.t().double() - want).abs() <= bound).all())
