"""trmm and the inverses built on it, whose products go to the tensor cores whole:
accuracy against FP64, and the same finite results around infinities as the
FP64 route with its k ranges (a child process with FLENS_GB300_DGEMM=fma)."""
from __future__ import annotations

import os
import subprocess
import sys

import numpy as np
import pytest

import flens_gb300 as fg
import oracle

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
CASES = [(s, u, t, d) for s in "LR" for u in "LU" for t in "NT" for d in "NU"]


def _inputs(i, side, special):
    ka, other = 513, 600
    A = np.asfortranarray(oracle.uniform(50 + i, ka, ka))
    B = np.asfortranarray(oracle.uniform(90 + i, *((ka, other) if side == "L" else (other, ka))))
    if special:
        B[100, 200], B[300, 5], A[7, 7] = np.inf, np.nan, 1e300
    return A, B


def run_special():
    out = {}
    for i, (s, u, t, d) in enumerate(CASES):
        A, B = _inputs(i, s, True)
        fg.dtrmm(s, u, t, d, 1.5, A, B)
        out[s + u + t + d] = np.isfinite(B)
    return out


@pytest.mark.parametrize("i", range(len(CASES)))
def test_trmm(cuda, i):
    s, u, t, d = CASES[i]
    A, B = _inputs(i, s, False)
    T = np.tril(A) if u == "L" else np.triu(A)
    if d == "U":
        np.fill_diagonal(T, 1.0)
    T = T if t == "N" else T.T
    before = fg.lib().flens_gb300_launch_count()
    X = B.copy(order="F")
    fg.dtrmm(s, u, t, d, -0.75, A, X)
    assert fg.lib().flens_gb300_launch_count() - before >= 6
    want = -0.75 * (T @ B if s == "L" else B @ T)
    mag = np.abs(T) @ np.abs(B) if s == "L" else np.abs(B) @ np.abs(T)
    # operand rounding 4 u, one rounding of the sum and two of alpha; numpy's own sum
    assert np.all(np.abs(X - want) <= (8 + 513) * U * mag)


def test_infinities_reach_what_they_reached(cuda, tmp_path):
    path = str(tmp_path / "fma.npz")
    here = os.path.dirname(os.path.abspath(__file__))
    code = ("import sys, numpy as np; sys.path[:0] = [%r, %r]\nimport test_gpu_trmm_route as t\n"
            "np.savez(%r, **t.run_special())" % (os.path.dirname(here), here, path))
    subprocess.run([sys.executable, "-c", code], env=dict(os.environ, FLENS_GB300_DGEMM="fma"), check=True, timeout=300)
    want, got = np.load(path), run_special()
    for k in got:
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("side", "LR")
@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("trans", "NT")
def test_triangle_in_parts_is_exact(cuda, side, uplo, trans):
    """4200 rows: two parts of the triangle, whose blocks are zero, triangles or full.
    Integers, so the result is the product itself; what lies in the other triangle is
    never part of it."""
    ka, other = 4200, 300
    r = np.random.default_rng(ka)
    A = np.asfortranarray(r.integers(-999, 1000, (ka, ka)).astype(np.float64))
    B = np.asfortranarray(r.integers(-999, 1000, (ka, other) if side == "L" else (other, ka)).astype(np.float64))
    T = np.tril(A) if uplo == "L" else np.triu(A)
    T = T if trans == "N" else T.T
    want = T @ B if side == "L" else B @ T
    A[~(np.tril(np.ones((ka, ka), dtype=bool)) if uplo == "L" else np.triu(np.ones((ka, ka), dtype=bool)))] = np.nan
    before = fg.lib().flens_gb300_launch_count()
    fg.dtrmm(side, uplo, trans, "N", 1.0, A, B)
    assert fg.lib().flens_gb300_launch_count() - before >= 10
    assert np.array_equal(B, want)
