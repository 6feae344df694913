"""The one-cluster LU panel against the grid panel: the same operations per
element in the same order, so factors, pivots and INFO are equal bit for bit.
The grid panel runs in a child process (FLENS_GB300_PANEL_CLUSTER=0)."""
from __future__ import annotations

import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import flens_gb300 as fg
import oracle

pytestmark = pytest.mark.gpu

# one row block of a CTA and its edges, warps of rows, more than 512 rows per
# CTA (FP32), the largest FP64 cluster panel and the first grid panel
SHAPES = [(1, 1), (15, 15), (16, 20), (17, 3), (64, 64), (65, 64), (130, 63), (511, 64), (513, 64), (1040, 100),
          (2100, 64), (5990, 64), (6100, 70), (300, 300), (1111, 257)]
SHAPES32 = SHAPES + [(9000, 64), (13500, 64), (14000, 64)]


def _input(kind, m, n):
    A = oracle.uniform(m * 7 + n, m, n)
    if kind == "ties":
        A = np.sign(A) * np.where(np.abs(A) < 0.3, 0.0, 1.0)
    elif kind == "special":
        A[m // 2, 0] = np.nan
        A[:, n // 2] = 0.0
        A[m // 3, n - 1] = np.inf
    elif kind == "tiny":
        A *= 1e-310 if n < 64 else 1e-30
        A[0, 0] = np.nan if m > 20 else A[0, 0]
    return A


def _cases():
    for dt, shapes in (("d", SHAPES), ("s", SHAPES32)):
        for m, n in shapes:
            for kind in ("uniform", "ties", "special", "tiny"):
                if m > 2100 and kind in ("special", "tiny"):
                    continue
                yield dt, m, n, kind


def run_all():
    """{case: (factors, pivots, info)}, as raw bytes."""
    import torch
    f = fg.lib().flens_gb300_sgetrf_tc
    v, i = ctypes.c_void_p, ctypes.c_int
    f.argtypes = [i, i, i, v, i, v, v, v]
    out = {}
    for dt, m, n, kind in _cases():
        T = torch.float64 if dt == "d" else torch.float32
        A = fg.to_colmajor(torch.from_numpy(_input(kind, m, n)).cuda().to(T))
        piv = torch.zeros(min(m, n), dtype=torch.int32, device="cuda")
        info = torch.zeros(1, dtype=torch.int32, device="cuda")
        if dt == "d":
            fg.dgetrf_dev(A, piv, info)
        else:
            st = f(3, m, n, A.data_ptr(), m, piv.data_ptr(), info.data_ptr(),
                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert st == 0, fg.last_error()
        fg.sync()
        name = "%s_%d_%d_%s" % (dt, m, n, kind)
        X = A.cpu().numpy()
        out[name + "_f"] = np.where(np.isnan(X), np.float64(0.5), X).astype(X.dtype)
        out[name + "_nan"] = np.isnan(X)
        out[name + "_p"] = piv.cpu().numpy()
        out[name + "_i"] = info.cpu().numpy()
    return out


def test_cluster_panel_equals_grid_panel(cuda, tmp_path):
    path = str(tmp_path / "grid.npz")
    code = ("import sys, numpy as np; sys.path.insert(0, %r); sys.path.insert(0, %r)\n"
            "import test_gpu_panel_cluster as t; np.savez(%r, **t.run_all())"
            % (os.path.dirname(os.path.dirname(os.path.abspath(__file__))), os.path.dirname(os.path.abspath(__file__)),
               path))
    env = dict(os.environ, FLENS_GB300_PANEL_CLUSTER="0")
    subprocess.run([sys.executable, "-c", code], env=env, check=True, timeout=300)
    want = np.load(path)
    got = run_all()
    assert set(got) == set(want.files)
    for k in want.files:
        assert np.array_equal(got[k], want[k]), k
