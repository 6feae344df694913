"""LU with look-ahead where few CTAs (FLENS_GB300_PANEL_CTAS) make the grid panels of
the first rows narrower than 32 columns: as many panels per outer block as its
lists of row moves hold (8 columns wide, 256-column blocks), and more (no
look-ahead then).  Each case in a child process: the settings are read once.
Bound: 4 n u |L||U| with u of the storage."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


def run_one(storage, m, n):
    import ctypes

    import numpy as np
    import torch

    import flens_gb300 as fg
    import oracle
    T, u = (torch.float64, 2.0 ** -53) if storage == "d" else (torch.float32, 2.0 ** -24)
    A0 = fg.to_colmajor(torch.from_numpy(oracle.uniform(m + n, m, n)).cuda().to(T))
    A = fg.to_colmajor(A0.clone())
    piv = torch.zeros(n, dtype=torch.int32, device="cuda")
    info = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    if storage == "d":
        fg.dgetrf_dev(A, piv, info)
    else:
        f = fg.lib().flens_gb300_sgetrf_tc
        v, i = ctypes.c_void_p, ctypes.c_int
        f.argtypes = [i, i, i, v, i, v, v, v]
        assert f(3, m, n, A.data_ptr(), m, piv.data_ptr(), info.data_ptr(), fg._stream(None)) == 0
    fg.sync()
    assert int(info.item()) == 0
    perm = np.arange(m)
    for r, p in enumerate(piv.cpu().numpy() - 1):
        perm[[r, p]] = perm[[p, r]]
    A = A.double()
    L = torch.tril(A, -1) + torch.eye(m, n, dtype=torch.float64, device="cuda")
    R = torch.triu(A[:n])
    PA = A0.double()[torch.from_numpy(perm).cuda()]
    assert bool(((L @ R - PA).abs() <= 4 * n * u * (L.abs() @ R.abs())).all())


@pytest.mark.parametrize("storage,ctas,block,m", [("d", 6, 256, 16000), ("d", 5, 256, 16000), ("d", 4, 256, 16000),
                                                  ("d", 4, 1024, 16000), ("d", 152, 1024, 9000), ("s", 2, 256, 17000)])
def test_more_panels_than_lists(storage, ctas, block, m):
    env = dict(os.environ, FLENS_GB300_PANEL_CTAS=str(ctas), FLENS_GB300_LOOKAHEAD_NB=str(block))
    code = "import test_gpu_panel_narrow as t; t.run_one(%r, %d, 2100)" % (storage, m)
    here = os.path.dirname(os.path.abspath(__file__))
    env["PYTHONPATH"] = os.pathsep.join([here, os.path.dirname(here), env.get("PYTHONPATH", "")])
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
