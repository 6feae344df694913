"""The work that users of this library have it do, as cases that can be timed.

listed() names the cases, draw() gives more of the same ranges, prepare() makes
what a program holds before the call (matrices on the GPU, host arrays for the
Fortran-ABI calls, kept factors or a batch plan), run() is one pass through the
public entry points, work() the bytes and operations that pass cannot do
without, and exact() the same outputs from plain torch or numpy in 64 bits.
"""
import ctypes
import math

import numpy as np
import torch

import flens_gb300 as fg

# precisions of the tensor-core entry points, as include/flens_gb300.h numbers them
TF32, BF16, FP8, F32X3, SPLIT, FP8X3 = 0, 1, 2, 3, 4, 6


def listed():
    return [
        # a block product inside a user's own loop: the call itself is the cost
        {"name": "gemm_small", "kind": "gemm", "ta": "N", "tb": "T", "m": 64, "n": 48, "k": 80,
         "alpha": 1.0, "beta": 1.0},
        # blas::mm on the plain FP64 GEMM configuration: 1024^3, alpha 1.5, beta 0.5
        {"name": "gemm_1024", "kind": "gemm", "ta": "N", "tb": "N", "m": 1024, "n": 1024, "k": 1024,
         "alpha": 1.5, "beta": 0.5},
        # a tall ragged product with a transposed operand (normal equations, projections)
        {"name": "gemm_ragged_tn", "kind": "gemm", "ta": "T", "tb": "N", "m": 3001, "n": 1111, "k": 2047,
         "alpha": -1.0, "beta": 1.0},
        # the LU + solve configuration: n = 8192, uniform[-1,1) + n/4 I, one right-hand side
        {"name": "lu_solve_8192", "kind": "lu", "n": 8192, "nrhs": 1, "shift": True},
        # an ordinary dense system with row interchanges in every column and several right-hand sides
        {"name": "gesv_1000", "kind": "lu", "n": 1000, "nrhs": 16, "shift": False},
        # a Fortran / FLENS program relinked: dgesv_ on pageable host arrays
        {"name": "gesv_host_500", "kind": "gesv_host", "n": 500, "nrhs": 4},
        # time stepping with a kept factorisation: one right-hand side per call
        {"name": "solve_4096", "kind": "solve", "n": 4096, "nrhs": 1, "trans": "N"},
        # a symmetric positive definite system: Cholesky and one right-hand side
        {"name": "posv_4000", "kind": "posv", "n": 4000, "nrhs": 1, "uplo": "L"},
        # the split-precision GEMM configuration: 8192^3, entries u * 2^e, e in [-16, 16]
        {"name": "split_gemm_8192", "kind": "split", "m": 8192, "n": 8192, "k": 8192, "e": 16},
        # the mixed-precision configuration: n = 16384, kappa = 1e2, FP32-accurate factors
        {"name": "mixed_16384", "kind": "mixed", "n": 16384, "nrhs": 1, "precision": F32X3},
        # FP32 matrices multiplied on the tensor cores in bfloat16, sizes off the tile edges
        {"name": "sgemm_bf16", "kind": "sgemm_tc", "m": 4100, "n": 4000, "k": 3000, "precision": BF16},
        # many uneven systems in one launch: n log-uniform in [8, 512], 1, 4 or 16 right-hand sides
        {"name": "batched_3000", "kind": "batched", "count": 3000, "n_max": 512, "sizes": 55,
         "precision": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "lu", "lu", "gesv_host", "solve", "posv", "split", "mixed",
                       "sgemm_tc", "batched"])
    if kind == "gemm":
        return {"kind": kind, "ta": rng.choice("NT"), "tb": rng.choice("NT"), "m": _log_int(rng, 32, 4200),
                "n": _log_int(rng, 32, 4200), "k": _log_int(rng, 32, 4200),
                "alpha": rng.choice([1.0, -1.0, 1.5]), "beta": rng.choice([0.0, 0.5, 1.0])}
    if kind == "lu":
        return {"kind": kind, "n": _log_int(rng, 100, 6500), "nrhs": rng.choice([1, 4, 16, 64]),
                "shift": rng.random() < 0.5}
    if kind == "gesv_host":
        return {"kind": kind, "n": _log_int(rng, 10, 2000), "nrhs": rng.choice([1, 4, 16])}
    if kind == "solve":
        return {"kind": kind, "n": _log_int(rng, 500, 6500), "nrhs": rng.choice([1, 2, 16, 100]),
                "trans": rng.choice("NT")}
    if kind == "posv":
        return {"kind": kind, "n": _log_int(rng, 200, 6500), "nrhs": rng.choice([1, 8]),
                "uplo": rng.choice("LU")}
    if kind == "split":
        return {"kind": kind, "m": _log_int(rng, 300, 6000), "n": _log_int(rng, 300, 6000),
                "k": _log_int(rng, 300, 6000), "e": rng.choice([0, 16, 48])}
    if kind == "mixed":
        return {"kind": kind, "n": _log_int(rng, 800, 8192), "nrhs": rng.choice([1, 64]),
                "precision": rng.choice([F32X3, TF32, FP8X3, SPLIT])}
    if kind == "sgemm_tc":
        return {"kind": kind, "m": _log_int(rng, 200, 8192), "n": _log_int(rng, 200, 8192),
                "k": _log_int(rng, 100, 8192), "precision": rng.choice([TF32, BF16, FP8, F32X3, FP8X3])}
    return {"kind": "batched", "count": _log_int(rng, 200, 6000), "n_max": rng.randrange(60, 513),
            "sizes": rng.randrange(1 << 20), "precision": rng.choice([0, 2])}


def _gen(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return g


def _uniform(g, m, n, dtype=torch.float64):
    """Column-major m x n, entries uniform[-1, 1)."""
    return torch.rand((n, m), generator=g, dtype=dtype, device="cuda").mul_(2).sub_(1).t()


def _hartley(X, dim):
    """The orthogonal real transform cas(2 pi i j / n) / sqrt(n) along dim."""
    F = torch.fft.fft(X, dim=dim, norm="ortho")
    return F.real - F.imag


def _kappa_matrix(g, n, kappa):
    """U diag(s) V^T, column-major: s geometric from 1 to 1/kappa, U and V random dense
    orthogonal matrices (Hartley transforms between random signs and permutations)."""
    s = kappa ** (-torch.arange(n, dtype=torch.float64, device="cuda") / (n - 1))
    sign = [torch.randint(0, 2, (n,), generator=g, device="cuda").double().mul_(2).sub_(1) for _ in range(3)]
    perm = torch.randperm(n, generator=g, device="cuda")
    M = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    M[torch.arange(n, device="cuda"), perm] = s * sign[0]
    M = _hartley(_hartley(M, 0).mul_(sign[1][:, None]), 1).mul_(sign[2][None, :])
    return fg.to_colmajor(M)


def _batch_shape(case):
    r = np.random.default_rng(case["sizes"])
    n = np.floor(np.exp(r.uniform(np.log(8), np.log(case["n_max"] + 0.999), size=case["count"]))).astype(np.int32)
    k = r.choice(np.array([1, 4, 16], dtype=np.int32), size=case["count"])
    a = np.concatenate([[0], np.cumsum(n.astype(np.int64) ** 2)])
    b = np.concatenate([[0], np.cumsum(n.astype(np.int64) * k)])
    return n, k, a, b


def _batch_inputs(case, seed):
    n, k, a, b = _batch_shape(case)
    g = _gen(seed)
    F = torch.rand(int(a[-1]), generator=g, dtype=torch.float64, device="cuda").mul_(2).sub_(1)
    diag = np.concatenate([a[i] + np.arange(n[i]) * (n[i] + 1) for i in range(len(n))])
    shift = np.repeat(n / 4.0, n)
    F[torch.from_numpy(diag).cuda()] += torch.from_numpy(shift).cuda()
    G = torch.rand(int(b[-1]), generator=g, dtype=torch.float64, device="cuda").mul_(2).sub_(1)
    return n, k, a, b, F, G


class _Batch:
    """A batch plan and the buffers it works on; the plan is released with it."""

    def __init__(self, case, seed):
        n, k, a, b, self.F0, self.G0 = _batch_inputs(case, seed)
        self.F, self.G = self.F0.clone(), self.G0.clone()
        self.piv = torch.zeros(int(n.sum()), dtype=torch.int32, device="cuda")
        p = np.concatenate([[0], np.cumsum(n.astype(np.int64))])
        self.info = torch.zeros(case["count"], dtype=torch.int32, device="cuda")
        self.iters = torch.zeros(case["count"], dtype=torch.int32, device="cuda")
        self.berr = torch.zeros(case["count"], dtype=torch.float64, device="cuda")
        pa = (self.F.data_ptr() + 8 * a[:-1]).astype(np.uint64)
        pb = (self.G.data_ptr() + 8 * b[:-1]).astype(np.uint64)
        pp = (self.piv.data_ptr() + 4 * p[:-1]).astype(np.uint64)
        L, v = fg.lib(), ctypes.c_void_p
        f = L.flens_gb300_dgesv_batched_plan
        f.argtypes = [ctypes.c_int, v, v, v, v, v, v, v, v, ctypes.c_int, v, v, ctypes.c_int, v,
                      ctypes.POINTER(v)]
        L.flens_gb300_batched_execute.argtypes = [v, v]
        L.flens_gb300_batched_destroy.argtypes = [v]
        self.plan = v()
        st = f(case["count"], n.ctypes.data, k.ctypes.data, pa.ctypes.data, n.ctypes.data, pp.ctypes.data,
               pb.ctypes.data, n.ctypes.data, self.info.data_ptr(), case["precision"], self.iters.data_ptr(),
               self.berr.data_ptr(), 10, _stream(), ctypes.byref(self.plan))
        if st != 0:
            raise RuntimeError(fg.last_error())

    def __del__(self):
        if getattr(self, "plan", None):
            torch.cuda.synchronize()
            fg.lib().flens_gb300_batched_destroy(self.plan)


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _shape(t, r, c):
    return (r, c) if t == "N" else (c, r)


def _lu_inputs(case, seed):
    g, n = _gen(seed), case["n"]
    A = _uniform(g, n, n)
    if case.get("shift", True):
        A.diagonal().add_(n / 4.0)
    return A, _uniform(g, n, case["nrhs"])


def _spd_inputs(case, seed):
    g, n = _gen(seed), case["n"]
    G = _uniform(g, n, n)
    A = torch.mm(G, G.t()).div_(n)
    A.diagonal().add_(1.0)
    return fg.to_colmajor(A), _uniform(g, n, case["nrhs"])


def _wide(g, m, n, e):
    X = _uniform(g, m, n)
    if e:
        X = X * torch.exp2(torch.randint(-e, e + 1, (n, m), generator=g, device="cuda").double()).t()
    return X


def prepare(case, seed):
    kind = case["kind"]
    if kind == "gemm":
        g = _gen(seed)
        return {"case": case, "A": _uniform(g, *_shape(case["ta"], case["m"], case["k"])),
                "B": _uniform(g, *_shape(case["tb"], case["k"], case["n"])),
                "C0": _uniform(g, case["m"], case["n"]), "C": fg.colmajor_empty(case["m"], case["n"])}
    if kind in ("lu", "solve", "posv"):
        A0, B0 = _spd_inputs(case, seed) if kind == "posv" else _lu_inputs(case, seed)
        s = {"case": case, "A0": A0, "B0": B0, "A": fg.to_colmajor(A0.clone()), "B": fg.to_colmajor(B0.clone()),
             "piv": torch.zeros(case["n"], dtype=torch.int32, device="cuda"),
             "info": torch.zeros(1, dtype=torch.int32, device="cuda")}
        if kind == "solve":
            fg.dgetrf_dev(s["A"], s["piv"], s["info"])
            del s["A0"]
        return s
    if kind == "gesv_host":
        r = np.random.default_rng(seed)
        n = case["n"]
        return {"case": case, "A0": np.asfortranarray(r.uniform(-1, 1, (n, n))),
                "B0": np.asfortranarray(r.uniform(-1, 1, (n, case["nrhs"])))}
    if kind == "split":
        g = _gen(seed)
        return {"case": case, "A": _wide(g, case["m"], case["k"], case["e"]),
                "B": _wide(g, case["k"], case["n"], case["e"]),
                "C": torch.zeros((case["n"], case["m"]), dtype=torch.float64, device="cuda").t()}
    if kind == "mixed":
        g = _gen(seed)
        A = _kappa_matrix(g, case["n"], 1e2)
        B = fg.to_colmajor(A @ _uniform(g, case["n"], case["nrhs"]))
        return {"case": case, "A": A, "B": B, "X": fg.colmajor_empty(case["n"], case["nrhs"])}
    if kind == "sgemm_tc":
        g = _gen(seed)
        return {"case": case, "A": _uniform(g, case["m"], case["k"], torch.float32),
                "B": _uniform(g, case["k"], case["n"], torch.float32),
                "C": torch.zeros((case["n"], case["m"]), dtype=torch.float32, device="cuda").t()}
    return {"case": case, "batch": _Batch(case, seed)}


def _check(st):
    if st != 0:
        raise RuntimeError("status %d: %s" % (st, fg.last_error()))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "gemm":
        state["C"].copy_(state["C0"])
        return fg.dgemm_dev(case["ta"], case["tb"], case["alpha"], state["A"], state["B"], case["beta"], state["C"])
    if kind == "lu":
        A, B, piv, info = (state[k] for k in ("A", "B", "piv", "info"))
        A.copy_(state["A0"])
        B.copy_(state["B0"])
        fg.dgetrf_dev(A, piv, info)
        fg.dgetrs_dev("N", A, piv, B)
        return {"lu": A, "x": B, "piv": piv, "info": info}
    if kind == "gesv_host":
        A, B = state["A0"].copy(order="F"), state["B0"].copy(order="F")
        piv, info = fg.dgesv(A, B)
        return {"lu": A, "x": B, "piv": piv, "info": info}
    if kind == "solve":
        state["B"].copy_(state["B0"])
        return fg.dgetrs_dev(case["trans"], state["A"], state["piv"], state["B"])
    if kind == "posv":
        A, B, info = (state[k] for k in ("A", "B", "info"))
        A.copy_(state["A0"])
        B.copy_(state["B0"])
        fg.dposv_dev(case["uplo"], A, B, info)
        return {"factor": A, "x": B, "info": info}
    if kind == "split":
        fg.dgemm_split_dev("N", "N", 1.0, state["A"], state["B"], 0.0, state["C"])
        return state["C"]
    if kind == "mixed":
        A, B, X = (state[k] for k in ("A", "B", "X"))
        f = fg.lib().flens_gb300_dgesv_mixed
        i, v, d = ctypes.c_int, ctypes.c_void_p, ctypes.c_double
        f.argtypes = [i, i, v, i, v, i, v, i, i, i, i, d, ctypes.POINTER(i), ctypes.POINTER(d),
                      ctypes.POINTER(i), v]
        iters, berr, info = i(), d(), i()
        n = case["n"]
        _check(f(n, case["nrhs"], A.data_ptr(), n, B.data_ptr(), n, X.data_ptr(), n, case["precision"], 2, 30, 0.0,
                 ctypes.byref(iters), ctypes.byref(berr), ctypes.byref(info), _stream()))
        return {"x": X, "info": info.value}
    if kind == "sgemm_tc":
        A, B, C = (state[k] for k in ("A", "B", "C"))
        f = fg.lib().flens_gb300_sgemm_tc
        i, v, c, x = ctypes.c_int, ctypes.c_void_p, ctypes.c_char, ctypes.c_float
        f.argtypes = [i, c, c, i, i, i, x, v, i, v, i, x, v, i, v]
        m, n, k = case["m"], case["n"], case["k"]
        _check(f(case["precision"], b"N", b"N", m, n, k, 1.0, A.data_ptr(), m, B.data_ptr(), k, 0.0,
                 C.data_ptr(), m, _stream()))
        return C
    b = state["batch"]
    b.F.copy_(b.F0)
    b.G.copy_(b.G0)
    _check(fg.lib().flens_gb300_batched_execute(b.plan, _stream()))
    return {"lu": b.F, "x": b.G, "piv": b.piv, "info": b.info}


def work(case):
    kind = case["kind"]
    if kind in ("gemm", "split", "sgemm_tc"):
        m, n, k = case["m"], case["n"], case["k"]
        size = 4 if kind == "sgemm_tc" else 8
        return {"bytes": size * (m * k + k * n + 2.0 * m * n), "flops": 2.0 * m * n * k}
    if kind == "batched":
        n, k, a, b = _batch_shape(case)
        n = n.astype(np.float64)
        return {"bytes": 16.0 * float(a[-1] + b[-1]), "flops": float(np.sum(2 / 3 * n ** 3 + 2 * n ** 2 * k))}
    n, r = float(case["n"]), case["nrhs"]
    if kind == "solve":
        return {"bytes": 8.0 * (n * n + 2 * n * r), "flops": 2 * n * n * r}
    if kind == "posv":
        return {"bytes": 8.0 * (n * n + 2 * n * r), "flops": n ** 3 / 3 + 2 * n * n * r}
    reads = 1 if kind == "mixed" else 2          # the mixed solve leaves A as it is
    return {"bytes": 8.0 * (reads * n * n + 2 * n * r), "flops": 2 / 3 * n ** 3 + 2 * n * n * r}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("gemm", "split", "sgemm_tc", "mixed"):
        s = prepare(case, seed)
        if kind == "gemm":
            op = lambda X, t: X if t == "N" else X.t()  # noqa: E731
            return case["beta"] * s["C0"] + case["alpha"] * (op(s["A"], case["ta"]) @ op(s["B"], case["tb"]))
        if kind == "mixed":
            return {"x": torch.linalg.solve(s["A"], s["B"]), "info": None}
        return s["A"].double() @ s["B"].double()
    if kind == "gesv_host":
        s = prepare(case, seed)
        A, B = torch.from_numpy(s["A0"]), torch.from_numpy(s["B0"])
        lu, piv = torch.linalg.lu_factor(A)
        return {"lu": lu, "x": torch.linalg.lu_solve(lu, piv, B), "piv": piv, "info": 0}
    if kind == "posv":
        A, B = _spd_inputs(case, seed)
        L = torch.linalg.cholesky(A)
        keep = A.triu(1) + L if case["uplo"] == "L" else A.tril(-1) + L.t()
        return {"factor": keep, "x": torch.cholesky_solve(B, L), "info": torch.zeros(1, dtype=torch.int32)}
    if kind in ("lu", "solve"):
        A, B = _lu_inputs(case, seed)
        lu, piv = torch.linalg.lu_factor(A)
        if kind == "solve":
            return torch.linalg.lu_solve(lu, piv, B, adjoint=case["trans"] == "T")
        return {"lu": lu, "x": torch.linalg.lu_solve(lu, piv, B), "piv": piv,
                "info": torch.zeros(1, dtype=torch.int32)}
    if case["precision"] != 0:
        return None
    n, k, a, b, F, G = _batch_inputs(case, seed)
    X = torch.empty_like(G)
    for i in range(len(n)):
        A = F[a[i]:a[i + 1]].view(n[i], n[i]).t()
        X[b[i]:b[i + 1]] = torch.linalg.solve(A, G[b[i]:b[i + 1]].view(k[i], n[i]).t()).t().reshape(-1)
    return {"lu": None, "x": X, "piv": None, "info": None}
