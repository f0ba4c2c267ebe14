"""Timed cases of the dense solve path, each through the public calls of `lmb200` on device tensors.

A case is a dict of plain values; its "op" names the call:

  lu      luSolve(A, B): FP64 LU with partial pivoting and the substitutions (vector or n x nrhs)
  chol    choleskySolve(A, B): FP64 Cholesky and the substitutions
  gemm    gemm(alpha, A, B, beta, C), or matMul(A, B) when beta is 0
  ir      luSolveIR(A, B): FP32 factor, FP64 iterative refinement
  batch   Batch(...).solve(A, B, X): uneven systems in one persistent launch, FP64 or FP32 + refinement
  matvec  matvec(A, x): bitwise the reference's order of operations
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "linear-massiv_b200"))
import lmb200  # noqa: E402


def listed():
    return [
        # the reference's own benchmark orders (10 .. 500): latency and launches decide
        {"name": "lu_100", "op": "lu", "n": 100, "nrhs": 1},
        {"name": "lu_500", "op": "lu", "n": 500, "nrhs": 1},
        # an odd order: rows that do not start on 16 bytes, a ragged last panel, a few right-hand sides
        {"name": "lu_2999_r3", "op": "lu", "n": 2999, "nrhs": 3},
        # many right-hand sides, where the substitutions are contractions
        {"name": "lu_8192_r64", "op": "lu", "n": 8192, "nrhs": 64},
        # the largest plain solve of the benchmark
        {"name": "lu_16384", "op": "lu", "n": 16384, "nrhs": 1},
        # Cholesky solves: an odd medium order with several right-hand sides, and the benchmark's order
        {"name": "chol_701_r16", "op": "chol", "n": 701, "nrhs": 16},
        {"name": "chol_8192", "op": "chol", "n": 8192, "nrhs": 1},
        # a ragged product with alpha and beta (one odd row length)
        {"name": "gemm_1500x1001x2000", "op": "gemm", "m": 1500, "n": 1001, "k": 2000, "alpha": 1.25, "beta": -0.5},
        # mixed precision on a dense matrix of chosen condition
        {"name": "ir_8192", "op": "ir", "n": 8192, "nrhs": 1, "kappa": 1e4},
        # ten thousand uneven systems, half general and half SPD, in FP64; fewer of them in FP32 + refinement
        {"name": "batch_10000", "op": "batch", "count": 10000, "nmin": 8, "nmax": 256, "rmax": 16, "ir": False,
         "sizes": 1},
        {"name": "batch_ir_3000", "op": "batch", "count": 3000, "nmin": 8, "nmax": 256, "rmax": 16, "ir": True,
         "sizes": 2},
        # the reference's matvec at a size that memory bounds
        {"name": "matvec_8192", "op": "matvec", "m": 8192, "n": 8192},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["lu", "lu", "chol", "gemm", "ir", "batch", "matvec"])
    if op == "lu":
        return {"op": op, "n": size(32, 9000), "nrhs": rng.choice([1, 1, 1, 2, 4, 5, 16, 33, 64])}
    if op == "chol":
        return {"op": op, "n": size(32, 9000), "nrhs": rng.choice([1, 1, 2, 3, 8, 17, 64])}
    if op == "gemm":
        return {"op": op, "m": size(48, 6000), "n": size(48, 6000), "k": size(48, 6000),
                "alpha": round(rng.uniform(-2.0, 2.0), 3), "beta": rng.choice([0.0, 0.0, 1.0, -0.5])}
    if op == "ir":
        return {"op": op, "n": size(512, 6000), "nrhs": rng.choice([1, 1, 4, 16]),
                "kappa": 10.0 ** round(rng.uniform(1.0, 5.0), 2)}
    if op == "batch":
        nmin = size(4, 64)
        return {"op": op, "count": size(32, 8000), "nmin": nmin, "nmax": min(256, nmin + size(8, 250)),
                "rmax": rng.choice([1, 4, 16]), "ir": rng.random() < 0.4, "sizes": rng.randrange(1 << 30)}
    return {"op": op, "m": size(64, 16384), "n": size(64, 16384)}


# ---- inputs -------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(shape, g):
    return torch.rand(shape, dtype=torch.float64, device="cuda", generator=g).mul_(2.0).sub_(1.0)


def _spd(M):
    """M M^T + n I, exactly symmetric."""
    S = M @ M.mT
    S = 0.5 * (S + S.mT)
    S.diagonal(dim1=-2, dim2=-1).add_(float(M.shape[-1]))
    return S


def _randsvd(n, kappa, g):
    """U diag(sigma) V^T with U, V the Q factors of Gaussian matrices, sigma geometric from 1 to 1 / kappa."""
    s = kappa ** (-torch.arange(n, dtype=torch.float64, device="cuda") / max(n - 1, 1))
    U = torch.linalg.qr(torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g))[0]
    V = torch.linalg.qr(torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g))[0]
    return (U * s) @ V.mT


def _batch_shapes(case):
    g = np.random.Generator(np.random.Philox(case["sizes"]))
    cnt = case["count"]
    n = g.integers(case["nmin"], case["nmax"] + 1, cnt).astype(np.int32)
    r = g.integers(1, case["rmax"] + 1, cnt).astype(np.int32)
    kind = (np.arange(cnt) % 2).astype(np.int32)
    a = np.concatenate([[0], np.cumsum(n.astype(np.int64) ** 2)])
    b = np.concatenate([[0], np.cumsum(n.astype(np.int64) * r)])
    return n, r, kind, a, b


def _inputs(case, seed):
    g = _gen(seed)
    op = case["op"]
    if op == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"A": _uniform((m, k), g), "B": _uniform((k, n), g),
                "C": _uniform((m, n), g) if case["beta"] != 0.0 else None}
    if op == "matvec":
        return {"A": _uniform((case["m"], case["n"]), g), "x": _uniform((case["n"],), g)}
    if op == "batch":
        n, r, kind, a, b = _batch_shapes(case)
        A, B = _uniform((int(a[-1]),), g), _uniform((int(b[-1]),), g)
        for i in np.flatnonzero(kind == 1):
            m = int(n[i])
            v = A[int(a[i]):int(a[i + 1])].view(m, m)
            v.copy_(_spd(v.clone()))
        return {"A": A, "B": B}
    n, r = case["n"], case["nrhs"]
    if op == "ir":
        A = _randsvd(n, case["kappa"], g)
    else:
        A = _uniform((n, n), g)
        if op == "chol":
            A = _spd(A)
    return {"A": A, "B": _uniform((n,) if r == 1 else (n, r), g)}


def prepare(case, seed):
    state = _inputs(case, seed)
    state["case"] = case
    if case["op"] == "batch":
        n, r, kind, _, _ = _batch_shapes(case)
        state["plan"] = lmb200.Batch(n, r, kind, lmb200.PREC_FP32_IR if case["ir"] else lmb200.PREC_FP64)
        state["X"] = torch.empty_like(state["B"])
    return state


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "lu":
        return lmb200.luSolve(state["A"], state["B"])
    if op == "chol":
        return lmb200.choleskySolve(state["A"], state["B"])
    if op == "ir":
        return lmb200.luSolveIR(state["A"], state["B"])[0]
    if op == "batch":
        return state["plan"].solve(state["A"], state["B"], state["X"])
    if op == "matvec":
        return lmb200.matvec(state["A"], state["x"])
    if case["beta"] == 0.0:
        return lmb200.matMul(state["A"], state["B"])
    return lmb200.gemm(case["alpha"], state["A"], state["B"], case["beta"], state["C"])


# ---- what a pass cannot do without ----------------------------------------------------------

def work(case):
    op = case["op"]
    if op == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 8.0 * (m * k + k * n + (2 if case["beta"] != 0.0 else 1) * m * n), "flops": 2.0 * m * n * k}
    if op == "matvec":
        m, n = case["m"], case["n"]
        return {"bytes": 8.0 * (m * n + n + m), "flops": 2.0 * m * n}
    if op == "batch":
        lo, hi = case["nmin"], case["nmax"]
        k = np.arange(lo, hi + 1, dtype=np.float64)
        r = (1 + case["rmax"]) / 2.0
        # general and SPD instances alternate: 2/3 and 1/3 n^3; an SPD instance reads its lower triangle
        return {"bytes": float(case["count"] * np.mean(8.0 * (0.75 * k * k + 2.0 * k * r))),
                "flops": float(case["count"] * np.mean(0.5 * k ** 3 + 2.0 * k * k * r))}
    n, r = float(case["n"]), float(case["nrhs"])
    third = n ** 3 / 3.0
    return {"bytes": 8.0 * ((0.5 if op == "chol" else 1.0) * n * n + 2.0 * n * r),
            "flops": (third if op == "chol" else 2.0 * third) + 2.0 * n * n * r}


def tolerance(case):
    op = case["op"]
    if op == "matvec":
        return "exact"  # the reference's order of operations is part of the entry point's contract
    if op == "gemm":
        return {"rel": 1e-14}  # 1.6e-15 against another order of the sums
    if op == "chol":
        return {"rel": 5e-15}  # condition about 2: 0.6e-15 to 0.75e-15 over n = 701 .. 8192
    if op == "lu":
        # uniform matrices: the error is eps times a condition number with a heavy tail (P(kappa > t) ~ 1 / t).
        # Median 6e-16 n; over four seeds 2.3e-13 at n = 100 and 6.2e-9 at n = 16384.
        return {"rel": 1e-12 * case["n"]}
    if op == "ir":
        # the stopping test is a backward error of 1e-15 n, kappa times that in the solution: 0.45 of it at n = 8192
        return {"rel": 2e-15 * case["n"] * case["kappa"]}
    # the worst conditioned of the general instances decides the norm: 1e-11 .. 4e-10 in FP64, 2e-10 .. 3e-8 refined
    return {"rel": 4e-6 if case["ir"] else 4e-8}


# ---- the same results in 64 bits, in plain torch ---------------------------------------------

def _dot_rows(A, x):
    """sum_j A[..., i, j] x[..., j], the products and the sums with their rounding errors carried along."""
    def split(v):
        c = v * 134217729.0
        h = c - (c - v)
        return h, v - h

    x = x.unsqueeze(-2)
    p = A * x
    ah, al = split(A)
    xh, xl = split(x)
    e = ((ah * xh - p) + ah * xl + al * xh) + al * xl
    del ah, al
    while p.shape[-1] > 1:
        k = p.shape[-1]
        if k % 2:
            p, e = torch.nn.functional.pad(p, (0, 1)), torch.nn.functional.pad(e, (0, 1))
            k += 1
        a, b = p[..., :k // 2], p[..., k // 2:]
        s = a + b
        t = s - a
        e = (e[..., :k // 2] + e[..., k // 2:]) + ((a - (s - t)) + (b - t))
        p = s
    return p.squeeze(-1), e.squeeze(-1)


def _solve(A, B):
    """A^-1 B with residuals of about twice the precision (B has a column dimension)."""
    LU, piv = torch.linalg.lu_factor(A)
    X = torch.linalg.lu_solve(LU, piv, B)
    for _ in range(2):
        R = torch.empty_like(B)
        for c in range(B.shape[-1]):
            p, e = _dot_rows(A, X[..., c])
            R[..., c] = (B[..., c] - p) - e
        X = X + torch.linalg.lu_solve(LU, piv, R)
    return X


def exact(case, seed):
    op = case["op"]
    s = _inputs(case, seed)
    if op == "gemm":
        P = s["A"] @ s["B"]
        return P if case["beta"] == 0.0 else case["alpha"] * P + case["beta"] * s["C"]
    if op == "matvec":
        p, e = _dot_rows(s["A"], s["x"])
        return p + e
    if op == "batch":
        n, r, _, a, b = _batch_shapes(case)
        out = torch.empty_like(s["B"])
        for m in np.unique(n):
            ids, m = np.flatnonzero(n == m), int(m)
            A = torch.stack([s["A"][int(a[i]):int(a[i + 1])].view(m, m) for i in ids])
            B = torch.zeros((len(ids), m, int(r[ids].max())), dtype=torch.float64, device="cuda")
            for q, i in enumerate(ids):
                B[q, :, :int(r[i])] = s["B"][int(b[i]):int(b[i + 1])].view(m, int(r[i]))
            X = _solve(A, B)
            for q, i in enumerate(ids):
                out[int(b[i]):int(b[i + 1])] = X[q, :, :int(r[i])].reshape(-1)
        return out
    B = s["B"]
    X = _solve(s["A"], B.unsqueeze(1) if B.dim() == 1 else B)
    return X[:, 0] if B.dim() == 1 else X
