"""The batch kernel at the edges of its shapes: 16-row panels and blocks, one and
two rows per thread (128), 32-row warps, 96-column update chunks, eight right-hand
sides; both kinds and both precisions, with factors in LAPACK order."""
import ctypes

import numpy as np
import pytest
import torch

import lmb200
import oracle as O
from conftest import philox

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16
SIZES = [1, 2, 3, 15, 16, 17, 31, 32, 33, 48, 96, 112, 113, 127, 128, 129, 144, 160, 255, 256]


def instances(seed, scale=1.0):
    g = philox(seed)
    n = np.repeat(np.array(SIZES, np.int32), 4)
    kind = np.tile(np.array([0, 1, 0, 1], np.int32), len(SIZES))
    nrhs = np.tile(np.array([1, 8, 9, 16], np.int32), len(SIZES))
    A, B = [], []
    for m, k, r in zip(n, kind, nrhs):
        M = g.uniform(-1, 1, (m, m))
        if k == 1:
            M = M @ M.T + m * np.eye(m)
            M = 0.5 * (M + M.T)
        A.append(M * scale)
        B.append(g.uniform(-1, 1, (m, r)) * scale)
    return n, nrhs, kind, A, B


def solve(plan, A, B, **kw):
    dA = torch.from_numpy(np.concatenate([a.ravel() for a in A])).cuda()
    dB = torch.from_numpy(np.concatenate([b.ravel() for b in B])).cuda()
    dX = torch.empty_like(dB)
    plan.solve(dA, dB, dX, **kw)
    X = dX.cpu().numpy()
    out, at = [], 0
    for b in B:
        out.append(X[at:at + b.size].reshape(b.shape))
        at += b.size
    return out


def backward(A, X, B):
    with np.errstate(all="ignore"):
        return np.abs(B - A @ X).max(0) / (np.abs(A).sum(1).max() * np.abs(X).max(0) + np.abs(B).max(0))


@pytest.mark.parametrize("prec", [lmb200.PREC_FP64, lmb200.PREC_FP32_IR])
@pytest.mark.parametrize("nb", [8, 16, 32])
def test_sizes(prec, nb):
    n, nrhs, kind, A, B = instances(8100)
    old = lmb200.batch_tune_get()
    lmb200.batch_tune_set([[nb] * 4] * 2)
    try:
        plan = lmb200.Batch(n, nrhs, kind, prec)
    finally:
        lmb200.batch_tune_set(old)
    X = solve(plan, A, B)
    info, iters, berr = plan.results()
    assert (info == 0).all()
    for a, x, b in zip(A, X, B):
        assert backward(a, x, b).max() <= 1e-15 * max(len(a), 8)
    if prec == lmb200.PREC_FP64:
        fptr, pptr = plan.factors()
        F = np.empty(int((n.astype(np.int64) ** 2).sum()))
        P = np.empty(int(n.sum()), np.int32)
        for h, p in ((F, fptr), (P, pptr)):
            assert lmb200.lib().lm_d2h(plan.ctx.h, ctypes.c_void_p(h.ctypes.data), ctypes.c_void_p(p), h.nbytes) == 0
        at = pt = 0
        for m, k, a in zip(n, kind, A):
            f, ip = F[at:at + m * m].reshape(m, m), P[pt:pt + m]
            at, pt = at + m * m, pt + m
            L, U = (np.tril(f, -1) + np.eye(m), np.triu(f)) if k == 0 else (np.tril(f), np.tril(f).T)
            if k == 0:
                assert np.array_equal(ip, O.lu_solve_p(a, np.ones(m))[2])
                a = a[lmb200.ipiv_to_perm(ip.tolist())]
            # |A - LU| <= gamma_n |L||U| (Higham, Theorems 9.3 and 10.3), and the check's own product
            assert np.all(np.abs(a - L @ U) <= 2 * (m + 1) * EPS * (np.abs(L) @ np.abs(U)))


@pytest.mark.parametrize("scale", [1e-200, 1e200])
def test_outside_the_reciprocal_range(scale):
    # pivots there are divided by; the systems are the plain ones times a power of ten
    n, nrhs, kind, A, B = instances(8200, scale)
    plan = lmb200.Batch(n, nrhs, kind, lmb200.PREC_FP64)
    X = solve(plan, A, B)
    assert (plan.results()[0] == 0).all()
    for a, x, b in zip(A, X, B):
        assert backward(a / scale, x, b / scale).max() <= 1e-15 * max(len(a), 8)


def test_nan_and_ties():
    # a NaN on the diagonal stays the pivot, NaNs below never win, the lowest row wins a tie
    n = np.array([40, 40], np.int32)
    g = philox(8300)
    A0 = g.uniform(-1, 1, (40, 40))
    A0[:, 0] = np.where(np.arange(40) % 2, -1.0, 1.0)
    A1 = g.uniform(-1, 1, (40, 40))
    A1[5:, 3] = np.nan
    A = [A0, A1]
    B = [np.ones((40, 1))] * 2
    plan = lmb200.Batch(n, np.ones(2, np.int32), np.zeros(2, np.int32), lmb200.PREC_FP64)
    X = solve(plan, A, B)
    _, pptr = plan.factors()
    P = np.empty(80, np.int32)
    assert lmb200.lib().lm_d2h(plan.ctx.h, ctypes.c_void_p(P.ctypes.data), ctypes.c_void_p(pptr), P.nbytes) == 0
    assert np.array_equal(P[:40], O.lu_solve_p(A0, B[0][:, 0])[2])
    assert np.array_equal(P[40:], O.lu_solve_p(A1, B[1][:, 0])[2])
    assert np.isfinite(X[0]).all()


def test_refinement_never_accepts_what_is_not_finite():
    # entries beyond FP32's range, NaN and infinities beside ordinary systems: the former
    # must come from the FP64 fallback, the latter must not be reported as converged
    g = philox(8400)
    m, r = 40, 3
    plain = g.uniform(-1, 1, (m, m)) + 4 * np.eye(m)
    spd = plain @ plain.T + m * np.eye(m)
    spd = 0.5 * (spd + spd.T)
    rhs = g.uniform(-1, 1, (m, r))
    bad_a, bad_b, inf_a, inf_b = plain.copy(), rhs.copy(), plain.copy(), rhs.copy()
    bad_a[7, 3], bad_b[5, 1], inf_a[2, 9], inf_b[11, 2] = np.nan, np.nan, np.inf, -np.inf
    cases = [(plain, rhs, 0, "refined"), (plain * 1e39, rhs, 0, "fp64"), (spd, rhs, 1, "refined"),
             (spd * 1e39, rhs, 1, "fp64"), (plain, rhs * 1e39, 0, "fp64"), (spd, rhs * 1e39, 1, "fp64"),
             (bad_a, rhs, 0, "never"), (plain, bad_b, 0, "never"), (spd, bad_b, 1, "never"),
             (inf_a, rhs, 0, "never"), (plain, inf_b, 0, "never"), (spd, inf_b, 1, "never"),
             (plain, rhs, 0, "refined")]
    A, B = [c[0] for c in cases], [c[1] for c in cases]
    plan = lmb200.Batch(np.full(len(cases), m, np.int32), np.full(len(cases), r, np.int32),
                        np.array([c[2] for c in cases], np.int32), lmb200.PREC_FP32_IR)
    X = solve(plan, A, B)
    info, iters, berr = plan.results()
    for i, (a, b, _, want) in enumerate(cases):
        if want == "refined":
            assert info[i] == 0 and iters[i] >= 0 and berr[i] <= 1e-15 * m, i
        else:
            assert iters[i] == -1 and not berr[i] <= 1e-15 * m, (i, iters[i], berr[i])
        if want != "never":
            assert info[i] == 0 and backward(a, X[i], b).max() <= 1e-15 * m, i


@pytest.mark.parametrize("scale", [1.0, 1e-200])  # 1e-200: the diagonal blocks take their divisions
@pytest.mark.parametrize("prec", [lmb200.PREC_FP64, lmb200.PREC_FP32_IR])
def test_first_pivot_that_is_not_positive(prec, scale):
    # L D L^T with one negative d: the Cholesky pivots are d, so info is its place, in
    # every column of the 16-column blocks, of their halves and of ragged last blocks
    g = philox(8500)
    cases = [(n, p) for n in (4, 8, 9, 16, 24, 40) for p in range(n)]
    A, B = [], []
    for n, p in cases:
        L = np.tril(g.uniform(-0.5, 0.5, (n, n)), -1) + np.eye(n)
        d = g.uniform(1, 2, n)
        d[p] = -1.5
        M = (L * d) @ L.T
        A.append(0.5 * (M + M.T) * scale)
        B.append(g.uniform(-1, 1, (n, 2)))
    plan = lmb200.Batch(np.array([n for n, _ in cases], np.int32), np.full(len(cases), 2, np.int32),
                        np.ones(len(cases), np.int32), prec)
    solve(plan, A, B)
    info = plan.results()[0]
    assert np.array_equal(info, [p + 1 for _, p in cases])


def test_tuner_keeps_a_width_that_the_kernel_has():
    ctx = lmb200.Context(0)
    for prec in (lmb200.PREC_FP64, lmb200.PREC_FP32_IR):
        lmb200.batch_tune_set([[32] * 4] * 2, ctx)  # accepted, and runs as 16
        assert lmb200.batch_tune_get(ctx) == [[32] * 4] * 2
        table = lmb200.batch_tune(prec, None, ctx)
        assert set(table[prec]) <= {8, 16}, table
        assert table[1 - prec] == [32] * 4
