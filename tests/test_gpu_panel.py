"""The cluster panel kernel and the row-block kernel at the edges of their shapes.

The panel kernel picks its CTAs and rows per thread from the number of rows:
32-row CTAs up to 512 rows, 16 CTAs beyond; one row per thread up to 8192 rows
in FP64 (two in FP32 up to 16384), then 2, 4 and 8.  The leaf narrows with it
(32, 16, 8, 4 columns).  Each order below is the first or last of a shape, or
leaves ragged leaves, panels and column blocks.
"""
import numpy as np
import pytest
import torch

import lmb200
import oracle as O
from conftest import philox

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda")


@pytest.mark.parametrize("n", [31, 32, 33, 41, 127, 129, 160, 161, 255, 257, 383, 385, 511, 513, 545, 1025])
def test_pivots_and_factor(ctx, n):
    g = philox(9100 + n)
    A, b = g.uniform(-1, 1, (n, n)), g.uniform(-1, 1, n)
    LU, ipiv, info = lmb200.lu_factor(dev(A), ctx)
    _, _, ipo = O.lu_solve_p(A, b)
    assert info == 0 and np.array_equal(ipiv.cpu().numpy(), ipo)
    F = LU.cpu().numpy()
    L, U = np.tril(F, -1) + np.eye(n), np.triu(F)
    PA = A[lmb200.ipiv_to_perm(ipo.tolist())]
    # |PA - LU| <= gamma_n |L||U| (Higham, Theorem 9.3), gamma_n = n eps / (1 - n eps)
    assert np.all(np.abs(PA - L @ U) <= 2 * n * EPS * (np.abs(L) @ np.abs(U)) + 1e-300)


@pytest.mark.parametrize("scale", [1e-290, 1e290, 5e-324 * 2.0 ** 60])
def test_pivots_outside_the_reciprocal_range(ctx, scale):
    # pivots too small or too large for multipliers by reciprocal take true divisions
    n = 200
    A = philox(77).uniform(-1, 1, (n, n)) * scale
    LU, ipiv, info = lmb200.lu_factor(dev(A), ctx)
    _, _, ipo = O.lu_solve_p(A, np.ones(n))
    assert info == 0 and np.array_equal(ipiv.cpu().numpy(), ipo)
    F = LU.cpu().numpy()
    assert np.all(np.abs(np.tril(F, -1)) <= 1.0) and np.all(np.isfinite(F))


@pytest.mark.parametrize("n", [8193, 16385, 32769])
def test_rows_per_thread(ctx, n):
    # the first panels take 2, 4 and 8 rows per thread; partial pivoting bounds |L| by 1,
    # and the solve's normwise backward error is the suite's 1e-15 n
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    A = torch.rand((n, n), dtype=torch.float64, device="cuda", generator=gen).mul_(2).sub_(1)
    b = torch.rand((n, 1), dtype=torch.float64, device="cuda", generator=gen).mul_(2).sub_(1)
    LU, ipiv, info = lmb200.lu_factor(A, ctx)
    assert info == 0
    worst = max(float(LU[i:i + 512, :i].abs().max()) for i in range(512, n, 512))
    assert worst <= 1.0
    x = lmb200.dgetrs(LU, ipiv, b.clone(), ctx)
    del LU
    r = (A @ x - b).abs().max()
    anorm = max(float(A[i:i + 1024].abs().sum(1).max()) for i in range(0, n, 1024))
    assert float(r) <= 1e-15 * n * (anorm * float(x.abs().max()) + float(b.abs().max()))


@pytest.mark.parametrize("n", [16385, 32769])
def test_rows_per_thread_fp32_factor(ctx, n):
    # the FP32 panel's shapes of 4 and 8 rows per thread (a shifted matrix: kappa is small,
    # so refinement converges whatever the factor's growth)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    A = torch.rand((n, n), dtype=torch.float64, device="cuda", generator=gen).mul_(2).sub_(1)
    A.diagonal().add_(2.0 * n ** 0.5)
    b = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen).mul_(2).sub_(1)
    x, iters, berr, st = lmb200.luSolveIR(A, b, ctx=ctx)
    assert st == 0 and berr <= 1e-15 * n and iters <= 10
