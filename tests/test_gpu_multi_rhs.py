"""Substitutions with more than four right-hand sides: the 128-row block solves
(blocks of 32 rows, eight columns per CTA) at their edges, and the composed
interchanges, against componentwise error bounds."""
import numpy as np
import pytest
import torch

import lmb200
from conftest import philox

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda")


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 96, 127, 128, 129, 161, 300])
@pytest.mark.parametrize("nrhs", [5, 8, 9, 17, 64, 65])
def test_lu_blocks(ctx, n, nrhs):
    g = philox(7000 + 100 * n + nrhs)
    # a factor with |l| <= 1 and diagonals of mixed size, and a random swap list
    LU = g.uniform(-1, 1, (n, n)) / np.sqrt(n)
    LU[np.arange(n), np.arange(n)] = 10.0 ** g.uniform(-2, 2, n)
    ipiv = np.array([g.integers(i, n) for i in range(n)], dtype=np.int32)
    B = g.uniform(-1, 1, (n, nrhs))
    X = lmb200.dgetrs(dev(LU), dev(ipiv), dev(B), ctx).cpu().numpy()
    L, U = np.tril(LU, -1) + np.eye(n), np.triu(LU)
    PB = B[lmb200.ipiv_to_perm(ipiv.tolist())]
    # two substitutions: |PB - L U X| <= (2 gamma_n + gamma_n^2) |L||U||X|  (Higham, Theorem 8.5);
    # the check's own products are within another 2 gamma_n of that
    assert np.all(np.abs(PB - L @ (U @ X)) <= 5 * (n + 2) * EPS * (np.abs(L) @ (np.abs(U) @ np.abs(X))) + 1e-300)


@pytest.mark.parametrize("n,nrhs", [(1, 5), (33, 6), (128, 16), (200, 9), (257, 33)])
def test_cholesky_blocks(ctx, n, nrhs):
    g = philox(7900 + n)
    M = g.uniform(-1, 1, (n, n))
    S = M @ M.T + n * np.eye(n)
    S = 0.5 * (S + S.T)
    B = g.uniform(-1, 1, (n, nrhs))
    X = lmb200.choleskySolve(dev(S), dev(B), ctx).cpu().numpy()
    # factor and two substitutions: (3 n + 1) eps |G||G^T||X|, and |G||G^T| <= n max S (Higham, Theorem 10.4)
    bound = (5 * n + 5) * EPS * n * np.abs(S).max() * np.abs(X).sum(0)
    assert np.all(np.abs(B - S @ X) <= bound)


@pytest.mark.parametrize("scale", [1e-200, 1e200])
def test_diagonals_outside_the_reciprocal_range(ctx, scale):
    # every quotient is a plain division there: a diagonal solve gives it exactly
    n = 70
    d = philox(7990).uniform(1, 2, n) * scale
    B = philox(7991).uniform(-1, 1, (n, 7)) * scale
    B[3, 2], B[40, 5] = 0.0, np.inf
    X = lmb200.dgetrs(dev(np.diag(d)), dev(np.arange(n, dtype=np.int32)), dev(B), ctx).cpu().numpy()
    ref = B / d[:, None]
    keep = np.ones((n, 7), bool)
    keep[:, 5] = False  # an infinity times the zeros of its block is NaN
    assert np.array_equal(X[keep], ref[keep])
    assert not np.isfinite(X[40, 5])
