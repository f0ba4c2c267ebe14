"""The persistent substitutions (up to four right-hand sides) at the edges of their
64-row blocks, and with solution entries whose bits are those of the scratch's
"not yet published" mark (all ones, a NaN)."""
import numpy as np
import pytest
import torch

import lmb200
from conftest import philox

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda")


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 128, 129, 200, 700])
@pytest.mark.parametrize("nrhs", [1, 2, 4])
def test_lu_blocks(ctx, n, nrhs):
    g = philox(9300 + 10 * n + nrhs)
    LU = g.uniform(-1, 1, (n, n)) / np.sqrt(n)
    LU[np.arange(n), np.arange(n)] = 10.0 ** g.uniform(-2, 2, n)
    ipiv = np.array([g.integers(i, n) for i in range(n)], dtype=np.int32)
    B = g.uniform(-1, 1, (n, nrhs))
    X = [lmb200.dgetrs(dev(LU), dev(ipiv), dev(B), ctx).cpu().numpy() for _ in range(3)]
    assert all(np.array_equal(X[0], x) for x in X[1:])
    L, U = np.tril(LU, -1) + np.eye(n), np.triu(LU)
    PB = B[lmb200.ipiv_to_perm(ipiv.tolist())]
    # two substitutions whose quotients are products with a reciprocal (two more roundings each):
    # |PB - L U X| <= (2 gamma_(n+2) + gamma^2) |L||U||X| (Higham, Theorem 8.5), and the check's own products
    assert np.all(np.abs(PB - L @ (U @ X[0])) <= 6 * (n + 4) * EPS * (np.abs(L) @ (np.abs(U) @ np.abs(X[0]))) + 1e-300)


@pytest.mark.parametrize("row", [0, 63, 64, 199])
def test_mark_as_a_value(ctx, row):
    n = 200
    B = np.ones((n, 2))
    B[row, 1] = np.frombuffer(b"\xff" * 8, dtype=np.float64)[0]
    LU = np.eye(n) + np.tril(np.full((n, n), 1e-3), -1)
    X = lmb200.dgetrs(dev(LU), dev(np.arange(n, dtype=np.int32)), dev(B), ctx).cpu().numpy()
    ctx.check()
    assert np.isfinite(X[:, 0]).all()
    assert np.isnan(X[:, 1]).all()  # forward below it, and above it by the zeros of U
