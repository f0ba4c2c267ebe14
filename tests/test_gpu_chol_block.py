"""The Cholesky block column: 128-column blocks, their 16-column diagonal chain and the
64-row substitution below, where a pivot fails and at the ends of the exponent range."""
import numpy as np
import pytest
import torch

import lmb200
from conftest import philox

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda")


@pytest.mark.parametrize("n,p", [(n, p) for n in (60, 128, 300) for p in (0, 1, 15, 16, 17, 31, 32, 47, 59, 111, 112, 127,
                                                                        128, 143, 144, 255, 256, 272, 299) if p < n])
def test_first_pivot_that_is_not_positive(ctx, n, p):
    # L D L^T with one negative d: the Cholesky pivots are d, so info is its place
    g = philox(9600 + n)
    L = np.tril(g.uniform(-1, 1, (n, n)), -1) / np.sqrt(n) + np.eye(n)
    d = g.uniform(1, 2, n)
    d[p] = -1.5
    S = (L * d) @ L.T
    S = dev(0.5 * (S + S.T))
    assert lmb200.dpotrf(S, ctx) == p + 1
    d[p] = 1.5
    S = (L * d) @ L.T
    assert lmb200.dpotrf(dev(0.5 * (S + S.T)), ctx) == 0  # nothing of the failure stays behind


@pytest.mark.parametrize("exp", [-1000, -600, 0, 600, 1000])
def test_exponent_range(ctx, exp):
    # diagonals of the factor between 2^-500 and 2^500 and their reciprocals
    n = 200
    M = philox(9700).uniform(-1, 1, (n, n))
    S = M @ M.T + n * np.eye(n)
    S = 0.5 * (S + S.T)
    G = dev(S * 2.0 ** exp)
    assert lmb200.dpotrf(G, ctx) == 0
    G = G.cpu().numpy() * 2.0 ** (-exp // 2)
    # |S - G G^T| <= gamma_(n+1) |G||G^T| (Higham, Theorem 10.3; products with reciprocals add
    # two roundings to each entry), and the check's own product
    assert np.all(np.abs(S - G @ G.T) <= 2 * (n + 4) * EPS * (np.abs(G) @ np.abs(G).T))
