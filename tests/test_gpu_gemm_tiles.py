"""The FP64 GEMM at the edges of its 64 x 64 tiles, of the 16-deep k-slices and of
the k = 256 line between its two forms, and that the CTAs of one SM do not disturb
each other's operand rings: more tiles than CTAs, repeated, bit for bit."""
import numpy as np
import pytest
import torch

import lmb200
from conftest import philox

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


@pytest.mark.parametrize("m,n", [(1, 1), (63, 65), (64, 64), (65, 63), (128, 130), (200, 20), (700, 900)])
@pytest.mark.parametrize("k", [1, 15, 16, 17, 256, 257])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-1.0, 1.0), (0.75, -0.5)])
def test_tile_edges(ctx, m, n, k, alpha, beta):
    g = philox(100 * m + 10 * n + k)
    A, B, C = g.uniform(-1, 1, (m, k)), g.uniform(-1, 1, (k, n)), g.uniform(-1, 1, (m, n))
    D = torch.from_numpy(C).cuda()
    lmb200.dgemm(alpha, torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), beta, D, ctx)
    # |fl - exact| <= gamma_(k+3) (|alpha| |A||B| + |beta| |C|), for either of two orders
    bound = 2 * (k + 3) * EPS * (abs(alpha) * (np.abs(A) @ np.abs(B)) + abs(beta) * np.abs(C))
    assert np.all(np.abs(D.cpu().numpy() - (alpha * (A @ B) + beta * C)) <= bound + 1e-300)


@pytest.mark.parametrize("m,n,k", [(1500, 1002, 2000), (6000, 300, 1000), (2000, 2000, 128)])
def test_repeats_bitwise(ctx, m, n, k):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(m + n + k)
    A, B, C = (torch.rand(s, dtype=torch.float64, device="cuda", generator=gen) for s in ((m, k), (k, n), (m, n)))
    ref = None
    for i in range(60):
        D = C.clone()
        if i % 3 == 0:
            A @ B  # other work just before: the CTAs then run less in step
        lmb200.dgemm(1.0, A, B, 1.0, D, ctx)
        ref = D if ref is None else ref
        assert torch.equal(D, ref), f"run {i}: {int((D != ref).sum())} entries differ"


@pytest.mark.parametrize("k", [4, 16, 48])
def test_staged_c_repeats_bitwise(ctx, k):
    # one to three k-slices per tile: the staged C tile and the ring slots are given back
    # and refilled as fast as they can be, many tiles per CTA
    gen = torch.Generator(device="cuda")
    gen.manual_seed(k)
    A, B, C = (torch.rand(s, dtype=torch.float64, device="cuda", generator=gen) for s in ((3000, k), (k, 3002), (3000, 3002)))
    ref = None
    for i in range(60):
        D = C.clone()
        if i % 3 == 0:
            A @ B
        lmb200.dgemm(-1.0, A, B, 1.0, D, ctx)
        ref = D if ref is None else ref
        assert torch.equal(D, ref), f"run {i}: {int((D != ref).sum())} entries differ"
    exact = C - A @ B
    # |fl - exact| <= gamma_(k+2) (|A||B| + |C|) for either of two orders; all entries are positive
    assert bool(((ref - exact).abs() <= 2 * (k + 2) * EPS * (A @ B + C)).all())
