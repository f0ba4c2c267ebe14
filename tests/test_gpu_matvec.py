"""The staged matvec at the edges of its chunks: rows in eights, 64-column
chunks six deep, the 16-byte and the 8-byte copies, and the last n mod 4
columns.  The oracle follows the reference's order, so the bar is equality."""
import numpy as np
import pytest
import torch

import lmb200
import oracle as O
from conftest import philox

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 7, 8, 9, 65])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 63, 64, 66, 319, 320, 384, 388, 1027])
def test_matvec_chunk_edges(m, n):
    g = philox(1000 * m + n)
    A = g.uniform(-1.0, 1.0, (m, n))
    x = g.uniform(-1.0, 1.0, n)
    ref = O.matvec_p(A, x)
    y = lmb200.matvec(torch.from_numpy(A).cuda(), torch.from_numpy(x).cuda()).cpu().numpy()
    assert np.array_equal(y, ref)
    # rows that start on 8 bytes only, inside a wider matrix; x on 8 bytes
    big = torch.zeros((m, n + 4), dtype=torch.float64, device="cuda")
    big[:, 1:n + 1] = torch.from_numpy(A)
    xs = torch.zeros(n + 1, dtype=torch.float64, device="cuda")
    xs[1:] = torch.from_numpy(x)
    y = lmb200.matvec(big[:, 1:n + 1], xs[1:]).cpu().numpy()
    assert np.array_equal(y, ref)


def test_matvec_nonfinite():
    A = np.ones((9, 130))
    x = np.ones(130)
    A[0, 3], A[1, 128], A[2, 129], x[64] = np.inf, np.nan, -np.inf, -0.0
    y = lmb200.matvec(torch.from_numpy(A).cuda(), torch.from_numpy(x).cuda()).cpu().numpy()
    assert np.array_equal(y, O.matvec_p(A, x), equal_nan=True)


@pytest.mark.parametrize("m,n", [(65, 127), (65, 128), (65, 129), (8, 130),  # the short-row line
                                 (200, 1), (1001, 7), (300, 128),
                                 # rows that fill the chip once, its edge at 85% of a wave, a wave and a half
                                 (75776, 129), (75776, 1024), (75776, 1025), (64409, 150), (64410, 150),
                                 (113664, 131)])
def test_matvec_forms(m, n):
    g = philox(3 * m + n)
    A = g.uniform(-1.0, 1.0, (m, n))
    x = g.uniform(-1.0, 1.0, n)
    y = lmb200.matvec(torch.from_numpy(A).cuda(), torch.from_numpy(x).cuda()).cpu().numpy()
    assert np.array_equal(y, O.matvec_p(A, x))
