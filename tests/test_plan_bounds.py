"""Pivot labels and row plans that a healthy panel never produces: after a wait that
gave up, both can hold anything, and neither may lead a write out of range."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import lmb200
from conftest import ROOT, philox

INT_MAX, INT_MIN = 2**31 - 1, -2**31
PLAN_ROWS, PLAN_INTS = 256, 1 + 2 * 256 + 15  # kSwapPlanRows, kSwapPlanInts
BOUNDS = 2                                    # LM_DEVERR_BOUNDS


def test_a_wait_that_gave_up_makes_no_interchange(tmp_path):
    # the device function itself, compiled for the host
    src = tmp_path / "t.cu"
    src.write_text("""
#include <cstdio>
#include "pivot.cuh"
int main() {
  int label, J, gave_up;
  while (scanf("%d %d %d", &label, &J, &gave_up) == 3) printf("%d\\n", lm::pivot_position(label, J, gave_up != 0));
}
""")
    exe = tmp_path / "t"
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(ROOT, "linear-massiv_b200", "csrc"),
                    "-o", str(exe), str(src)], check=True)
    J = 40
    rows = [(lab, J, g) for g in (0, 1) for lab in (INT_MIN, -1, 0, J, J + 1, 65535, INT_MAX - 1, INT_MAX)]
    out = subprocess.run([str(exe)], input="\n".join("%d %d %d" % r for r in rows), capture_output=True, text=True,
                         check=True).stdout.split()
    assert len(out) == len(rows)
    for (lab, J, g), p in zip(rows, map(int, out)):
        assert p == (J if g or lab == INT_MAX else lab), (lab, J, g, p)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,sym", [("float64", "_ZN2lm9row_blockIdEEiPT_xPKiiiiiiiiPiP11CUstream_st"),
                                       ("float32", "_ZN2lm9row_blockIfEEiPT_xPKiiiiiiiiPiP11CUstream_st")])
def test_row_block_leaves_out_rows_outside_the_panel(dtype, sym):
    import torch

    fn = getattr(lmb200.lib(), sym)
    n, k0, w, lda, guard = 300, 32, 128, 260, 64
    g = philox(9500)
    # `guard` rows of the allocation before and after the matrix
    buf = g.uniform(-1, 1, (n + 2 * guard, lda)).astype(dtype)
    A = buf[guard:guard + n]
    A[k0:k0 + w, k0:k0 + w] *= 0.1
    moves = {40: 200, 200: 40, 33: 34, 34: 33}  # destination: source
    bad = [(-1, 50), (k0 - 1, 60), (n, 70), (n + 5, 80), (INT_MIN, 40), (INT_MAX, 40), (100, -7), (101, n + 9),
           (250, k0 - 2), (INT_MIN, INT_MAX)]
    plan = np.zeros(PLAN_INTS, np.int32)
    rows = bad[:5] + list(moves.items()) + bad[5:]
    plan[0] = len(rows)
    for e, (d, s) in enumerate(rows):
        plan[1 + e], plan[1 + PLAN_ROWS + e] = d, s
    dev = torch.from_numpy(buf.copy()).cuda()
    dplan, status = torch.from_numpy(plan).cuda(), torch.zeros(8, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream()
    ll, p = ctypes.c_longlong, ctypes.c_void_p
    ca0, ca1, cb0, cb1 = 0, 20, k0 + w, lda  # columns moved only; columns moved and solved
    esz = buf.itemsize
    assert fn(p(dev.data_ptr() + guard * lda * esz), ll(lda), p(dplan.data_ptr()), n, k0, w, ca0, ca1, cb0, cb1,
              p(status.data_ptr()), p(st.cuda_stream)) == 0
    torch.cuda.synchronize()
    assert int(status[0]) == BOUNDS
    ref = A.copy()
    for d, s in moves.items():
        ref[d, ca0:ca1], ref[d, cb0:cb1] = A[s, ca0:ca1], A[s, cb0:cb1]
    got = dev.cpu().numpy()
    assert np.array_equal(got[:guard], buf[:guard]) and np.array_equal(got[guard + n:], buf[guard + n:])
    got = got[guard:guard + n]
    solved = np.zeros((n, lda), bool)
    solved[k0:k0 + w, cb0:cb1] = True
    assert np.array_equal(got[~solved], ref[~solved])
    # the block solve of the moved rows: |L X - B| <= gamma_w |L||X| (Higham, Theorem 8.5), and the check's own product
    L = np.tril(A[k0:k0 + w, k0:k0 + w].astype(np.float64), -1) + np.eye(w)
    X, B = got[k0:k0 + w, cb0:cb1].astype(np.float64), ref[k0:k0 + w, cb0:cb1].astype(np.float64)
    eps = np.finfo(dtype).eps
    with np.errstate(all="ignore"):
        assert np.all(np.abs(L @ X - B) <= 2 * (w + 1) * eps * (np.abs(L) @ np.abs(X)) + np.finfo(dtype).tiny)
