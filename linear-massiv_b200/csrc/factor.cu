// Host-side drivers of the FP64 factorisations and triangular solves.
//
// dgetrf — right-looking blocked LU, outer panels of kNB = 128 columns so the
//   trailing update is a k = 128 DMMA GEMM (compute-bound on B200, unlike the
//   reference's k = 32 update, LU.hs:311-357).  A panel is one cluster launch
//   (panel_lu); its row interchanges and U12 = L11^-1 A12
//   (rawTriSolvePanelTrail, LU.hs:364-407) reach the other columns in one
//   launch each side of the look-ahead (row_block).  Row interchanges are
//   applied to every column of A, matching the reference's full-row
//   rawSwapRows (fromCol = 0, LU.hs:324-325).
// dpotrf — right-looking blocked Cholesky, kNB = 128: diagonal block in SMEM,
//   L21 = A21 L11^-T by substitution, then A22 -= L21 L21^T as a
//   lower-triangle-only GEMM (SYRK tile skip).  Same
//   mathematics as the reference's left-looking panelCholFactor
//   (Chol.hs:279-321), different association.
// dgetrs / dpotrs — blocked substitutions: a 128 x 128 triangular block
//   solve, then the rest of the right-hand side updated by GEMM; dgetrs with
//   at most 4 right-hand sides runs one persistent launch per direction
//   (trsv.cu).
#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace lm {

namespace {

constexpr int kNB = 128;

// B (w x ncols, ldb) <- inv(unit lower L11) B (the no-pivot factorisation's
// row block).  Small blocks in one fused launch; otherwise inv(L11) (Linv,
// kNB x kNB scratch) times a copy of B (W, kNB x (ncols + 1) scratch) on the
// tensor cores.
int trsm_unit_lower_gemm(Ctx& c, const double* L11, long long lda, int w, double* B, long long ldb, int ncols,
                         double* Linv, double* W, cudaStream_t st) {
  if (w <= 0 || ncols <= 0) return LM_OK;
  if (w <= 64 && ncols <= 128) {
    Prof p(c, kPhaseTrsm, (double)w * w * ncols, 8.0 * ((double)w * w / 2 + 2.0 * w * ncols), st);
    return trsm_lower_small<double>(L11, lda, w, true, B, ldb, ncols, st);
  }
  const long long ldw = (ncols + 1) & ~1;
  {
    Prof p(c, kPhaseTrsm, (double)w * w * w / 3.0, 8.0 * (double)w * w + 16.0 * w * ncols, st);
    LM_TRY(tri_inv_lower<double>(L11, lda, w, true, Linv, kNB, nullptr, st));
    LM_TRY(copy2d<double>(W, ldw, B, ldb, w, ncols, st));
  }
  GemmDesc d;
  d.m = w; d.n = ncols; d.k = w;
  d.alpha = 1.0; d.beta = 0.0;
  d.A = Linv; d.lda = kNB;
  d.B = W; d.ldb = ldw;
  d.C = B; d.ldc = ldb;
  return dgemm(c, d, st);
}

}  // namespace

// Order from which a panel (or block column) is factored beside the trailing
// update, and the SMs that the Cholesky update leaves for it.
constexpr int kLookaheadSms = 16;
constexpr int kLookaheadMinN = 384;

// The chain from one panel to the next holds only what the next panel needs:
// the interchanges, block solve and update of its own 128 columns.  With
// look-ahead it is then factored on the priority stream while the same three
// operations run on the rest of the matrix, on the SMs that the panel's
// cluster leaves and, once it is done, on those too (tiles by ticket).  Nothing waits across the two streams inside a kernel; at
// worst the panel starts when the update ends.
int dgetrf(Ctx& c, int n, double* A, long long lda, int* ipiv, cudaStream_t st) {
  int* plan[2];  // row plans of the current panel and of the one factored beside its update
  {
    void* ws = nullptr;
    LM_TRY(ctx_workspace(c, 1, 2 * sizeof(int) * kSwapPlanInts, &ws));
    plan[0] = static_cast<int*>(ws);
    plan[1] = plan[0] + kSwapPlanInts;
  }
  const int nsm = ctx_num_sms(c);
  const bool la = n >= kLookaheadMinN && nsm > 2 * kLookaheadSms && ctx_lookahead(c);
  cudaStream_t aux = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  if (la) LM_TRY(ctx_aux(c, &aux, &ev_fork, &ev_join));
  auto panel = [&](int k0, cudaStream_t s) {
    const int w = std::min(kNB, n - k0);
    Prof p(c, kPhasePanel, (double)(n - k0) * w * w, 16.0 * (n - k0) * w, s);
    return panel_lu<double>(c, A, lda, n, k0, w, ipiv, plan[(k0 / kNB) & 1], s);
  };
  LM_TRY(panel(0, st));
  for (int k0 = 0; k0 < n; k0 += kNB) {
    const int w = std::min(kNB, n - k0);
    const int m = n - k0 - w;
    const int wn = std::min(kNB, m);  // next panel
    const int* pl = plan[(k0 / kNB) & 1];
    auto rows = [&](int ca0, int ca1, int cb0, int cb1) {
      Prof p(c, kPhaseTrsm, (double)w * w * (cb1 - cb0), 8.0 * (4.0 * w * (ca1 - ca0 + cb1 - cb0) + 0.5 * w * w), st);
      return row_block<double>(A, lda, pl, n, k0, w, ca0, ca1, cb0, cb1, ctx_status(c), st);
    };
    if (m <= 0) {
      LM_TRY(rows(0, k0, n, n));
      break;
    }
    const int nx = k0 + w, rx = nx + wn;  // first columns of the next panel and of the rest
    LM_TRY(rows(0, 0, nx, rx));
    double* A11 = A + (long long)k0 * lda + k0;
    GemmDesc d;  // A22 -= L21 U12, the next panel's columns first
    d.m = m; d.n = wn; d.k = w;
    d.alpha = -1.0; d.beta = 1.0;
    d.A = A11 + (long long)w * lda; d.lda = lda;
    d.B = A11 + w; d.ldb = lda;
    d.C = A11 + (long long)w * lda + w; d.ldc = lda;
    LM_TRY(dgemm(c, d, st));
    GemmDesc r = d;  // the rest of the columns
    r.n = m - wn;
    r.B = A11 + w + wn;
    r.C = A11 + (long long)w * lda + w + wn;
    if (la) {
      LM_CUDA_TRY(cudaEventRecord(ev_fork, st));
      LM_CUDA_TRY(cudaStreamWaitEvent(aux, ev_fork, 0));
      LM_TRY(panel(nx, aux));
      LM_CUDA_TRY(cudaEventRecord(ev_join, aux));
      r.sched = ctx_status(c) + 2;
    }
    LM_TRY(rows(0, k0, rx, n));
    if (r.n > 0) LM_TRY(dgemm(c, r, st));
    if (la)
      LM_CUDA_TRY(cudaStreamWaitEvent(st, ev_join, 0));
    else
      LM_TRY(panel(nx, st));
  }
  return LM_OK;
}

// Right-looking blocked Cholesky with look-ahead: once the trailing update
// has reached the next block column (its diagonal block and everything
// below), that column is factored on the priority stream (diagonal block,
// L21) while the rest of the lower-triangle update runs on the
// other SMs.  The two streams touch disjoint columns: the update reads the
// current L21 and writes columns right of the next block column.
int dpotrf(Ctx& c, int n, double* A, long long lda, cudaStream_t st) {
  const int nsm = ctx_num_sms(c);
  const bool la = n >= kLookaheadMinN && nsm > 2 * kLookaheadSms && ctx_lookahead(c);
  cudaStream_t aux = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  if (la) LM_TRY(ctx_aux(c, &aux, &ev_fork, &ev_join));
  auto factor_column = [&](int j0, cudaStream_t s) {
    const int w = std::min(kNB, n - j0);
    const int R = n - j0 - w;
    {
      Prof p(c, kPhasePanel, (double)w * w * w / 3.0, 8.0 * w * w, s);
      LM_TRY(potrf_block(c, A + (long long)j0 * lda + j0, lda, w, j0, s));
    }
    Prof p(c, kPhaseTrsm, (double)R * w * w, 16.0 * R * w, s);
    return chol_rows(c, A + (long long)j0 * lda + j0, lda, R, s);
  };
  LM_TRY(factor_column(0, st));
  for (int j0 = 0; j0 < n; j0 += kNB) {
    const int w = std::min(kNB, n - j0);
    const int R = n - j0 - w;
    if (R <= 0) break;
    double* A21 = A + (long long)(j0 + w) * lda + j0;
    double* A22 = A21 + w;
    const int wn = std::min(kNB, R);  // next block column
    // A22 -= L21 L21^T: the next block column first (all R rows of it)
    GemmDesc d;
    d.m = R; d.n = wn; d.k = w; d.alpha = -1.0; d.beta = 1.0;
    d.A = A21; d.lda = lda; d.B = A21; d.ldb = lda; d.b_trans = true;
    d.C = A22; d.ldc = lda;
    LM_TRY(dgemm(c, d, st));
    const int rest = R - wn;
    GemmDesc r;  // then the lower triangle right of it
    r.m = rest; r.n = rest; r.k = w; r.alpha = -1.0; r.beta = 1.0;
    r.A = A21 + (long long)wn * lda; r.lda = lda; r.B = r.A; r.ldb = lda; r.b_trans = true;
    r.lower_only = true;
    r.C = A22 + (long long)wn * lda + wn; r.ldc = lda;
    if (la) {
      LM_CUDA_TRY(cudaEventRecord(ev_fork, st));
      LM_CUDA_TRY(cudaStreamWaitEvent(aux, ev_fork, 0));
      LM_TRY(factor_column(j0 + w, aux));
      LM_CUDA_TRY(cudaEventRecord(ev_join, aux));
      if (rest > 0) {
        r.sched = ctx_status(c) + 2;
        r.keep_sms = kLookaheadSms;
        LM_TRY(dgemm(c, r, st));
      }
      LM_CUDA_TRY(cudaStreamWaitEvent(st, ev_join, 0));
    } else {
      if (rest > 0) LM_TRY(dgemm(c, r, st));
      LM_TRY(factor_column(j0 + w, st));
    }
  }
  return zero_upper<double>(A, lda, n, st);
}

// luNoPivot (LU.hs:196-214) blocked: right-looking with 128-wide diagonal
// blocks, each factored without interchanges in one CTA (registers); then
// U12 = inv(L11) A12 and L21 = A21 inv(U11) as products with the blocks'
// inverses on the DMMA GEMM (the reference's precondition, e.g. diagonal
// dominance, keeps the diagonal blocks well conditioned), and
// A22 -= L21 U12.  A zero pivot is recorded in status[1] and, as in the
// reference, the division by it still happens.
int dgetrf_nopiv(Ctx& c, int n, double* A, long long lda, cudaStream_t st) {
  void* ws = nullptr;
  const size_t blk = (size_t)kNB * kNB;
  LM_TRY(ctx_workspace(c, 1, sizeof(double) * (3 * blk + (size_t)n * kNB), &ws));
  double* Linv = static_cast<double*>(ws);
  double* Ut = Linv + blk;
  double* Uinv = Ut + blk;
  double* W21 = Uinv + blk;
  for (int j0 = 0; j0 < n; j0 += kNB) {
    const int w = std::min(kNB, n - j0);
    const int R = n - j0 - w;
    double* A11 = A + (long long)j0 * lda + j0;
    {
      Prof p(c, kPhasePanel, 2.0 / 3.0 * w * w * w, 16.0 * w * w, st);
      LM_TRY(lu_nopiv_block(A11, lda, w, j0, ctx_status(c), st));
    }
    if (R <= 0) break;
    double* A12 = A11 + w;
    double* A21 = A11 + (long long)w * lda;
    LM_TRY(trsm_unit_lower_gemm(c, A11, lda, w, A12, lda, R, Linv, W21, st));
    {
      Prof p(c, kPhaseTrsm, (double)w * w * w / 3.0, 24.0 * (double)w * w, st);
      LM_TRY(transpose_block(Ut, kNB, A11, lda, w, st));
      LM_TRY(tri_inv_lower<double>(Ut, kNB, w, false, Uinv, kNB, nullptr, st));
    }
    {
      Prof p(c, kPhaseOther, 0.0, 16.0 * R * w, st);
      LM_TRY(copy2d<double>(W21, kNB, A21, lda, R, w, st));
    }
    GemmDesc t;  // L21 = A21 inv(U11) = W21 (inv(U11^T))^T
    t.m = R; t.n = w; t.k = w; t.alpha = 1.0; t.beta = 0.0;
    t.A = W21; t.lda = kNB; t.B = Uinv; t.ldb = kNB; t.b_trans = true;
    t.C = A21; t.ldc = lda;
    LM_TRY(dgemm(c, t, st));
    GemmDesc d;  // A22 -= L21 U12
    d.m = R; d.n = R; d.k = w; d.alpha = -1.0; d.beta = 1.0;
    d.A = A21; d.lda = lda; d.B = A12; d.ldb = lda;
    d.C = A21 + w; d.ldc = lda;
    LM_TRY(dgemm(c, d, st));
  }
  return LM_OK;
}

namespace {

// Copy to even-stride, 16-byte aligned buffers when the caller's are not
// (TMA row alignment); returns the buffers to use.  With `perm_ints` the
// workspace also holds the right-hand side's interchanges: that many ints,
// then n x nrhs doubles.
struct SolveBufs {
  const double* M;
  long long ldm;
  double* X;
  long long ldx;
  bool copied_x;
  int* perm;
  double* W;
};

int solve_bufs(Ctx& c, int n, int nrhs, const double* M, long long ldm, double* B, long long ldb, int perm_ints,
               SolveBufs& sb, cudaStream_t st) {
  sb.M = M; sb.ldm = ldm; sb.X = B; sb.ldx = ldb; sb.copied_x = false; sb.perm = nullptr; sb.W = nullptr;
  const bool m_ok = !(reinterpret_cast<uintptr_t>(M) & 15) && !(ldm & 1);
  const bool x_ok = !(reinterpret_cast<uintptr_t>(B) & 15) && !(ldb & 1);
  const long long ldm2 = m_ok ? 0 : (n + 7) / 8 * 8;
  const long long ldx2 = x_ok ? 0 : (nrhs + 7) / 8 * 8;
  const size_t perm_doubles = (size_t)(perm_ints + 7) / 8 * 4;
  const size_t bytes = sizeof(double) * ((size_t)n * ldm2 + (size_t)n * ldx2 +
                                         (perm_ints ? perm_doubles + (size_t)n * nrhs : 0));
  if (bytes == 0) return LM_OK;
  void* ws = nullptr;
  LM_TRY(ctx_workspace(c, 2, bytes, &ws));
  double* p = static_cast<double*>(ws);
  if (!m_ok) {
    LM_TRY(copy2d<double>(p, ldm2, M, ldm, n, n, st));
    sb.M = p; sb.ldm = ldm2;
    p += (size_t)n * ldm2;
  }
  if (!x_ok) {
    LM_TRY(copy2d<double>(p, ldx2, B, ldb, n, nrhs, st));
    sb.X = p; sb.ldx = ldx2; sb.copied_x = true;
    p += (size_t)n * ldx2;
  }
  if (perm_ints) {
    sb.perm = reinterpret_cast<int*>(p);
    sb.W = p + perm_doubles;
  }
  return LM_OK;
}

// Forward substitution with the lower triangle of M (unit or not), blocked.
int forward_blocked(Ctx& c, int n, int nrhs, const double* M, long long ldm, bool unit, double* X,
                    long long ldx, cudaStream_t st) {
  for (int i0 = 0; i0 < n; i0 += kNB) {
    const int w = std::min(kNB, n - i0);
    const double* Mii = M + (long long)i0 * ldm + i0;
    {
      Prof p(c, kPhaseTrsm, (double)w * w * nrhs, 8.0 * ((double)w * w / 2 + 2.0 * w * nrhs), st);
      LM_TRY(trsm_left(Mii, ldm, w, true, unit, false, X + (long long)i0 * ldx, ldx, nrhs, st));
    }
    if (i0 + w < n) {
      GemmDesc d;
      d.m = n - i0 - w; d.n = nrhs; d.k = w; d.alpha = -1.0; d.beta = 1.0;
      d.A = Mii + (long long)w * ldm; d.lda = ldm;
      d.B = X + (long long)i0 * ldx; d.ldb = ldx;
      d.C = X + (long long)(i0 + w) * ldx; d.ldc = ldx;
      LM_TRY(dgemm(c, d, st));
    }
  }
  return LM_OK;
}

}  // namespace

int dgetrs(Ctx& c, int n, int nrhs, const double* LU, long long lda, const int* ipiv, double* B,
           long long ldb, cudaStream_t st) {
  if (nrhs <= 4) {
    // few right-hand sides: P b, then one persistent launch per direction
    void* ws = nullptr;
    const size_t sync_bytes = trsv_sync_bytes<double>(n, nrhs);
    LM_TRY(ctx_workspace(c, 2, sync_bytes + sizeof(double) * (size_t)n * nrhs, &ws));
    {
      Prof p(c, kPhaseSwap, 0.0, 32.0 * n * nrhs, st);
      LM_TRY(laswp_narrow<double>(B, ldb, n, nrhs, ipiv, reinterpret_cast<double*>(static_cast<char*>(ws) + sync_bytes),
                                  ctx_status(c), st));
    }
    Prof p(c, kPhaseTrsm, 2.0 * n * n * nrhs, 8.0 * n * n, st);
    return trsv_lu<double>(LU, lda, n, nrhs, nullptr, nullptr, B, ldb, ws, ctx_status(c), st);
  }
  SolveBufs sb;
  LM_TRY(solve_bufs(c, n, nrhs, LU, lda, B, ldb, n, sb, st));
  // P b (applyPivotsForward, LU.hs:493-507): the swaps composed once, then a
  // gather (n = 8192, 64 columns: 2.2 ms as 64 launches of 128 swaps each, 0.12 ms
  // now)
  {
    Prof p(c, kPhaseSwap, 0.0, 32.0 * n * nrhs, st);
    LM_TRY(perm_from_swaps(ipiv, n, sb.perm, ctx_status(c), st));
    LM_TRY(laswp_perm<double>(sb.X, sb.ldx, n, nrhs, sb.perm, sb.W, st));
  }
  LM_TRY(forward_blocked(c, n, nrhs, sb.M, sb.ldm, true, sb.X, sb.ldx, st));
  const int nblk = (n + kNB - 1) / kNB;
  for (int b = nblk - 1; b >= 0; --b) {
    const int i0 = b * kNB;
    const int w = std::min(kNB, n - i0);
    const double* Uii = sb.M + (long long)i0 * sb.ldm + i0;
    {
      Prof p(c, kPhaseTrsm, (double)w * w * nrhs, 8.0 * ((double)w * w / 2 + 2.0 * w * nrhs), st);
      LM_TRY(trsm_left(Uii, sb.ldm, w, false, false, false, sb.X + (long long)i0 * sb.ldx, sb.ldx, nrhs,
                               st));
    }
    if (i0 > 0) {
      GemmDesc d;
      d.m = i0; d.n = nrhs; d.k = w; d.alpha = -1.0; d.beta = 1.0;
      d.A = sb.M + i0; d.lda = sb.ldm;
      d.B = sb.X + (long long)i0 * sb.ldx; d.ldb = sb.ldx;
      d.C = sb.X; d.ldc = sb.ldx;
      LM_TRY(dgemm(c, d, st));
    }
  }
  if (sb.copied_x) LM_TRY(copy2d<double>(B, ldb, sb.X, sb.ldx, n, nrhs, st));
  return LM_OK;
}

int dpotrs(Ctx& c, int n, int nrhs, const double* G, long long lda, double* B, long long ldb,
           cudaStream_t st) {
  if (nrhs <= 4) {
    // few right-hand sides: G packed with G^T above the diagonal, then one
    // persistent launch per direction (the same kernels as dgetrs, with the
    // stored diagonal of G)
    const long long ldp = (n + 7) / 8 * 8;
    void* ws = nullptr;
    const size_t sync_bytes = trsv_sync_bytes<double>(n, nrhs);
    LM_TRY(ctx_workspace(c, 2, sync_bytes + sizeof(double) * (size_t)n * ldp, &ws));
    double* P = reinterpret_cast<double*>(static_cast<char*>(ws) + sync_bytes);
    {
      Prof p(c, kPhaseOther, 0.0, 16.0 * n * n, st);
      LM_TRY(pack_lower_sym(P, ldp, G, lda, n, st));
    }
    Prof p(c, kPhaseTrsm, 2.0 * n * n * nrhs, 8.0 * n * n, st);
    return trsv_lu<double>(P, ldp, n, nrhs, nullptr, nullptr, B, ldb, ws, ctx_status(c), st, nullptr, true, false);
  }
  SolveBufs sb;
  LM_TRY(solve_bufs(c, n, nrhs, G, lda, B, ldb, 0, sb, st));
  LM_TRY(forward_blocked(c, n, nrhs, sb.M, sb.ldm, false, sb.X, sb.ldx, st));
  // G^T x = y, bottom-up; the off-diagonal update uses G's row block transposed.
  const int nblk = (n + kNB - 1) / kNB;
  for (int b = nblk - 1; b >= 0; --b) {
    const int i0 = b * kNB;
    const int w = std::min(kNB, n - i0);
    const double* Gii = sb.M + (long long)i0 * sb.ldm + i0;
    {
      Prof p(c, kPhaseTrsm, (double)w * w * nrhs, 8.0 * ((double)w * w / 2 + 2.0 * w * nrhs), st);
      LM_TRY(trsm_left(Gii, sb.ldm, w, true, false, true, sb.X + (long long)i0 * sb.ldx, sb.ldx, nrhs,
                               st));
    }
    if (i0 > 0) {
      GemmDesc d;
      d.m = i0; d.n = nrhs; d.k = w; d.alpha = -1.0; d.beta = 1.0;
      d.A = sb.M + (long long)i0 * sb.ldm; d.lda = sb.ldm; d.a_trans = true;
      d.B = sb.X + (long long)i0 * sb.ldx; d.ldb = sb.ldx;
      d.C = sb.X; d.ldc = sb.ldx;
      LM_TRY(dgemm(c, d, st));
    }
  }
  if (sb.copied_x) LM_TRY(copy2d<double>(B, ldb, sb.X, sb.ldx, n, nrhs, st));
  return LM_OK;
}

}  // namespace lm
