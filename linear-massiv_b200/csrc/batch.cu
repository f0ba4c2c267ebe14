// Batched uneven-size factor + solve in one persistent launch.
//
// Thousands of independent systems A_i X_i = B_i (n_i <= 256, nrhs_i <= 16),
// each general (LU with partial pivoting: luSolveP, LU.hs:265-357, pivot rule
// of rawPivotSearch K.hs:1541-1556) or SPD (Cholesky: choleskySolveP,
// Chol.hs:241-321), are solved by one persistent grid.  Each CTA takes the
// next instance from a ticket counter (the host orders the instances by
// decreasing cost, longest-processing-time first), factors it in a private
// workspace region that stays L2-resident (at most 512 KB per instance), and
// solves.  Inside an instance everything is CTA-local — no grid-wide
// synchronisation and no spin-waits.  An instance is a chain of columns, so
// what bounds it is the latency of a column, and what fills the SM is how many
// instances run beside each other: CTAs of 128 threads, four per SM.
//   LU     : right-looking, panels of 16 columns held in registers, one thread
//            per row that is still active (two when there are more than 128).
//            A column takes one barrier: the warps vote with redux.sync, stage
//            their candidates, and every warp votes over the four.  Rows do not
//            move: an interchange swaps two labels, and the factor is put in
//            order once at the end.  U12 by per-thread columns; the trailing
//            update on 32 x 32 warp tiles (DMMA for FP64, FFMA for FP32).
//   Cholesky: the 16 x 16 diagonal block in one warp (shuffles), the rows below
//            by one thread each, the same trailing update on the lower triangle.
//   solve  : 16-row blocks; a thread keeps its rows of the right-hand side in
//            registers, the diagonal block goes by shuffles (16 lanes per right-
//            hand side), and the block column arrives by cp.async meanwhile.
// 10,000 systems of order 8 to 256, FP64: 14.7 ms with 256-thread CTAs, panels in
// shared memory (ten shuffles, three barriers and a serial row loop per column)
// and row interchanges through L2, 9.5 ms now; 3,000 with FP32 factors and
// refinement 8.25 and 3.9 ms.  What is left is latency: a warp issues every 17
// cycles, waiting at barriers (28%: the 16 x 16 diagonal blocks and the pivot
// votes), for instructions (19%) and for fixed latencies (13%).
//
// Mixed precision (LM_PREC_FP32_IR): the factorisation and the correction
// solves run in FP32; the solution is refined in FP64 inside the same CTA —
// r = B - A X with the original FP64 A (DMMA), correction from the FP32 factors,
// X += D — until the normwise backward error max_h ||r_h|| / (||A|| ||x_h|| +
// ||b_h||) (infinity norms) is <= tol, which a column with a NaN or an infinity in
// any of these norms never is.  An instance that has not converged after max_iter
// corrections is refactored and solved in FP64 (iters = -1).
#include <algorithm>
#include <cfloat>
#include <climits>
#include <type_traits>

#include "common.cuh"
#include "internal.h"
#include "pivot.cuh"

namespace lm {

namespace {

constexpr int kBT = 128;        // threads per CTA
constexpr int kPW = 16;         // widest panel, and the substitutions' row block
constexpr int kLdP = kPW + 4;   // panel row stride: 16-byte rows, DMMA operand reads without conflicts
constexpr int kUC = 96;         // trailing-update column chunk
constexpr int kLdU = kUC + 4;
constexpr int kMaxR = BatchLimits::kMaxRhs;

__device__ __forceinline__ int tid_() { return threadIdx.x; }

template <typename T>
struct PivMsg {
  typename PivKey<T>::K key;
  int label;  // position from the panel's first row, or INT_MAX: no candidate
  T rcp;      // reciprocal of the leading entry
  alignas(16) T v[kPW];
};

// Fixed scratch at the start of dynamic shared memory.
struct Fixed {
  double red[2][kBT / 32][kMaxR];  // column maxima by warp: residual, solution
  double bnorm[kMaxR];
  double anorm, be;
  int info, slot;
  int plain;  // Cholesky: the panel's quotients are divisions
  alignas(16) unsigned char msg[2 * (kBT / 32) * sizeof(PivMsg<double>)];
  unsigned char src[BatchLimits::kMaxN];  // position -> row of the workspace (and of B)
  unsigned char cur[BatchLimits::kMaxN];  // the same for the rows of the current panel
  unsigned char act[BatchLimits::kMaxN];  // panel rows that stay active, in order
  unsigned char pidx[kPW];                // panel rows that became pivots
};
constexpr size_t kFixed = (sizeof(Fixed) + 15) / 16 * 16;

__device__ __forceinline__ void sub_bar(int nthreads) {
  asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
}
template <int BYTES>
__device__ __forceinline__ void cp_async_elem(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A row of kPW elements between registers and 16-byte aligned shared memory.
template <typename T>
__device__ __forceinline__ void row_ld(T (&x)[kPW], const T* p) {
  constexpr int V = 16 / (int)sizeof(T);
#pragma unroll
  for (int c = 0; c < kPW; c += V) {
    T v[V];
    *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(p + c);
#pragma unroll
    for (int e = 0; e < V; ++e) x[c + e] = v[e];
  }
}
template <typename T>
__device__ __forceinline__ void row_st(T* p, const T (&x)[kPW]) {
  constexpr int V = 16 / (int)sizeof(T);
#pragma unroll
  for (int c = 0; c < kPW; c += V) {
    T v[V];
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = x[c + e];
    *reinterpret_cast<uint4*>(p + c) = *reinterpret_cast<const uint4*>(v);
  }
}

// ---------------------------------------------------------------------------
// Factorisations of one instance (F: n x n, ld n, in global memory).
// ---------------------------------------------------------------------------

// C -= L U on one 32 x 32 warp tile at (rb, cb).  prow(q): row q of L (w columns,
// shared); frow(q): row q of C; u(k, c): element of U (shared).  Only rows < M,
// columns < Nc and, with LOWER, columns <= row are stored; operand indices past
// the edges are clamped.  The MMA's column pairs are mapped to columns c, c + 4,
// so that a quad covers 32 contiguous bytes of C.
template <typename T, bool LOWER, typename PRow, typename FRow, typename U>
__device__ __forceinline__ void update_tile(int rb, int cb, int M, int Nc, int w, PRow prow, FRow frow, U u) {
  const int lane = tid_() & 31;
  const int g = lane >> 2, t = lane & 3;
  if constexpr (sizeof(T) == 8) {
    const double* pr[4];
    double* fr[4];
    double acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int q = rb + i * 8 + g;
      pr[i] = prow(min(q, M - 1)) + t;
      fr[i] = frow(min(q, M - 1));
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c = cb + ni * 8 + t + 4 * e;
          acc[i >> 1][ni][(i & 1) * 2 + e] = q < M && c < Nc && (!LOWER || c <= q) ? fr[i][c] : 0.0;
        }
    }
    const int gc = (g >> 1) + 4 * (g & 1);
    int uc[4];
#pragma unroll
    for (int ni = 0; ni < 4; ++ni) uc[ni] = min(cb + ni * 8 + gc, Nc - 1);
    __syncwarp();
#pragma unroll 2
    for (int k = 0; k < w; k += 4) {
      double b[4];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) b[ni] = u(k + t, uc[ni]);
#pragma unroll
      for (int mi = 0; mi < 2; ++mi) {
        const double a0 = -pr[2 * mi][k], a1 = -pr[2 * mi + 1][k];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) dmma_16x8x4(acc[mi][ni], a0, a1, b[ni]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int q = rb + i * 8 + g;
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c = cb + ni * 8 + t + 4 * e;
          if (q < M && c < Nc && (!LOWER || c <= q)) fr[i][c] = acc[i >> 1][ni][(i & 1) * 2 + e];
        }
    }
  } else {
    const float* pr[4];
    float* fr[4];
    float acc[4][8];
    int uc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) uc[e] = min(cb + t + 4 * e, Nc - 1);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int q = rb + i * 8 + g;
      pr[i] = prow(min(q, M - 1));
      fr[i] = frow(min(q, M - 1));
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int c = cb + t + 4 * e;
        acc[i][e] = q < M && c < Nc && (!LOWER || c <= q) ? fr[i][c] : 0.f;
      }
    }
#pragma unroll 4
    for (int k = 0; k < w; ++k) {
      float a[4], b[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = pr[i][k];
#pragma unroll
      for (int e = 0; e < 8; ++e) b[e] = u(k, uc[e]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[i][e] = fmaf(-a[i], b[e], acc[i][e]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int q = rb + i * 8 + g;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int c = cb + t + 4 * e;
        if (q < M && c < Nc && (!LOWER || c <= q)) fr[i][c] = acc[i][e];
      }
    }
  }
}

// One panel of LU: the M active rows of P (w columns; panel row i is the active
// row at position k0 + i) factored in registers, RPT rows per thread.  On exit
// P holds the multipliers and U rows in place, src[k0 ..] the new order, pidx the
// pivots' panel rows and act those of the others, in order.
template <typename T, int RPT>
__device__ __forceinline__ void lu_panel(T* P, int M, int w, int k0, int* ipiv, Fixed* fx) {
  using Key = typename PivKey<T>::K;
  using Msg = PivMsg<T>;
  constexpr int V = 16 / (int)sizeof(T);
  const int lane = tid_() & 31, warp = tid_() >> 5;
  const int nwa = RPT > 1 ? kBT / 32 : (M + 31) / 32;  // warps with rows
  if (warp >= nwa) return;
  Msg* wm = reinterpret_cast<Msg*>(fx->msg);
  T y[RPT][kPW];  // rotated: slot 0 is the current column
  int lr[RPT];    // position from k0, -1: no row here
  int phys[RPT];
#pragma unroll
  for (int s = 0; s < RPT; ++s) {
    const int i = s * kBT + tid_();
    lr[s] = i < M ? i : -1;
    phys[s] = i < M ? fx->cur[i] : 0;
    row_ld<T>(y[s], P + min(i, M - 1) * kLdP);
  }
  Key bk = 0;
  int bi = INT_MAX, bs = 0;
  T xb = T(1);
  auto consider = [&](int s, T v, int J) {
    Key k = PivKey<T>::of(v);
    if (k == 0 && lr[s] == J && v != v) k = PivKey<T>::kForced;
    if (RPT == 1 || bi == INT_MAX || k > bk || (k == bk && lr[s] < bi)) { bk = k; bi = lr[s]; bs = s; xb = v; }
  };
#pragma unroll
  for (int s = 0; s < RPT; ++s)
    if (lr[s] >= 0) consider(s, y[s][0], 0);
#pragma unroll 1
  for (int j = 0; j < w; ++j) {
    Msg* ms = wm + (j & 1) * (kBT / 32);
    const T rc = PivKey<T>::rcp(xb);
    const int wl = warp_winner(bk, bi);
    if (lane == wl) {
      Msg* out = ms + warp;
      out->key = bk;
      out->label = bi;
      out->rcp = rc;
#pragma unroll
      for (int s = 0; s < RPT; ++s)
        if (s == bs) row_st<T>(out->v, y[s]);
    }
    int wo = 0;
    if (nwa > 1) {
      sub_bar(nwa * 32);
      wo = warp_winner(lane < nwa ? ms[lane].key : Key(0), lane < nwa ? ms[lane].label : INT_MAX);
      if (wo >= nwa) wo = 0;
    } else {
      __syncwarp();
    }
    const Msg* win = ms + wo;
    const int p = win->label == INT_MAX ? j : win->label;  // (row j itself is always a candidate)
    const T rcp = win->rcp, piv = win->v[0];
    const bool safe = PivKey<T>::safe(piv);
    if (tid_() == 0) {
      ipiv[k0 + j] = k0 + p;
      if (piv == T(0) && fx->info == 0) fx->info = k0 + j + 1;
    }
    bk = 0;
    bi = INT_MAX;
#pragma unroll
    for (int s = 0; s < RPT; ++s) {
      if (lr[s] == p) lr[s] = j;
      else if (lr[s] == j) lr[s] = p;
      T m = y[s][0];
      if (lr[s] > j) {
        m = div_by(y[s][0], piv, rcp);
        if (!safe) m = y[s][0] / piv;
#pragma unroll
        for (int c = 0; c < kPW; c += V) {
          if (c < kPW - j) {  // (the slots past it hold finished multipliers)
            T u[V];
            *reinterpret_cast<uint4*>(u) = *reinterpret_cast<const uint4*>(win->v + c);
#pragma unroll
            for (int e = 0; e < V; ++e)
              if (c + e > 0 && c + e < kPW - j) y[s][c + e] = fma(-m, u[e], y[s][c + e]);
          }
        }
        if (j + 1 < w) consider(s, y[s][1], j + 1);
      }
      __syncwarp();  // rejoin at once: split, the warp would run all that follows twice
#pragma unroll
      for (int c = 0; c + 1 < kPW; ++c) y[s][c] = y[s][c + 1];
      y[s][kPW - 1] = m;
    }
  }
#pragma unroll 1
  for (int j = w; j < kPW; ++j)
#pragma unroll
    for (int s = 0; s < RPT; ++s) {
      const T m = y[s][0];
#pragma unroll
      for (int c = 0; c + 1 < kPW; ++c) y[s][c] = y[s][c + 1];
      y[s][kPW - 1] = m;
    }
#pragma unroll
  for (int s = 0; s < RPT; ++s) {
    const int i = s * kBT + tid_();
    if (lr[s] >= 0) {
      row_st<T>(P + i * kLdP, y[s]);
      fx->src[k0 + lr[s]] = (unsigned char)phys[s];
      if (lr[s] < w) fx->pidx[lr[s]] = (unsigned char)i;
      else fx->act[lr[s] - w] = (unsigned char)i;
    }
  }
}

// LU with partial pivoting in place; ipiv (global, n) receives the swap list
// (0-based), fx->src the composed order, fx->info the LAPACK-style info (first
// zero pivot + 1, or 0).  nb: the panel width (at most kPW is used).
template <typename T>
__device__ void lu_factor(T* F, int n, int nb, int* ipiv, unsigned char* region, Fixed* fx) {
  T* P = reinterpret_cast<T*>(region);                                // [n][kLdP]
  T* Us = P + (size_t)n * kLdP;                                       // [kPW][kLdU]
  nb = min(nb, kPW);
  const int pc = tid_() & (kPW - 1), pr0 = tid_() / kPW;  // panel column and first row in a staged copy
  constexpr int PR = kBT / kPW;
  for (int i = tid_(); i < n; i += kBT) fx->src[i] = (unsigned char)i;
  if (tid_() == 0) fx->info = 0;
  __syncthreads();
  for (int k0 = 0; k0 < n; k0 += nb) {
    const int w = min(nb, n - k0), M = n - k0, M2 = M - w;
    for (int i = tid_(); i < M; i += kBT) fx->cur[i] = fx->src[k0 + i];
    __syncthreads();
    for (int i = pr0; i < M; i += PR) {
      if (pc < w) cp_async_elem<sizeof(T)>(P + i * kLdP + pc, F + fx->cur[i] * n + k0 + pc);
      else P[i * kLdP + pc] = T(0);
    }
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    if (M > kBT) lu_panel<T, 2>(P, M, w, k0, ipiv, fx);
    else lu_panel<T, 1>(P, M, w, k0, ipiv, fx);
    __syncthreads();
#pragma unroll 4
    for (int i = pr0; i < M; i += PR)
      if (pc < w) F[fx->cur[i] * n + k0 + pc] = P[i * kLdP + pc];
    // (M2 > 0 only where w = nb, a multiple of 4)
    for (int c0 = 0; c0 < M2; c0 += kUC) {
      const int cw = min(kUC, M2 - c0);
      if (tid_() < cw) {
        // U12 = L11^-1 A12 (unit lower), a column per thread
        T u[kPW];
#pragma unroll
        for (int i = 0; i < kPW; ++i) u[i] = i < w ? F[fx->cur[fx->pidx[i]] * n + k0 + w + c0 + tid_()] : T(0);
#pragma unroll
        for (int i = 1; i < kPW; ++i)
          if (i < w) {
            const T* l = P + fx->pidx[i] * kLdP;
#pragma unroll
            for (int q = 0; q < i; ++q) u[i] = fma(-l[q], u[q], u[i]);
          }
#pragma unroll
        for (int i = 0; i < kPW; ++i)
          if (i < w) {
            F[fx->cur[fx->pidx[i]] * n + k0 + w + c0 + tid_()] = u[i];
            Us[i * kLdU + tid_()] = u[i];
          }
      }
      __syncthreads();
      const int tc = (cw + 31) / 32, tiles = ((M2 + 31) / 32) * tc;
      for (int t = tid_() >> 5; t < tiles; t += kBT / 32)
        update_tile<T, false>(
            (t / tc) * 32, (t % tc) * 32, M2, cw, w, [&](int q) { return P + fx->act[q] * kLdP; },
            [&](int q) { return F + fx->cur[fx->act[q]] * n + k0 + w + c0; },
            [&](int k, int c) { return Us[k * kLdU + c]; });
      __syncthreads();
    }
  }
  // the rows into their final order, 16 columns at a time
  __syncthreads();
  for (int c0 = 0; c0 < n; c0 += kPW) {
    for (int i = pr0; i < n; i += PR)
      if (c0 + pc < n) cp_async_elem<sizeof(T)>(P + i * kLdP + pc, F + fx->src[i] * n + c0 + pc);
    cp_commit();
    cp_wait<0>();
    __syncthreads();
#pragma unroll 4
    for (int i = pr0; i < n; i += PR)
      if (c0 + pc < n) F[i * n + c0 + pc] = P[i * kLdP + pc];
    __syncthreads();
  }
}

// The w x w diagonal block (w <= 16) at the top of P by one warp, lane = row; Fd
// is the block in global memory, still as it was; rd receives the reciprocals of
// the diagonal.  The columns are a rolled loop over rotating registers, each
// finished one going to P at once: unrolled, the 16 steps were the largest piece of
// code of the kernel, ran whole for the smallest block, and waited for instructions.
// The last eight columns (all of a block of up to eight) shuffle half as much.
// 148 SPD systems of order 4, 16, 32, 64: 21, 23, 39, 68 us unrolled, 13, 17, 31,
// 56 us now (11, 21, 36, 70 us with a barrier per column).
template <typename T>
__device__ __forceinline__ void chol_diag(T* P, const T* Fd, int n, int w, int k0, T* rd, Fixed* fx) {
  const int lane = tid_() & 31;
  T a[kPW];  // slot 0 is the current column
#pragma unroll
  for (int c = 0; c < kPW; ++c) a[c] = c <= lane && lane < w ? P[lane * kLdP + c] : T(0);
  bool ok = true;
  T rj = T(0);
  int j = 0;
  auto column = [&](auto live) {  // slots in use
    constexpr int N = decltype(live)::value;
    __syncwarp();  // a split warp would serialise the shuffles
    const T d = __shfl_sync(0xffffffffu, a[0], j);
    if (lane == 0 && !(d > T(0)) && fx->info == 0) fx->info = k0 + j + 1;
    __syncwarp();
    const T s = sqrt(d), r = PivKey<T>::rcp(s);
    ok = ok && PivKey<T>::safe(s) && (lane <= j || lane >= w || quotient_safe(a[0]));
    const T q = div_by(a[0], s, r), l = lane == j ? s : q;
    rj = lane == j ? r : rj;
    if (lane >= j && lane < w) P[lane * kLdP + j] = l;
    __syncwarp();
    // (rows above the entry, and lanes that hold none, are left alone: lane < j + c)
#pragma unroll
    for (int c = 1; c < N; ++c) {
      const T lc = __shfl_sync(0xffffffffu, l, j + c);
      a[c - 1] = lane >= j + c ? fma(-l, lc, a[c]) : a[c];
    }
  };
  if (w > kPW / 2)
#pragma unroll 1
    for (; j < kPW / 2; ++j) column(std::integral_constant<int, kPW>());
#pragma unroll 1
  for (; j < w; ++j) column(std::integral_constant<int, kPW / 2>());
  // a quotient by reciprocal was not safe: the same steps again with divisions
  if (!__all_sync(0xffffffffu, ok)) {
    if (lane == 0 && fx->info > k0) fx->info = 0;
    for (int c = 0; c <= lane && lane < w; ++c) P[lane * kLdP + c] = Fd[lane * n + c];
    __syncwarp();
    for (j = 0; j < w; ++j) {
      const T d = P[j * kLdP + j], s = sqrt(d);
      if (lane == 0 && !(d > T(0)) && fx->info == 0) fx->info = k0 + j + 1;
      __syncwarp();
      T l = s;
      if (lane > j && lane < w) l = P[lane * kLdP + j] / s;
      if (lane >= j && lane < w) P[lane * kLdP + j] = l;
      __syncwarp();
      for (int c = j + 1; c < w; ++c)
        if (lane >= c && lane < w) P[lane * kLdP + c] = fma(-l, P[c * kLdP + j], P[lane * kLdP + c]);
      __syncwarp();
    }
    if (lane == 0) fx->plain = 1;
    return;
  }
  if (lane == 0) fx->plain = 0;
  if (lane < kPW) rd[lane] = rj;
}

// Cholesky (lower) in place: G in the lower triangle, the strict upper
// triangle left as it was.  fx->info: the first non-positive pivot + 1, or 0.
template <typename T>
__device__ void chol_factor(T* F, int n, int nb, unsigned char* region, Fixed* fx) {
  T* P = reinterpret_cast<T*>(region);  // [n][kLdP]
  T* rd = P + (size_t)n * kLdP;         // [kPW]
  nb = min(nb, kPW);
  const int pc = tid_() & (kPW - 1), pr0 = tid_() / kPW;
  constexpr int PR = kBT / kPW;
  if (tid_() == 0) fx->info = 0;
  for (int k0 = 0; k0 < n; k0 += nb) {
    const int w = min(nb, n - k0), M = n - k0, M2 = M - w;
    for (int i = pr0; i < M; i += PR) {
      if (pc < w) cp_async_elem<sizeof(T)>(P + i * kLdP + pc, F + (k0 + i) * n + k0 + pc);
      else P[i * kLdP + pc] = T(0);
    }
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    // (not the same warp in every CTA of an SM: those share a scheduler)
    if ((tid_() >> 5) == (fx->slot & (kBT / 32 - 1))) chol_diag<T>(P, F + k0 * n + k0, n, w, k0, rd, fx);
    __syncthreads();
    for (int i = w + tid_(); i < M; i += kBT) {
      // row i: x L11^T = a, by columns of L11
      T x[kPW];
      row_ld<T>(x, P + i * kLdP);
      bool ok = fx->plain == 0;
#pragma unroll
      for (int k = 0; k < kPW; ++k)
        if (k < w) {
          ok = ok && quotient_safe(x[k]);
          x[k] = div_by(x[k], P[k * kLdP + k], rd[k]);
#pragma unroll
          for (int j = k + 1; j < kPW; ++j)
            if (j < w) x[j] = fma(-x[k], P[j * kLdP + k], x[j]);
        }
      if (!ok) {
        for (int k = 0; k < w; ++k) {
          const T q = P[i * kLdP + k] / P[k * kLdP + k];
          P[i * kLdP + k] = q;
          for (int j = k + 1; j < w; ++j) P[i * kLdP + j] = fma(-q, P[j * kLdP + k], P[i * kLdP + j]);
        }
        continue;
      }
      row_st<T>(P + i * kLdP, x);
    }
    __syncthreads();
#pragma unroll 4
    for (int i = pr0; i < M; i += PR)
      if (pc < w && (i >= w || pc <= i)) F[(k0 + i) * n + k0 + pc] = P[i * kLdP + pc];
    if (M2 > 0) {
      const int tr = (M2 + 31) / 32, tiles = tr * (tr + 1) / 2;
      int ti = 0, tj = tid_() >> 5;  // tile t of the lower triangle, row by row
      for (int t = tid_() >> 5; t < tiles; t += kBT / 32, tj += kBT / 32) {
        while (tj > ti) tj -= ++ti;
        update_tile<T, true>(
            ti * 32, tj * 32, M2, M2, w, [&](int q) { return P + (w + q) * kLdP; },
            [&](int q) { return F + (k0 + w + q) * n + k0 + w; },
            [&](int k, int c) { return P[(w + c) * kLdP + k]; });
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Triangular solves of the n x r right-hand side held in registers (thread t:
// rows t and t + 128, NR >= r columns, zeros past r and n), with the factor in F.
//   mode 0: unit lower (LU's L)      forward
//   mode 1: upper (LU's U)           backward
//   mode 2: lower G (Cholesky)       forward
//   mode 3: upper G^T (Cholesky)     backward, T(i, k) = G(k, i)
// ---------------------------------------------------------------------------
template <typename T, int NR, int mode>
__device__ __forceinline__ void tri_solve(const T* F, int n, T (&y)[2][NR], int r, unsigned char* region) {
  constexpr int LDT = kPW + 1, LDX = NR + 4;
  T* S = reinterpret_cast<T*>(region);  // [n][kLdP] the block column
  T* X = S + (size_t)n * kLdP;          // [kPW][LDX] the block of the right-hand side
  T* Tb = X + kPW * LDX;                // [kPW][LDT] the diagonal block
  constexpr bool fwd = (mode == 0 || mode == 2);
  constexpr bool unit = (mode == 0);
  const int nblk = (n + kPW - 1) / kPW;
  const int l = tid_() & (kPW - 1), g = tid_() / kPW;
  constexpr int PR = kBT / kPW;
  for (int b = 0; b < nblk; ++b) {
    const int i0 = (fwd ? b : nblk - 1 - b) * kPW, bw = min(kPW, n - i0);
    for (int rr = g; rr < bw; rr += PR)
      if (l < bw)
        cp_async_elem<sizeof(T)>(mode == 3 ? Tb + l * LDT + rr : Tb + rr * LDT + l, F + (i0 + rr) * n + i0 + l);
    cp_commit();
    const int q0 = fwd ? i0 + bw : 0, q1 = fwd ? n : i0;  // rows still to be solved
    if (mode != 3) {
      for (int i = q0 + g; i < q1; i += PR)
        if (l < bw) cp_async_elem<sizeof(T)>(S + i * kLdP + l, F + i * n + i0 + l);
    } else {  // (by columns: entry (i, k) at k n + i)
      for (int k = tid_() >> 5; k < bw; k += kBT / 32)
        for (int i = tid_() & 31; i < q1; i += 32) cp_async_elem<sizeof(T)>(S + k * n + i, F + (i0 + k) * n + i);
    }
    cp_commit();
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int row = s * kBT + tid_();
      if (row >= i0 && row < i0 + bw)
#pragma unroll
        for (int h = 0; h < NR; ++h) X[(row - i0) * LDX + h] = y[s][h];
    }
    cp_wait<1>();
    __syncthreads();
    for (int h0 = 0; h0 < r; h0 += PR) {
      const int h = h0 + g;  // 16 lanes per right-hand side, lane = row
      const bool in = l < bw;
      T x = in ? X[l * LDX + h] : T(0);
      const T d = unit || !in ? T(1) : Tb[l * LDT + l];
      const T rd = unit || !in ? T(1) : T(1) / d;
      x = tri_sweep<T, kPW>(x, Tb + l * LDT, d, rd, l, bw, fwd, unit);
      if (in) X[l * LDX + h] = x;
    }
    cp_wait<0>();
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int row = s * kBT + tid_();
      if (row >= i0 && row < i0 + bw) {
#pragma unroll
        for (int h = 0; h < NR; ++h) y[s][h] = X[(row - i0) * LDX + h];
      } else if (row >= q0 && row < q1) {
#pragma unroll 4
        for (int k = 0; k < bw; ++k) {
          const T a = mode == 3 ? S[k * n + row] : S[row * kLdP + k];
#pragma unroll
          for (int h = 0; h < NR; ++h) y[s][h] = fma(-a, X[k * LDX + h], y[s][h]);
        }
      }
    }
    __syncthreads();
  }
}

// load(row, h) gives the right-hand side (for LU of the row that the
// interchanges bring there), store(i, h, x) takes the solution.
template <typename T, int NR, typename Load, typename Store>
__device__ __noinline__ void solve_nr(const T* F, int n, int kind, const Fixed* fx, int r, unsigned char* region,
                                      Load load, Store store) {
  T y[2][NR];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int row = s * kBT + tid_();
    const int from = row < n ? (kind == LM_BATCH_GENERAL ? fx->src[row] : row) : 0;
#pragma unroll
    for (int h = 0; h < NR; ++h) y[s][h] = row < n && h < r ? load(from, h) : T(0);
  }
  __syncthreads();  // (load may read the region that the solves stage into)
  if (kind == LM_BATCH_GENERAL) {
    tri_solve<T, NR, 0>(F, n, y, r, region);
    tri_solve<T, NR, 1>(F, n, y, r, region);
  } else {
    tri_solve<T, NR, 2>(F, n, y, r, region);
    tri_solve<T, NR, 3>(F, n, y, r, region);
  }
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int row = s * kBT + tid_();
    if (row < n)
#pragma unroll
      for (int h = 0; h < NR; ++h)
        if (h < r) store(row, h, y[s][h]);
  }
  __syncthreads();
}
template <typename T, typename Load, typename Store>
__device__ __forceinline__ void solve_factored(const T* F, int n, int kind, const Fixed* fx, int r,
                                               unsigned char* region, Load load, Store store) {
  if (r <= 8) solve_nr<T, 8>(F, n, kind, fx, r, region, load, store);
  else solve_nr<T, kMaxR>(F, n, kind, fx, r, region, load, store);
}

// Shared-memory carve (byte offsets from the start of dynamic shared memory):
//   FP64: [Fixed][panel or block column, U12 chunk or solved block]
//   IR  : [Fixed][Xd: the FP64 solution][the same for FP32, D over it]
// whose FP64 fallback takes the FP64 layout.
constexpr int xd_ld(int rmax) { return rmax > 8 ? kMaxR + 4 : 12; }  // DMMA operand reads without conflicts
constexpr size_t region_bytes(int nmax, size_t elem) { return ((size_t)nmax * kLdP + kPW * kLdU) * elem; }
static_assert(kPW * (kMaxR + 4) + kPW * (kPW + 1) <= kPW * kLdU, "the solves' blocks fit the U12 chunk");
__host__ __device__ inline size_t ir_region(int nmax, int rmax) { return kFixed + (size_t)nmax * xd_ld(rmax) * 8; }

// Input loads: L2-only (ld.global.cg) for the device-resident consumer, whose
// CTAs outlive the requests they read (an arena block is reused by later
// requests, and an SM's L1 is not coherent with the copies that refill it).
template <bool CG>
__device__ __forceinline__ double ld_in(const double* p) {
  if constexpr (CG) return __ldcg(p);
  else return *p;
}

// Factor + solve one instance entirely in FP64, X to global memory.
template <bool CG = false>
__device__ __forceinline__ void run_fp64(const BatchItem& it, const BatchArgs& g, unsigned char* sm, Fixed* fx) {
  unsigned char* region = sm + kFixed;
  const int n = it.n, r = it.nrhs;
  double* F = g.F + it.f_off;
  int* ipiv = g.ipiv + it.p_off;
  // (16 loads at a time: F may alias A for all the compiler knows)
  const double* A = g.A + it.a_off;
  for (int e0 = tid_(); e0 < n * n; e0 += 16 * kBT) {
    double v[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = e0 + q * kBT < n * n ? ld_in<CG>(A + e0 + q * kBT) : 0.0;
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if (e0 + q * kBT < n * n) F[e0 + q * kBT] = v[q];
  }
  __syncthreads();
  if (it.kind == LM_BATCH_GENERAL) lu_factor<double>(F, n, it.nb, ipiv, region, fx);
  else chol_factor<double>(F, n, it.nb, region, fx);
  if (r == 0) return;
  const double* B = g.B + it.b_off;
  double* X = g.X + it.x_off;
  solve_factored<double>(
      F, n, it.kind, fx, r, region, [&](int i, int h) { return ld_in<CG>(B + i * r + h); },
      [&](int i, int h, double x) { X[i * r + h] = x; });
}

// Norms of the refinement: a NaN counts as infinity, which fmax keeps where it
// would drop the NaN.
__device__ __forceinline__ double norm_abs(double v) { return v != v ? INFINITY : fabs(v); }

// Column maxima of |get(i, h)| over n rows into red (by warp).
template <typename Get>
__device__ __forceinline__ void col_max(int n, int r, double (*red)[kMaxR], Get get) {
  const int h = tid_() & 15;
  double m = 0.0;
  if (h < r)
    for (int i = tid_() >> 4; i < n; i += kBT / 16) m = fmax(m, norm_abs(get(i, h)));
  __syncwarp();
  m = fmax(m, __shfl_xor_sync(0xffffffffu, m, 16));
  if ((tid_() & 31) < kMaxR) red[tid_() >> 5][h] = m;
}
__device__ __forceinline__ double red_max(const double (*red)[kMaxR], int h) {
  double m = red[0][h];
#pragma unroll
  for (int w = 1; w < kBT / 32; ++w) m = fmax(m, red[w][h]);
  return m;
}

// D (n x r) <- B - A X in FP64 on the tensor cores, 16 rows per warp and step,
// and the column maxima of |r| into fx->red[0].  NT: 8-column tiles.
template <int NT>
__device__ __forceinline__ void batch_residual(const double* A, const double* B, int n, int r, const double* Xd,
                                               int ldx, float* D, Fixed* fx) {
  const int lane = tid_() & 31, warp = tid_() >> 5, q = lane >> 2, t = lane & 3;
  double mx[NT][2];
#pragma unroll
  for (int ni = 0; ni < NT; ++ni) mx[ni][0] = mx[ni][1] = 0.0;
  for (int rb = warp * 16; rb < n; rb += kBT / 2) {
    double acc[NT][4];
#pragma unroll
    for (int ni = 0; ni < NT; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[ni][e] = 0.0;
    const double* a0 = A + min(rb + q, n - 1) * n;
    const double* a1 = A + min(rb + q + 8, n - 1) * n;
    __syncwarp();
#pragma unroll 4
    for (int k = 0; k < n; k += 4) {
      const bool in = k + t < n;
      const int kc = in ? k + t : 0;
      const double x0 = in ? a0[kc] : 0.0, x1 = in ? a1[kc] : 0.0;
#pragma unroll
      for (int ni = 0; ni < NT; ++ni) dmma_16x8x4(acc[ni], x0, x1, in ? Xd[kc * ldx + ni * 8 + q] : 0.0);
    }
#pragma unroll
    for (int ni = 0; ni < NT; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = rb + q + (e >> 1) * 8, h = ni * 8 + 2 * t + (e & 1);
        if (i < n && h < r) {
          const double res = B[i * r + h] - acc[ni][e];
          D[i * r + h] = (float)res;
          mx[ni][e & 1] = fmax(mx[ni][e & 1], norm_abs(res));
        }
      }
  }
  __syncwarp();
#pragma unroll
  for (int ni = 0; ni < NT; ++ni)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      double m = mx[ni][e];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (q == 0) fx->red[0][warp][ni * 8 + 2 * t + e] = m;
    }
}

// Factor in FP32, refine in FP64.  Returns the number of corrections, or -1
// when it fell back to FP64.
__device__ int run_ir(const BatchItem& it, const BatchArgs& g, unsigned char* sm, Fixed* fx, double* berr_out) {
  unsigned char* region = sm + ir_region(g.nmax, g.rmax);
  double* Xd = reinterpret_cast<double*>(sm + kFixed);
  const int ldx = xd_ld(g.rmax);
  const int n = it.n, r = it.nrhs;
  float* F = reinterpret_cast<float*>(g.F + it.f_off);
  int* ipiv = g.ipiv + it.p_off;
  const double* A = g.A + it.a_off;
  const double* B = g.B + it.b_off;
  const double tol = g.tol > 0.0 ? g.tol : 1e-15 * n;
  const int lane = tid_() & 31, warp = tid_() >> 5;
  // fl32(A), ||A||_inf and ||b_h||_inf
  {
    double m = 0.0;
    for (int i = warp; i < n; i += kBT / 32) {
      double s = 0.0;
      double v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = lane + 32 * q < n ? A[i * n + lane + 32 * q] : 0.0;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (lane + 32 * q < n) {
          F[i * n + lane + 32 * q] = (float)v[q];
          s += fabs(v[q]);
        }
      __syncwarp();
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      m = fmax(m, norm_abs(s));
    }
    if (lane == 0) fx->red[0][warp][0] = m;
    col_max(n, r, fx->red[1], [&](int i, int h) { return B[i * r + h]; });
    __syncthreads();
    if (tid_() < r) fx->bnorm[tid_()] = red_max(fx->red[1], tid_());
    if (tid_() == 0) fx->anorm = red_max(fx->red[0], 0);
    __syncthreads();
  }
  if (it.kind == LM_BATCH_GENERAL) lu_factor<float>(F, n, it.nb, ipiv, region, fx);
  else chol_factor<float>(F, n, it.nb, region, fx);
  const bool regular = fx->info == 0;
  float* D = reinterpret_cast<float*>(region);  // the residual, read before the solves stage over it
  // x0 from the FP32 factors
  for (int e = tid_(); e < n * ldx; e += kBT) Xd[e] = 0.0;
  __syncthreads();
  if (regular) {
    solve_factored<float>(
        F, n, it.kind, fx, r, region, [&](int i, int h) { return (float)B[i * r + h]; },
        [&](int i, int h, float x) { Xd[i * ldx + h] = (double)x; });
  } else {
    for (int e = tid_(); e < n * r; e += kBT) Xd[(e / r) * ldx + e % r] = (double)(float)B[e];
    __syncthreads();
  }
  int iters = 0;
  bool ok = false;
  double be = 0.0;
  for (;;) {
    if (r <= 8) batch_residual<1>(A, B, n, r, Xd, ldx, D, fx);
    else batch_residual<2>(A, B, n, r, Xd, ldx, D, fx);
    col_max(n, r, fx->red[1], [&](int i, int h) { return Xd[i * ldx + h]; });
    __syncthreads();
    if (warp == 0) {
      double bh = 0.0;
      if (lane < r) {
        const double rn = red_max(fx->red[0], lane);
        const double den = fx->anorm * red_max(fx->red[1], lane) + fx->bnorm[lane];
        // a residual or a denominator that is not finite says nothing: never converged
        // (rn / inf would be a perfect zero)
        bh = rn <= DBL_MAX && den <= DBL_MAX ? (den > 0.0 ? rn / den : (rn > 0.0 ? DBL_MAX : 0.0)) : DBL_MAX;
      }
      __syncwarp();
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) bh = fmax(bh, __shfl_xor_sync(0xffffffffu, bh, o));
      if (lane == 0) fx->be = bh;
    }
    __syncthreads();
    be = fx->be;
    if (be <= tol) { ok = true; break; }
    if (iters >= g.max_iter || !regular) break;
    solve_factored<float>(
        F, n, it.kind, fx, r, region, [&](int i, int h) { return D[i * r + h]; },
        [&](int i, int h, float x) { Xd[i * ldx + h] += (double)x; });
    ++iters;
  }
  *berr_out = be;
  if (ok) {
    if (tid_() == 0) fx->info = 0;
    for (int e = tid_(); e < n * r; e += kBT) g.X[it.x_off + e] = Xd[(e / r) * ldx + e % r];
    __syncthreads();
    return iters;
  }
  // FP64 fallback: refactor from A in the same workspace (n^2 doubles)
  __syncthreads();
  run_fp64(it, g, sm, fx);
  __syncthreads();
  return -1;
}

__global__ void __launch_bounds__(kBT, 4) batch_kernel(const BatchArgs g) {
  extern __shared__ __align__(16) unsigned char sm[];
  Fixed* fx = reinterpret_cast<Fixed*>(sm);
  for (;;) {
    if (tid_() == 0) fx->slot = atomicAdd(g.ticket, 1);
    __syncthreads();
    const int s = fx->slot;
    __syncthreads();
    if (s >= g.count) break;
    const BatchItem it = g.items[s];
    if (it.n <= 0) continue;
    int iters = 0;
    double be = 0.0;
    if (g.prec == LM_PREC_FP32_IR) iters = run_ir(it, g, sm, fx, &be);
    else run_fp64(it, g, sm, fx);
    __syncthreads();
    if (tid_() == 0) {
      g.info[it.index] = fx->info;
      g.iters[it.index] = iters;
      g.berr[it.index] = be;
    }
    __syncthreads();
  }
}

// Device-resident request loop (the serving loop's small requests): every CTA
// claims the next posted request from a ring in device memory (head < tail),
// solves it in FP64 exactly as batch_kernel would, writes X into the arena and
// publishes info and a completion sequence number into pinned host memory.
// An idle CTA sleeps between polls and returns after kServeIdlePolls polls
// without work (the host relaunches the loop when new work arrives); the stop
// word ends it at once.  No other wait.
constexpr uint32_t kServeIdlePolls = 4000;  // x ~2 us of sleep: ~8 ms idle before returning

__global__ void __launch_bounds__(kBT, 4) serve_loop_kernel(const BatchArgs g, const ServeRing rg) {
  extern __shared__ __align__(16) unsigned char sm[];
  Fixed* fx = reinterpret_cast<Fixed*>(sm);
  for (;;) {
    if (tid_() == 0) {
      int claimed = -1;
      for (uint32_t idle = 0; idle < kServeIdlePolls;) {
        if (*reinterpret_cast<volatile const int*>(rg.stop) != 0) break;
        const int h = *reinterpret_cast<volatile const int*>(rg.head);
        const int t = *reinterpret_cast<volatile const int*>(rg.tail);
        if (h < t) {
          if (atomicCAS(rg.head, h, h + 1) == h) {
            claimed = h;
            break;
          }
          continue;  // another CTA took it: look again at once
        }
        __nanosleep(2000);
        ++idle;
      }
      fx->slot = claimed;
    }
    __syncthreads();
    const int sq = fx->slot;
    __syncthreads();
    if (sq < 0) return;
    const int idx = sq % rg.cap;
    BatchItem it;
    {
      const long long* src = reinterpret_cast<const long long*>(rg.items + idx);
      long long* dst = reinterpret_cast<long long*>(&it);
#pragma unroll
      for (int w = 0; w < (int)(sizeof(BatchItem) / sizeof(long long)); ++w) dst[w] = __ldcg(src + w);
    }
    int info = 0;
    if (it.n > 0) {
      run_fp64<true>(it, g, sm, fx);
      __syncthreads();
      info = fx->info;
    }
    __syncthreads();
    if (tid_() == 0) {
      __threadfence();  // X visible in device memory before the host copies it out
      rg.h_info[idx] = info;
      __threadfence_system();
      *reinterpret_cast<volatile int*>(rg.h_done + idx) = sq + 1;
    }
    __syncthreads();
  }
}

}  // namespace

size_t batch_smem_bytes(int nmax, int rmax, int prec) {
  const size_t fp64 = kFixed + region_bytes(nmax, 8);
  return prec == LM_PREC_FP32_IR ? std::max(fp64, ir_region(nmax, rmax) + region_bytes(nmax, 4)) : fp64;
}

int serve_loop_launch(const BatchArgs& g, const ServeRing& rg, int grid, size_t smem, cudaStream_t st) {
  static size_t set_to[kMaxDevices] = {};
  int dev = 0;
  LM_CUDA_TRY(cudaGetDevice(&dev));
  if (set_to[dev] < smem) {
    LM_CUDA_TRY(cudaFuncSetAttribute(serve_loop_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    set_to[dev] = smem;
  }
  serve_loop_kernel<<<grid, kBT, smem, st>>>(g, rg);
  count_launch(1);
  LM_CUDA_TRY(cudaGetLastError());
  return LM_OK;
}

// Raise the kernel's dynamic shared-memory limit to `smem` (once per size and device).
int batch_set_smem(size_t smem) {
  static size_t set_to[kMaxDevices] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (set_to[dev] < smem) {
    LM_CUDA_TRY(cudaFuncSetAttribute(batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    set_to[dev] = smem;
  }
  return LM_OK;
}

int batch_launch(const BatchArgs& g, int grid, size_t smem, cudaStream_t st) {
  LM_TRY(batch_set_smem(smem));
  LM_CUDA_TRY(cudaMemsetAsync(g.ticket, 0, sizeof(int), st));
  batch_kernel<<<grid, kBT, smem, st>>>(g);
  count_launch(1);
  LM_CUDA_TRY(cudaGetLastError());
  return LM_OK;
}

int batch_occupancy(size_t smem, int* per_sm) {
  LM_TRY(batch_set_smem(smem));
  LM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, batch_kernel, kBT, smem));
  return LM_OK;
}

}  // namespace lm
