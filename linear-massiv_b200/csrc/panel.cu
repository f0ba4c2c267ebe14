// Panel kernel: the latency-bound, column-by-column part of LU.
//
// panel_lu  — partial-pivoting LU of a whole panel (rows [c0, n), up to 128
//   columns) in one launch, the B200 replacement for panelLUFactor's column
//   loop (LU.hs:320-327: rawPivotSearch K.hs:1541-1556, rawSwapRows
//   K.hs:1507-1537, rawLUEliminateColumnTo K.hs:1464-1503) together with the
//   block solves and updates inside the panel.  One thread-block cluster (up
//   to 16 CTAs); CTA q owns the rows [q rpc, (q + 1) rpc) of the panel from
//   the first column to the last.  Rows never move while the panel is
//   factored: each carries its logical index, an interchange swaps two
//   labels, and the panel's rows are put in order once at the end.  So the
//   32-column leaves inside a panel need no row exchange of their own:
//     leaf    : W columns in registers, one thread per row (RPT rows for tall
//               panels), in micro-panels of MW <= 8 columns;
//     solve   : the leaf's pivot rows of the remaining columns become U12 =
//               L11^-1 A12 in shared memory, in every CTA (L11 came with the
//               pivot rows, so only A12 is read);
//     update  : every CTA subtracts L21 U12 from its own rows (DMMA for FP64,
//               FFMA for FP32); the next leaf's columns stay on chip.
//   The column step is a latency chain: warp vote, CTA barrier, vote over the
//   warps, one message to every CTA, vote over the CTAs, multipliers, update
//   of the micro-panel.  Only the micro-panel's 8 columns are on it: they
//   (with the reciprocal of the leading entry, formed while the warp votes)
//   are all that a candidate sends, and the rest of the leaf's columns is
//   updated once per micro-panel with the 8 pivot rows, which their owners
//   send on the side.  What bounds a column is instruction latency: about 480
//   instructions per warp, with the solves and updates, at 7.4 cycles each and one
//   to four warps per scheduler.
//   A 128-column panel takes 205 us at 500 to 2000 rows (FP64); the 32-column
//   leaves before it took 63 us each, with 100 us of small solves, products
//   and interchanges between the four of them (8192 rows).
//   NaN rule of the reference scan: if |a_jj| is NaN it stays the pivot; NaNs
//   below it never win.
#include <algorithm>
#include <climits>

#include "common.cuh"
#include "internal.h"
#include "pivot.cuh"

namespace lm {

void count_launch(int n);

namespace {

constexpr int kPanelNB = 128;      // widest panel
constexpr int kPanelThreads = 512; // most threads per CTA (one row of the leaf each, times RPT)
constexpr int kPanelCtas = 16;     // largest cluster

// The candidate that each CTA sends to every CTA of the cluster, once per
// column: 16-byte chunks, header then the micro-panel's part of the row in
// the rotated register layout.
template <typename T, int MW>
struct LeafMsg {
  typename PivKey<T>::K key;  // PivKey of the candidate (kForced: row j with a NaN a_jj)
  int label;                  // its logical row in the panel, or INT_MAX: no candidate
  int row;                    // its row in the sending CTA
  T rcp;                      // reciprocal of its leading entry
  alignas(16) T v[MW];
};

template <typename T, int W_>
struct PanelCfg {
  static constexpr int W = W_;
  static constexpr int MW = W < 8 ? W : 8;  // micro-panel width
  static constexpr int ZW = W - MW;         // the leaf's columns outside the micro-panel
  using Msg = LeafMsg<T, MW>;
  static constexpr int MSG_CHUNKS = (int)sizeof(Msg) / 16;
  static_assert(sizeof(Msg) % 16 == 0 && MSG_CHUNKS <= 32, "whole 16-byte chunks, one per lane");
  static constexpr int SLD = W + 16 / (int)sizeof(T);  // slab row stride: 16-byte rows, distinct banks
  // U12 row stride; = 4 (mod 16) keeps the DMMA operand reads conflict-free
  static constexpr int LDU = kPanelNB - W + (W >= 8 ? 4 : 8);
  static constexpr size_t cand = 0;                                    // Msg[2][16] received
  static constexpr size_t wmsg = cand + 2 * kPanelCtas * sizeof(Msg);  // Msg[2][16] one per warp
  static constexpr size_t bars = wmsg + 2 * 16 * sizeof(Msg);          // uint64_t[3]
  static constexpr size_t zrow = bars + 32;                            // T[MW][ZW] pivot rows, other columns
  static constexpr size_t prow = zrow + MW * ZW * sizeof(T);           // int[2][W] pivot rows (panel-relative)
  static constexpr size_t list = (prow + 2 * W * 4 + 15) / 16 * 16;    // int[2][256] row plan
  static constexpr size_t l11 = list + 2 * kSwapPlanRows * 4;          // T[W][SLD], L11 by columns
  static constexpr size_t us = l11 + W * SLD * sizeof(T);              // T[W][LDU]
  static constexpr size_t lab = us + (size_t)W * LDU * sizeof(T);      // int[rpc]
  static size_t slab_off(int rpc) { return lab + ((size_t)rpc * 4 + 15) / 16 * 16; }
  // the slab, which also stages the moved rows 8 columns at a time
  __host__ __device__ static int slab_elems(int rpc) {
    return rpc * SLD > kSwapPlanRows * 8 ? rpc * SLD : kSwapPlanRows * 8;
  }
  static size_t bytes(int rpc) { return slab_off(rpc) + (size_t)slab_elems(rpc) * sizeof(T); }
};

// Block of 32 rows x BW columns of the in-panel update: C -= L U with L
// (rows r0.., W columns) in the slab and U (W x BW) in shared memory.  C comes
// from global memory; the result goes back there, or for the next leaf's
// columns (`keep`) into the slab rows.  Rows that are finished (label < done)
// keep their global contents.
template <typename T, int W, int SLD, int LDU, int BW>
__device__ __forceinline__ void panel_update(T* slab, const T* U, const int* lab, int done, int r0, int rcnt, T* C,
                                             long long lda, int nc, bool keep) {
  const int lane = threadIdx.x & 31;
  if constexpr (sizeof(T) == 8) {
    const int gq = lane >> 2, tq = lane & 3;
    double acc[2][BW / 8][4];
    bool live[2][2];
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = r0 + mi * 16 + h * 8 + gq;
        live[mi][h] = r < rcnt && lab[r] >= done;
#pragma unroll
        for (int ni = 0; ni < BW / 8; ++ni) {
          const int c = ni * 8 + 2 * tq;
          double2 v = make_double2(0.0, 0.0);
          if (live[mi][h]) {
            const double* p = C + (long long)r * lda + c;
            if (c + 1 < nc) v = *reinterpret_cast<const double2*>(p);
            else if (c < nc) v.x = *p;
          }
          acc[mi][ni][2 * h] = v.x;
          acc[mi][ni][2 * h + 1] = v.y;
        }
      }
    __syncwarp();
#pragma unroll 2
    for (int k = 0; k < W; k += 4) {
      double a[2][2], b[BW / 8];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int h = 0; h < 2; ++h) a[mi][h] = -slab[(r0 + mi * 16 + h * 8 + gq) * SLD + k + tq];
#pragma unroll
      for (int ni = 0; ni < BW / 8; ++ni) b[ni] = U[(k + tq) * LDU + ni * 8 + gq];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int ni = 0; ni < BW / 8; ++ni) dmma_16x8x4(acc[mi][ni], a[mi][0], a[mi][1], b[ni]);
    }
    if (keep) __syncwarp();  // every lane has read its slab operands
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = r0 + mi * 16 + h * 8 + gq;
#pragma unroll
        for (int ni = 0; ni < BW / 8; ++ni) {
          const int c = ni * 8 + 2 * tq;
          const double2 v = make_double2(acc[mi][ni][2 * h], acc[mi][ni][2 * h + 1]);
          if (keep && c < W) {
            if (r < rcnt) {
              slab[r * SLD + c] = c < nc ? v.x : 0.0;
              slab[r * SLD + c + 1] = c + 1 < nc ? v.y : 0.0;
            }
          } else if (live[mi][h]) {
            double* p = C + (long long)r * lda + c;
            if (c + 1 < nc) *reinterpret_cast<double2*>(p) = v;
            else if (c < nc) *p = v.x;
          }
        }
      }
  } else {
    // lane = (row group rg, column group tq): rows r0 + 8 i + rg, columns tq CT ..
    constexpr int CT = BW / 4;
    const int rg = lane >> 2, tq = lane & 3;
    float acc[4][CT];
    bool live[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + 8 * i + rg;
      live[i] = r < rcnt && lab[r] >= done;
#pragma unroll
      for (int c = 0; c < CT; ++c) {
        const int cc = tq * CT + c;
        acc[i][c] = live[i] && cc < nc ? C[(long long)r * lda + cc] : 0.f;
      }
    }
    __syncwarp();
#pragma unroll 4
    for (int k = 0; k < W; ++k) {
      float a[4], b[CT];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = slab[(r0 + 8 * i + rg) * SLD + k];
#pragma unroll
      for (int c = 0; c < CT; ++c) b[c] = U[k * LDU + tq * CT + c];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < CT; ++c) acc[i][c] = fmaf(-a[i], b[c], acc[i][c]);
    }
    if (keep) __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + 8 * i + rg;
#pragma unroll
      for (int c = 0; c < CT; ++c) {
        const int cc = tq * CT + c;
        if (keep && cc < W) {
          if (r < rcnt) slab[r * SLD + cc] = cc < nc ? acc[i][c] : 0.f;
        } else if (live[i] && cc < nc) {
          C[(long long)r * lda + cc] = acc[i][c];
        }
      }
    }
  }
}

// N elements between a thread's registers and 16-byte aligned shared memory.
template <typename T, int N>
__device__ __forceinline__ void vec_load(T* x, const T* p) {
  if constexpr (sizeof(T) == 8) {
#pragma unroll
    for (int c = 0; c < N; c += 2) {
      const double2 v = *reinterpret_cast<const double2*>(p + c);
      x[c] = v.x; x[c + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int c = 0; c < N; c += 4) {
      const float4 v = *reinterpret_cast<const float4*>(p + c);
      x[c] = v.x; x[c + 1] = v.y; x[c + 2] = v.z; x[c + 3] = v.w;
    }
  }
}
template <typename T, int N>
__device__ __forceinline__ void vec_store(T* p, const T* x) {
  if constexpr (sizeof(T) == 8) {
#pragma unroll
    for (int c = 0; c < N; c += 2) *reinterpret_cast<double2*>(p + c) = make_double2(x[c], x[c + 1]);
  } else {
#pragma unroll
    for (int c = 0; c < N; c += 4) *reinterpret_cast<float4*>(p + c) = make_float4(x[c], x[c + 1], x[c + 2], x[c + 3]);
  }
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// x <- L^-1 x for the unit lower triangle of order N held by columns in
// shared memory (column k at l + k ld): by columns, so that the updates of
// one step are independent, with 16-byte loads of L.
template <typename T, int N>
__device__ __forceinline__ void unit_lower_solve(T (&x)[N], const T* l, int ld) {
  constexpr int V = 16 / (int)sizeof(T);
#pragma unroll
  for (int k = 0; k + 1 < N; ++k)
#pragma unroll
    for (int i = (k + 1) / V * V; i < N; i += V) {
      T c[V];
      vec_load<T, V>(c, l + k * ld + i);
#pragma unroll
      for (int e = 0; e < V; ++e)
        if (i + e > k) x[i + e] = fma(-c[e], x[k], x[i + e]);
    }
}

// plan: [0] the number of rows of the panel that change place, then their
// destination rows and (kSwapPlanInts layout) their source rows.
template <typename T, int W, int RPT>
__global__ void __launch_bounds__(kPanelThreads, 1)
    panel_lu_kernel(T* A, long long lda, int n, int c0, int pw, int rpc, unsigned slab_off, int* ipiv, int* plan,
                    int* status) {
  using Cfg = PanelCfg<T, W>;
  using Msg = typename Cfg::Msg;
  using Key = typename PivKey<T>::K;
  constexpr int SLD = Cfg::SLD, LDU = Cfg::LDU, MW = Cfg::MW, ZW = Cfg::ZW;
  constexpr int V = 16 / (int)sizeof(T);
  extern __shared__ __align__(16) unsigned char sm[];
  Msg* cand = reinterpret_cast<Msg*>(sm + Cfg::cand);
  Msg* wmsg = reinterpret_cast<Msg*>(sm + Cfg::wmsg);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + Cfg::bars);  // candidates (by parity), pivot rows
  T* zrow = reinterpret_cast<T*>(sm + Cfg::zrow);
  int* prow_id = reinterpret_cast<int*>(sm + Cfg::prow);  // of this leaf and the one before
  int* list = reinterpret_cast<int*>(sm + Cfg::list);
  T* L11 = reinterpret_cast<T*>(sm + Cfg::l11);  // by columns: l_ik at k SLD + i
  T* Us = reinterpret_cast<T*>(sm + Cfg::us);
  int* lab = reinterpret_cast<int*>(sm + Cfg::lab);
  T* slab = reinterpret_cast<T*>(sm + slab_off);

  const int q = (int)cluster_ctarank();
  const int C = (int)cluster_nctarank();
  const int tid = threadIdx.x, NT = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = NT >> 5;
  const int R = n - c0;
  const int rbeg = q * rpc;
  const int rcnt = max(0, min(rpc, R - rbeg));
  T* P = A + (long long)c0 * lda + c0;  // panel
  T* Pm = P + (long long)rbeg * lda;    // this CTA's rows
  constexpr int RPI = 32 / W;           // rows per warp access of the leaf's columns

  if (tid == 0) {
#pragma unroll
    for (int b = 0; b < 3; ++b) mbar_init(&bars[b], 1);
    fence_barrier_init();
    if (q == 0) plan[0] = 0;
  }

  // logical row of each of this thread's rows (row s NT + tid of the CTA)
  int lr[RPT];
#pragma unroll
  for (int s = 0; s < RPT; ++s) {
    const int r = s * NT + tid;
    lr[s] = r < rcnt ? rbeg + r : -1;  // -1: no row here, never active
  }
  // first leaf through the slab (whole rows per access)
  {
    const int w0 = min(W, pw);
#pragma unroll 8
    for (int r = warp * RPI + lane / W; r < rcnt; r += nw * RPI) {
      const int c = lane % W;
      slab[r * SLD + c] = c < w0 ? Pm[(long long)r * lda + c] : T(0);
    }
  }
  __syncthreads();
  cluster_sync_all();  // every CTA's barriers exist before anyone pushes into them

  // this thread's part of a candidate's way to the other CTAs: chunk pch of
  // the message to CTA pd (C MSG_CHUNKS <= 96 threads have one)
  const int pd = tid / Cfg::MSG_CHUNKS, pch = tid % Cfg::MSG_CHUNKS;
  const uint32_t push_dst = pd < C ? dsmem_map(cand + q, pd) + pch * 16 : 0u;
  const uint32_t push_bar = pd < C ? dsmem_map(bars, pd) : 0u;

  bool timed_out = false;
  bool arrived = false;  // a cluster barrier arrival is outstanding (in-panel updates published)
  // Row of the CTA (or -1) whose columns outside the current micro-panel this
  // warp still has to send as pivot row j: its finished columns and its z, both
  // in the slab, become row j of zrow in every CTA.
  int zpush = -1;
  auto send_z = [&](int j, int m0) {
    if constexpr (ZW > 0) {
      if (zpush >= 0) {  // uniform in the warp
        __syncwarp();
        constexpr int ZCH = ZW / V;  // 16-byte chunks
        const T* sr = slab + zpush * SLD;
        for (int e = lane; e < C * ZCH; e += 32) {
          const int d = e / ZCH, c = (e % ZCH) * V;
          const uint4 v = *reinterpret_cast<const uint4*>(sr + (c < m0 ? c : c + MW));
          T* dst = zrow + j * ZW + c;
          if (C > 1)
            st_async_16(dsmem_map(dst, d), dsmem_map(&bars[2], d), v.x, v.y, v.z, v.w);
          else
            *reinterpret_cast<uint4*>(dst) = v;
        }
        zpush = -1;
      }
    }
  };
  int step = 0;  // columns so far: message buffer step & 1, mbarrier phase (step >> 1) & 1
  uint32_t zphase = 0;

  for (int o = 0, leaf = 0; o < pw; o += W, ++leaf) {
    const int w = min(W, pw - o);
    const int nc = pw - o - w;  // panel columns right of this leaf
    T* Pn = P + o + W;          // (the first of them)
    int* pid = prow_id + (leaf & 1) * W;
    T y[RPT][MW];                // the micro-panel, rotated: slot 0 is the current column
    T z[RPT][ZW > 0 ? ZW : 1];   // the leaf's columns right of it
#pragma unroll
    for (int s = 0; s < RPT; ++s) {
      const int r = s * NT + tid;
      if (r < rcnt) {
        vec_load<T, MW>(y[s], slab + r * SLD);
        if constexpr (ZW > 0) vec_load<T, ZW>(z[s], slab + r * SLD + MW);
      } else {
#pragma unroll
        for (int c = 0; c < MW; ++c) y[s][c] = T(0);
#pragma unroll
        for (int c = 0; c < ZW; ++c) z[s][c] = T(0);
      }
    }

#pragma unroll 1
    for (int m0 = 0; m0 < w; m0 += MW) {
      const int wm = min(MW, w - m0);
      if (ZW > 0 && C > 1 && tid == 0 && !timed_out) mbar_arrive_expect_tx(&bars[2], (uint32_t)(wm * ZW * sizeof(T)));
      // this thread's best candidate for the next column
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
        if (lr[s] >= o + m0) consider(s, y[s][0], o + m0);

      // One column per step.  The loop stays rolled, the registers rotating
      // instead: unrolled over the micro-panel every step fetched its
      // instructions anew and took a third longer.
#pragma unroll 1
      for (int j = 0; j < wm; ++j, ++step) {
        const int J = o + m0 + j;
        const int par = step & 1;
        // ---- the warp's candidate, staged; then the CTA's, by every warp ----
        const T rc = PivKey<T>::rcp(xb);
        const int wl = warp_winner(bk, bi);
        Msg* wms = wmsg + par * 16;
        if (lane == wl) {
          Msg* out = wms + warp;
          out->key = bk;
          out->label = bi;
          out->row = bs * NT + tid;
          out->rcp = rc;
#pragma unroll
          for (int s = 0; s < RPT; ++s)
            if (s == bs) vec_store<T, MW>(out->v, y[s]);
        }
        // (not again on a phase that did not end: its arrival is spent)
        if (C > 1 && tid == 0 && !timed_out) mbar_arrive_expect_tx(&bars[par], (uint32_t)(C * sizeof(Msg)));
        __syncthreads();
        const int wo = warp_winner(lane < nw ? wms[lane].key : Key(0), lane < nw ? wms[lane].label : INT_MAX);
        const Msg* win = wms + wo;
        int qw = 0;
        if (C > 1) {
          // ---- to every CTA; then the best of all ----
          Msg* in = cand + par * kPanelCtas;
          if (pd < C) {
            const uint4 v = reinterpret_cast<const uint4*>(win)[pch];
            st_async_16(push_dst + par * (uint32_t)(kPanelCtas * sizeof(Msg)), push_bar + par * 8u, v.x, v.y, v.z, v.w);
          }
          if (j > 0) send_z(j - 1, m0);
          if (!timed_out && !mbar_wait_spin(&bars[par], (uint32_t)((step >> 1) & 1), status)) timed_out = true;
          qw = warp_winner(lane < C ? in[lane].key : Key(0), lane < C ? in[lane].label : INT_MAX);
          if (qw >= C) qw = 0;
          win = in + qw;
        } else if (j > 0) {
          send_z(j - 1, m0);
        }
        // (row J itself is always a candidate, so some CTA wins)
        const int p = pivot_position(win->label, J, timed_out);
        const T rcp = win->rcp;
        T u[MW];
        vec_load<T, MW>(u, win->v);
        const T piv = u[0];
        const bool safe = PivKey<T>::safe(piv);
        const bool owner = qw == q && warp == wo && lane == wl;
        const int bs_out = bs;  // (the owner lane's row)
        // ---- interchange labels; multipliers; the micro-panel; next scan ----
        bk = 0;
        bi = INT_MAX;
#pragma unroll
        for (int s = 0; s < RPT; ++s) {
          if (lr[s] == p) lr[s] = J;
          else if (lr[s] == J) lr[s] = p;
          T m = y[s][0];
          if (lr[s] > J) {
            m = div_by(y[s][0], piv, rcp);
            if (!safe) m = y[s][0] / piv;
#pragma unroll
            for (int c = 1; c < MW; ++c)
              if (c < MW - j) y[s][c] = fma(-m, u[c], y[s][c]);
            consider(s, y[s][1], J + 1);
          }
          __syncwarp();  // rejoin at once: split, the warp would run all that follows twice
#pragma unroll
          for (int c = 0; c + 1 < MW; ++c) y[s][c] = y[s][c + 1];
          y[s][MW - 1] = m;
        }
        // ---- the pivot row's other columns: into the slab (this part of it is
        //      rewritten later), from where they go out beside the next exchange ----
        if constexpr (ZW > 0) {
          if (qw == q && warp == wo) {  // uniform in the warp
            const int prow = min(bs_out * NT + tid, rpc - 1);  // (a winner has a row; see pivot_position)
            if (owner) {
              T* sr = slab + prow * SLD + m0 + MW;
#pragma unroll
              for (int s = 0; s < RPT; ++s)
                if (s == bs_out) {
#pragma unroll
                  for (int g = 0; g < ZW; g += MW)
                    if (g < ZW - m0) vec_store<T, MW>(sr + g, z[s] + g);
                }
            }
            __syncwarp();
            zpush = __shfl_sync(0xffffffffu, prow, wl);
          }
        }
        // L11 and the pivot's place, for the solves; the swap list
        if (warp == nw - 1) {
          if (lane < j) L11[(m0 + lane) * SLD + m0 + j] = win->v[MW - j + lane];
          if (lane == 0) {
            pid[m0 + j] = min(max(qw * rpc + win->row, 0), R - 1);
            if (q == 0) {
              ipiv[c0 + J] = c0 + p;
              if (piv == T(0)) atomicCAS(status + 1, 0, c0 + J + 1);
            }
          }
        }
        __syncwarp();
        // The buffers of this parity are rewritten two columns later, behind
        // a barrier (here) and a message (elsewhere) that follow these reads.
      }
#pragma unroll 1
      for (int k = wm; k < MW; ++k) {  // a narrower micro-panel: finish the rotation
#pragma unroll
        for (int s = 0; s < RPT; ++s) {
          const T m = y[s][0];
#pragma unroll
          for (int c = 0; c + 1 < MW; ++c) y[s][c] = y[s][c + 1];
          y[s][MW - 1] = m;
        }
      }

      __syncwarp();
      if constexpr (ZW > 0) {
        send_z(wm - 1, m0);
        if (C > 1 && !timed_out && !mbar_wait(&bars[2], zphase, status)) timed_out = true;
        zphase ^= 1u;
        __syncwarp();
      }
#pragma unroll
      for (int s = 0; s < RPT; ++s) {
        const int r = s * NT + tid;
        if (r < rcnt) {
          vec_store<T, MW>(slab + r * SLD + m0, y[s]);
          lab[r] = lr[s];
        }
      }
      __syncwarp();
      if (m0 == 0 && arrived) cluster_wait();  // every CTA's updates of the columns from here on are visible
      __syncthreads();  // pivot rows, L11 and pid complete
      if (m0 == 0 && arrived) {
        // every CTA has read the A12 rows of the leaf before: its U12 can go to
        // its (unmoved) rows
        const int uc = pw - o;
        const int* id = prow_id + ((leaf & 1) ^ 1) * W;
        for (int k = warp; k < W; k += nw) {
          const int r = id[k];
          if (r >= rbeg && r < rbeg + rcnt)
            for (int c = lane; c < uc; c += 32) P[(long long)r * lda + o + c] = Us[k * LDU + c];
        }
        arrived = false;
        __syncthreads();
      }
      // A12 of these pivot rows on its way
      for (int k = m0 + warp; nc > 0 && k < m0 + wm; k += nw) {
        const T* src = Pn + (long long)pid[k] * lda;
        for (int c = lane * V; c < nc; c += 32 * V) {
          if (c + V <= nc) {
            cp_async16(Us + k * LDU + c, src + c);
          } else {
#pragma unroll
            for (int e = 0; e < V; ++e)
              if (c + e < nc) Us[k * LDU + c + e] = __ldcg(src + c + e);
          }
        }
      }
      if constexpr (ZW > 0) {
        const int zl = ZW - m0;  // leaf columns right of the micro-panel
        if (warp == 0) {
          // U = L^-1 Z on them, lane = column
          if (lane < zl && wm == MW) {
            T v[MW];
#pragma unroll
            for (int i = 0; i < MW; ++i) v[i] = zrow[i * ZW + m0 + lane];
            unit_lower_solve<T, MW>(v, L11 + m0 * SLD + m0, SLD);
#pragma unroll
            for (int i = 0; i < MW; ++i) zrow[i * ZW + m0 + lane] = v[i];
          }
        } else if (warp == 1) {
          // the pivot rows' finished columns complete L11
          for (int c = lane; c < m0; c += 32)
            for (int i = 0; i < wm; ++i) L11[c * SLD + m0 + i] = zrow[i * ZW + c];
        }
        __syncthreads();
        if (zl > 0 && wm == MW) {
          // rank-MW update of them: every row below, and pivot row i with the i rows above it
          int cnt[RPT];
          bool full = true;
#pragma unroll
          for (int s = 0; s < RPT; ++s) {
            const int d = lr[s] - (o + m0);
            cnt[s] = min(max(d, 0), MW);
            full = full && (d >= MW || lr[s] < 0);
          }
          full = __all_sync(0xffffffffu, full);
#pragma unroll
          for (int g = 0; g < ZW; g += MW) {
            if (g < zl) {
#pragma unroll
              for (int k = 0; k < MW; ++k) {
                T uk[MW];
                vec_load<T, MW>(uk, zrow + k * ZW + m0 + g);
#pragma unroll
                for (int s = 0; s < RPT; ++s)
                  if (full || k < cnt[s]) {
#pragma unroll
                    for (int c = 0; c < MW; ++c) z[s][g + c] = fma(-y[s][k], uk[c], z[s][g + c]);
                  }
              }
            }
          }
#pragma unroll
          for (int s = 0; s < RPT; ++s) {
#pragma unroll
            for (int c = 0; c < MW; ++c) y[s][c] = z[s][c];
#pragma unroll
            for (int c = 0; c + MW < ZW; ++c) z[s][c] = z[s][c + MW];
          }
        }
      }
    }

    // ---- the leaf's columns back to their rows in memory (rows finished in an
    //      earlier leaf hold U12 entries there) ----
#pragma unroll 8
    for (int r = warp * RPI + lane / W; r < rcnt; r += nw * RPI) {
      const int c = lane % W;
      if (c < w && lab[r] >= o) Pm[(long long)r * lda + o + c] = slab[r * SLD + c];
    }
    if (nc <= 0) break;
    cp_async_wait_all();
    __syncthreads();
    // ---- U12 = L11^-1 A12 (w = W here), in every CTA ----
    if (tid < nc) {
      T v[W];
#pragma unroll
      for (int i = 0; i < W; ++i) v[i] = Us[i * LDU + tid];
      unit_lower_solve<T, W>(v, L11, SLD);
#pragma unroll
      for (int i = 0; i < W; ++i) Us[i * LDU + tid] = v[i];
    }
    __syncthreads();
    // ---- own rows -= L21 U12 in blocks of 32 rows x BW columns over the
    //      warps, the next leaf's columns last: they replace L21 in the slab ----
    constexpr int BW = W < 8 ? 8 : W;
    const int nrb = (rcnt + 31) / 32, ncb = (nc + BW - 1) / BW;
    for (int t = warp; t < nrb * (ncb - 1); t += nw) {
      const int r0 = t % nrb * 32, cb = 1 + t / nrb;
      panel_update<T, W, SLD, LDU, BW>(slab, Us + cb * BW, lab, o + W, r0, rcnt,
                                       Pn + (long long)rbeg * lda + cb * BW, lda, nc - cb * BW, false);
    }
    __syncthreads();
    for (int t = warp; t < nrb; t += nw)
      panel_update<T, W, SLD, LDU, BW>(slab, Us, lab, o + W, t * 32, rcnt, Pn + (long long)rbeg * lda, lda, nc, true);
    __syncthreads();
    cluster_arrive();
    arrived = true;
  }

  // After a wait that gave up the result is void (status 0 says so), the labels are
  // still rows of the panel (pivot_position), and messages may be on their way: no
  // CTA leaves the cluster before they have had a millisecond to land.
  if (timed_out)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);

  // ---- the rows that change place: list them, then move the panel's own
  //      columns, a share of the columns per CTA ----
#pragma unroll
  for (int s = 0; s < RPT; ++s) {
    const int r = s * NT + tid;
    if (r < rcnt && lr[s] != rbeg + r) {
      const int at = atomicAdd(plan, 1);  // at most 2 pw rows move
      if (at < kSwapPlanRows) {
        plan[1 + at] = c0 + lr[s];
        plan[1 + kSwapPlanRows + at] = c0 + rbeg + r;
      }
    }
  }
  __syncthreads();
  cluster_sync_all();
  const int m = min(__ldcg(plan), kSwapPlanRows);
  if (m == 0) return;
  for (int e = tid; e < 2 * kSwapPlanRows; e += NT) list[e] = (e & (kSwapPlanRows - 1)) < m ? __ldcg(plan + 1 + e) : 0;
  __syncthreads();
  // (per warp access 4 rows x 8 columns; gathered to the slab, then scattered)
  const int cw = ((pw + C - 1) / C + 7) / 8 * 8, cbeg = q * cw, cend = min(pw, cbeg + cw);
  const int per = Cfg::slab_elems(rpc) / (8 * m) * 8;  // columns per pass through the slab
  const int nr4 = (m + 3) / 4;
  for (int cp = cbeg; cp < cend; cp += per) {
    const int units = nr4 * ((min(per, cend - cp) + 7) / 8);
    for (int t0 = warp; t0 < units; t0 += 8 * nw) {
      T v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int t = t0 + i * nw, g = t / nr4, r = (t - g * nr4) * 4 + (lane >> 3), c = cp + g * 8 + (lane & 7);
        v[i] = t < units && r < m && c < cend ? __ldcg(A + (long long)list[kSwapPlanRows + r] * lda + c0 + c) : T(0);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int t = t0 + i * nw, g = t / nr4, r = (t - g * nr4) * 4 + (lane >> 3);
        if (t < units && r < m) slab[(g * m + r) * 8 + (lane & 7)] = v[i];
      }
    }
    __syncthreads();
    for (int t = warp; t < units; t += nw) {
      const int g = t / nr4, r = (t - g * nr4) * 4 + (lane >> 3), c = cp + g * 8 + (lane & 7);
      if (r < m && c < cend) A[(long long)list[r] * lda + c0 + c] = slab[(g * m + r) * 8 + (lane & 7)];
    }
    __syncthreads();
  }
}

// Shape of the panel kernel for `rows` rows: leaf width W and rows per thread
// RPT (W RPT registers of row data per thread: the widest leaf that holds the
// rows), threads per CTA NT and CTAs C.  Short panels are spread over the
// whole cluster, down to 32 rows per CTA: the in-panel updates then run on
// more SMs.  Idle warps of a short CTA share its solves and updates.
struct PanelShape {
  int W = 0, RPT = 0, NT = 0, C = 0, rpc = 0;
};

int max_cluster(Ctx& c);

template <typename T>
PanelShape panel_shape(Ctx& c, int rows) {
  PanelShape p;
  const long long cm = max_cluster(c);
  constexpr bool f32 = sizeof(T) == 4;
  for (int lv = 0; lv < 4 && !p.W; ++lv) {
    const int rpt = 1 << lv;
    if (rows > cm * kPanelThreads * rpt) continue;
    p.RPT = rpt;
    p.W = f32 ? (lv < 2 ? 32 : 64 >> lv) : 32 >> lv;
  }
  if (!p.W) return p;
  p.C = (int)std::min<long long>(cm, cdiv(rows, p.RPT > 1 ? kPanelThreads * p.RPT : 32));
  p.rpc = cdiv(cdiv(rows, p.C), 32) * 32;  // whole 32-row blocks
  p.NT = p.RPT > 1 ? kPanelThreads : std::max(128, p.rpc);
  return p;
}

template <typename T, int W, int RPT>
int launch_panel(Ctx& c, const PanelShape& ps, T* A, long long lda, int n, int c0, int pw, int* ipiv, int* plan,
                 cudaStream_t st) {
  using Cfg = PanelCfg<T, W>;
  auto kern = panel_lu_kernel<T, W, RPT>;
  static bool attr_set[kMaxDevices] = {};
  const int dev = ctx_device(c);
  if (!attr_set[dev]) {
    LM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)Cfg::bytes(kPanelThreads * RPT)));
    LM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ps.C, 1, 1);
  cfg.blockDim = dim3(ps.NT, 1, 1);
  cfg.dynamicSmemBytes = Cfg::bytes(ps.rpc);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ps.C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  LM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, A, lda, n, c0, pw, ps.rpc, (unsigned)Cfg::slab_off(ps.rpc), ipiv, plan,
                                 ctx_status(c)));
  count_launch(1);
  return LM_OK;
}

int g_max_cluster[kMaxDevices] = {};

// Largest cluster the device schedules for the panel kernel (16 when allowed).
int max_cluster(Ctx& c) {
  const int dev = ctx_device(c);
  if (g_max_cluster[dev]) return g_max_cluster[dev];
  int best = 8;
  using Cfg = PanelCfg<double, 16>;
  auto kern = panel_lu_kernel<double, 16, 2>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::bytes(kPanelThreads * 2)) ==
          cudaSuccess &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kPanelCtas, 1, 1);
    cfg.blockDim = dim3(kPanelThreads, 1, 1);
    cfg.dynamicSmemBytes = Cfg::bytes(kPanelThreads * 2);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kPanelCtas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int nclusters = 0;
    if (cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg) == cudaSuccess && nclusters > 0) best = kPanelCtas;
  }
  cudaGetLastError();
  g_max_cluster[dev] = best;
  return best;
}

}  // namespace

template <typename T>
int panel_ctas(Ctx& c, int rows) {
  return panel_shape<T>(c, rows).C;
}

template <typename T>
int panel_lu(Ctx& c, T* A, long long lda, int n, int c0, int pw, int* ipiv, int* plan, cudaStream_t st) {
  if (pw <= 0) return LM_OK;
  if (pw > kPanelNB || c0 + pw > n) return LM_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (lda * (int)sizeof(T)) % 16 || (c0 * (int)sizeof(T)) % 16)
    return LM_ERR_ARG;
  const PanelShape ps = panel_shape<T>(c, n - c0);
  if constexpr (sizeof(T) == 8) {
    if (ps.W == 32) return launch_panel<T, 32, 1>(c, ps, A, lda, n, c0, pw, ipiv, plan, st);
    if (ps.W == 16) return launch_panel<T, 16, 2>(c, ps, A, lda, n, c0, pw, ipiv, plan, st);
    if (ps.W == 8) return launch_panel<T, 8, 4>(c, ps, A, lda, n, c0, pw, ipiv, plan, st);
    if (ps.W == 4) return launch_panel<T, 4, 8>(c, ps, A, lda, n, c0, pw, ipiv, plan, st);
  } else {
    if (ps.W == 32 && ps.RPT == 1) return launch_panel<T, 32, 1>(c, ps, A, lda, n, c0, pw, ipiv, plan, st);
    if (ps.W == 32) return launch_panel<T, 32, 2>(c, ps, A, lda, n, c0, pw, ipiv, plan, st);
    if (ps.W == 16) return launch_panel<T, 16, 4>(c, ps, A, lda, n, c0, pw, ipiv, plan, st);
    if (ps.W == 8) return launch_panel<T, 8, 8>(c, ps, A, lda, n, c0, pw, ipiv, plan, st);
  }
  return LM_ERR_UNSUPPORTED;
}

template int panel_ctas<float>(Ctx&, int);
template int panel_lu<double>(Ctx&, double*, long long, int, int, int, int*, int*, cudaStream_t);
template int panel_lu<float>(Ctx&, float*, long long, int, int, int, int*, int*, cudaStream_t);

}  // namespace lm
