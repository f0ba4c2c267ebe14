// Device helpers of the column-by-column kernels (panel.cu, batch.cu): the
// pivot order of the reference's scan and quotients by a known reciprocal.
#pragma once

#include <climits>

#include "common.cuh"

namespace lm {

// The pivot order of the reference's scan (strict '>' from row j down): the
// larger |a| wins, the lower row on ties, NaN never wins.  |a| becomes an
// integer key in that order, its IEEE bits, so that a warp reduces it with
// redux.sync.  NaN gets the key of zero: row j, which has the lowest label, is
// always among the candidates, so neither ever beats it.  Row j with a NaN
// a_jj stays the pivot (the reference scan starts at row j and NaN never
// compares greater): kForced beats every other key.
template <typename T>
struct PivKey;
template <>
struct PivKey<double> {
  using K = unsigned long long;
  static constexpr K kForced = ~0ull;
  __device__ static K of(double x) {
    const K u = (K)__double_as_longlong(x) & 0x7fffffffffffffffull;
    return u > 0x7ff0000000000000ull ? 0ull : u;
  }
  // the reciprocal of a pivot in this range and the remainders formed with
  // it neither overflow nor lose bits to underflow
  __device__ static bool safe(double p) { const double a = fabs(p); return a > 0x1p-500 && a < 0x1p500; }
  // 1 / p to about an ulp: the hardware estimate and two Newton steps
  __device__ static double rcp(double p) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(p));
    r = fma(r, fma(-p, r, 1.0), r);
    return fma(r, fma(-p, r, 1.0), r);
  }
};
template <>
struct PivKey<float> {
  using K = unsigned;
  static constexpr K kForced = ~0u;
  __device__ static K of(float x) {
    const K u = __float_as_uint(x) & 0x7fffffffu;
    return u > 0x7f800000u ? 0u : u;
  }
  __device__ static bool safe(float p) { const float a = fabsf(p); return a > 0x1p-60f && a < 0x1p60f; }
  __device__ static float rcp(float p) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(p));
    return fmaf(r, fmaf(-p, r, 1.f), r);
  }
};

// Lane (the same in every lane) holding the warp's best (key, label): the
// largest key, then the lowest label.  Lanes without a candidate pass key 0
// and label INT_MAX.  Usually one redux.sync and one vote: the later rounds
// run only when several lanes share the leading bits.
__device__ __forceinline__ int warp_winner(unsigned key, int label) {
  __syncwarp();  // reconverge: a split warp would serialise every *_sync below
  unsigned b = __ballot_sync(0xffffffffu, key == __reduce_max_sync(0xffffffffu, key));
  if (b & (b - 1)) {
    const unsigned l = (b >> (threadIdx.x & 31)) & 1 ? (unsigned)label : 0xffffffffu;
    b = __ballot_sync(0xffffffffu, l == __reduce_min_sync(0xffffffffu, l));
  }
  return __ffs(b) - 1;
}
__device__ __forceinline__ int warp_winner(unsigned long long key, int label) {
  __syncwarp();
  const unsigned hi = (unsigned)(key >> 32);
  unsigned b = __ballot_sync(0xffffffffu, hi == __reduce_max_sync(0xffffffffu, hi));
  if (b & (b - 1)) {
    const int lane = threadIdx.x & 31;
    const unsigned lo = (b >> lane) & 1 ? (unsigned)key : 0u;
    b &= __ballot_sync(0xffffffffu, lo == __reduce_max_sync(0xffffffffu, lo));
    if (b & (b - 1)) {
      const unsigned l = (b >> lane) & 1 ? (unsigned)label : 0xffffffffu;
      b &= __ballot_sync(0xffffffffu, l == __reduce_min_sync(0xffffffffu, l));
    }
  }
  return __ffs(b) - 1;
}

// The row that takes position J of a panel, from the label of the winning
// candidate: J itself where there is none (INT_MAX), and after a wait that gave up
// (the message's place then holds whatever was there).
__host__ __device__ inline int pivot_position(int label, int J, bool gave_up) {
  return gave_up || label == INT_MAX ? J : label;
}

// x / p from a reciprocal r of p: the estimate x r corrected once by its remainder.
// The correctly rounded quotient where r is the correctly rounded reciprocal
// (Markstein 1990; tri_sweep's callers divide for it); with PivKey::rcp, which is
// off by up to about an ulp, within an ulp of the quotient.
template <typename T>
__device__ __forceinline__ T div_by(T x, T p, T r) {
  const T q = x * r;
  return fma(fma(-p, q, x), r, q);
}

// Numerators for which div_by holds, its divisor being PivKey::safe: neither the
// quotient nor the remainder then overflows, underflows or meets an infinity.
// Callers divide where one is not.  In FP32 that is the usual case of systems whose
// entries decay (Gaussian kernels): 600 SPD systems of order 128, FP32 factor and
// refinement, 0.54 ms with entries down to zero, 0.47 ms without.
template <typename T>
__device__ __forceinline__ bool quotient_safe(T y) { return PivKey<T>::safe(y) || y == T(0); }

// One triangular block of up to W rows by the W lanes of a group, lane l = row:
// y its right-hand side, t its row of the triangle (readable over bw entries, for
// l >= bw too), d and r its diagonal entry and the reciprocal (ignored with
// `unit`).  An entry leaves by shuffle as soon as it is final and is applied to the
// lanes that wait for it (the rows after it, or before it when !fwd).  Branch-free
// with quotients by the reciprocal; where one of them was not safe (see
// quotient_safe) the block is solved again by divisions.
template <typename T, int W>
__device__ __forceinline__ T tri_sweep(T y0, const T* t, T d, T r, int l, int bw, bool fwd, bool unit) {
  const bool in = l < bw;
  T y = y0, pre = T(0);
  __syncwarp();
#pragma unroll 8
  for (int s = 0; s < bw; ++s) {
    const int k = fwd ? s : bw - 1 - s;
    const bool waits = in && (fwd ? l > k : l < k);
    const T tk = t[k];  // (read whether it is used or not: a branch would split the warp)
    if (!unit) {
      pre = l == k ? y : pre;
      const T q = div_by(y, d, r);
      y = l == k ? q : y;
    }
    const T x = __shfl_sync(0xffffffffu, y, k, W);
    y = waits ? fma(-tk, x, y) : y;
  }
  if (!unit && !__all_sync(0xffffffffu, !in || (PivKey<T>::safe(d) && quotient_safe(pre)))) {
    y = y0;
#pragma unroll 1
    for (int s = 0; s < bw; ++s) {
      const int k = fwd ? s : bw - 1 - s;
      if (l == k) y = y / d;
      __syncwarp();
      const T x = __shfl_sync(0xffffffffu, y, k, W);
      if (in && (fwd ? l > k : l < k)) y = fma(-t[k], x, y);
      __syncwarp();
    }
  }
  return y;
}

}  // namespace lm
