// A panel step on the columns outside the panel: the panel's row
// interchanges (rawSwapRows, K.hs:1507-1537, fromCol = 0) and, right of the
// panel, U12 = L11^-1 A12 (rawTriSolvePanelTrail, LU.hs:364-407).
//
// One CTA per 32 columns.  Every row that changes place is read once into
// shared memory (the w pivot rows to their place in the block, at most as
// many displaced rows beside it) and written once.  Right of the panel the
// block is solved before it is written: 32-row steps, one warp substituting
// with the 32 x 32 diagonal triangle (a lane per column), then all warps
// subtracting the step from the rows below (DMMA for FP64, FFMA for FP32).
// L11 streams through two shared-memory buffers, 32 columns ahead of use.
// Bound by the substitution's latency chain (4 x about 1 us); the product
// with an explicit inverse that it replaces needed a 20 us inversion, a pass
// of its own for the interchanges (21 us at n = 8192) and a 22 us GEMM.
#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace lm {

namespace {

constexpr int kRbThreads = 256, kRbWarps = kRbThreads / 32;
constexpr int kRbCols = 32;
constexpr int kRbMaxW = 128;

template <typename T>
struct RbCfg {
  static constexpr int LDX = 36;                       // block row stride (DMMA operand reads conflict-free)
  static constexpr int LDL = 32 + 16 / (int)sizeof(T);  // L buffer row stride: 16-byte rows
  static constexpr int XB = kRbMaxW * LDX, LB = kRbMaxW * LDL;
  static constexpr int SMEM = (XB + 2 * LB) * (int)sizeof(T) + (2 * kRbMaxW + kRbMaxW) * (int)sizeof(int);
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// rows [r0, w) x 32 columns from column r0 of the panel's diagonal block
template <typename T>
__device__ __forceinline__ void load_l(T* buf, const T* L, long long lda, int r0, int w) {
  constexpr int V = 16 / (int)sizeof(T), CH = 32 / V;
  for (int e = threadIdx.x; e < (w - r0) * CH; e += kRbThreads) {
    const int r = e / CH, c = (e % CH) * V;
    cp_async16(buf + r * RbCfg<T>::LDL + c, L + (long long)(r0 + r) * lda + r0 + c);
  }
}

template <typename T>
__global__ void __launch_bounds__(kRbThreads, 2)
    row_block_kernel(T* A, long long lda, const int* __restrict__ plan, int n, int k0, int w, int ca0, int ca1, int cb0,
                     int cb1, int ablocks, int* status) {
  using Cfg = RbCfg<T>;
  extern __shared__ __align__(16) unsigned char sm[];
  T* X = reinterpret_cast<T*>(sm);
  T* Lb = X + Cfg::XB;        // two buffers
  T* stage = Lb + Cfg::LB;  // displaced rows (at most w x 32), before the second L buffer is filled
  int* src = reinterpret_cast<int*>(Lb + 2 * Cfg::LB);  // [w] where the block's rows come from
  int* od = src + kRbMaxW;                              // [w] other destinations
  int* os = od + kRbMaxW;                               // [w] their sources
  __shared__ int others;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool solve = (int)blockIdx.x >= ablocks;
  const int col0 = solve ? cb0 + ((int)blockIdx.x - ablocks) * kRbCols : ca0 + (int)blockIdx.x * kRbCols;
  const int nc = min(kRbCols, (solve ? cb1 : ca1) - col0);
  const T* L11 = A + (long long)k0 * lda + k0;
  if (solve) {
    load_l<T>(Lb, L11, lda, 0, w);
    cp_async_commit();
  }
  if (tid == 0) others = 0;
  if (tid < w) src[tid] = k0 + tid;
  __syncthreads();
  const int m = min(__ldg(plan), kSwapPlanRows);
  for (int e = tid; e < m; e += kRbThreads) {
    const int d = __ldg(plan + 1 + e), s = __ldg(plan + 1 + kSwapPlanRows + e);
    // the panel moves rows [k0, n) only: anything else is recorded and left out
    if (min(d, s) < k0 || max(d, s) >= n) {
      atomicCAS(status, 0, LM_DEVERR_BOUNDS);
    } else if (d < k0 + w) {
      src[d - k0] = s;
    } else {
      const int at = atomicAdd(&others, 1);  // a displaced row comes from the block: at most w of them
      if (at < kRbMaxW) {
        od[at] = d;
        os[at] = s;
      }
    }
  }
  __syncthreads();
  const int no = min(others, kRbMaxW);
  T* Ac = A + col0 + lane;
  const bool on = lane < nc;
  // (16 loads in flight per lane, then their stores: the row lists and the
  // block are both shared memory, and an interleaved loop would wait for each load)
  {
    T v[kRbMaxW / kRbWarps];
#pragma unroll
    for (int i = 0; i < kRbMaxW / kRbWarps; ++i) {
      const int r = warp + i * kRbWarps;
      v[i] = on && r < w ? Ac[(long long)src[r] * lda] : T(0);
    }
#pragma unroll
    for (int i = 0; i < kRbMaxW / kRbWarps; ++i) X[(warp + i * kRbWarps) * Cfg::LDX + lane] = v[i];
#pragma unroll
    for (int i = 0; i < kRbMaxW / kRbWarps; ++i) {
      const int r = warp + i * kRbWarps;
      v[i] = on && r < no ? Ac[(long long)os[r] * lda] : T(0);
    }
#pragma unroll
    for (int i = 0; i < kRbMaxW / kRbWarps; ++i) stage[(warp + i * kRbWarps) * 32 + lane] = v[i];
  }
  __syncthreads();
#pragma unroll 8
  for (int i = warp; i < no; i += kRbWarps)
    if (on) Ac[(long long)od[i] * lda] = stage[i * 32 + lane];
  if (!solve) {
    for (int i = warp; i < w; i += kRbWarps)
      if (on && src[i] != k0 + i) Ac[(long long)(k0 + i) * lda] = X[i * Cfg::LDX + lane];
    return;
  }
  __syncthreads();  // the staging is free for the second L buffer
  for (int r0 = 0, b = 0; r0 < w; r0 += 32, b ^= 1) {
    if (r0 + 32 < w) {
      load_l<T>(Lb + (b ^ 1) * Cfg::LB, L11, lda, r0 + 32, w);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const T* L = Lb + b * Cfg::LB;
    const int bw = min(32, w - r0);
    if (warp == 0) {  // X[r0 ..] <- inv(L_bb) X[r0 ..], lane = column
      T v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = i < bw ? X[(r0 + i) * Cfg::LDX + lane] : T(0);
#pragma unroll
      for (int k = 0; k < 32; ++k)  // by columns: the updates of one step are independent
#pragma unroll
        for (int i = k + 1; i < 32; ++i) v[i] = fma(-L[i * Cfg::LDL + k], v[k], v[i]);
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (i < bw) X[(r0 + i) * Cfg::LDX + lane] = v[i];
    }
    __syncthreads();
    const int below = w - r0 - 32;
    if (below > 0) {  // (bw = 32 here)
      if constexpr (sizeof(T) == 8) {
        const int gq = lane >> 2, tq = lane & 3;
        const int mt = (below + 15) / 16;
        for (int t = warp; t < mt * 2; t += kRbWarps) {  // 16 rows x 16 columns each
          const int i0 = r0 + 32 + (t >> 1) * 16, j0 = (t & 1) * 16;
          double acc[2][4];
#pragma unroll
          for (int ni = 0; ni < 2; ++ni)
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const int r = i0 + gq + (h >> 1) * 8;
              acc[ni][h] = r < w ? X[r * Cfg::LDX + j0 + ni * 8 + 2 * tq + (h & 1)] : 0.0;
            }
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 32; k += 4) {
            double a[2], bb[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int r = i0 + gq + h * 8;
              a[h] = r < w ? -L[(r - r0) * Cfg::LDL + k + tq] : 0.0;
            }
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) bb[ni] = X[(r0 + k + tq) * Cfg::LDX + j0 + ni * 8 + gq];
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) dmma_16x8x4(acc[ni], a[0], a[1], bb[ni]);
          }
#pragma unroll
          for (int ni = 0; ni < 2; ++ni)
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const int r = i0 + gq + (h >> 1) * 8;
              if (r < w) X[r * Cfg::LDX + j0 + ni * 8 + 2 * tq + (h & 1)] = acc[ni][h];
            }
        }
      } else {
        for (int i0 = r0 + 32 + warp * 4; i0 < w; i0 += kRbWarps * 4) {  // 4 rows x 32 columns each
          T acc[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[i] = i0 + i < w ? X[(i0 + i) * Cfg::LDX + lane] : T(0);
#pragma unroll 8
          for (int k = 0; k < 32; ++k) {
            const T xv = X[(r0 + k) * Cfg::LDX + lane];
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] = fma(-L[(min(i0 + i, w - 1) - r0) * Cfg::LDL + k], xv, acc[i]);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (i0 + i < w) X[(i0 + i) * Cfg::LDX + lane] = acc[i];
        }
      }
    }
    __syncthreads();
  }
  for (int i = warp; i < w; i += kRbWarps)
    if (on) Ac[(long long)(k0 + i) * lda] = X[i * Cfg::LDX + lane];
}

}  // namespace

template <typename T>
int row_block(T* A, long long lda, const int* plan, int n, int k0, int w, int ca0, int ca1, int cb0, int cb1,
              int* status, cudaStream_t st) {
  if (w <= 0) return LM_OK;
  if (w > kRbMaxW) return LM_ERR_ARG;
  const int ablocks = cdiv(std::max(0, ca1 - ca0), kRbCols), bblocks = cdiv(std::max(0, cb1 - cb0), kRbCols);
  if (ablocks + bblocks == 0) return LM_OK;
  // a narrower block only ends a matrix, where nothing is right of it
  if (bblocks > 0 && w != kRbMaxW) return LM_ERR_ARG;
  static bool attr_set[kMaxDevices] = {};
  int dev = 0;
  LM_CUDA_TRY(cudaGetDevice(&dev));
  if (!attr_set[dev]) {
    LM_CUDA_TRY(cudaFuncSetAttribute(row_block_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, RbCfg<T>::SMEM));
    attr_set[dev] = true;
  }
  row_block_kernel<T><<<ablocks + bblocks, kRbThreads, RbCfg<T>::SMEM, st>>>(
      A, lda, plan, n, k0, w, ca0, ca1, cb0, cb1, ablocks, status);
  count_launch(1);
  LM_CUDA_TRY(cudaGetLastError());
  return LM_OK;
}

template int row_block<double>(double*, long long, const int*, int, int, int, int, int, int, int, int*, cudaStream_t);
template int row_block<float>(float*, long long, const int*, int, int, int, int, int, int, int, int*, cudaStream_t);

}  // namespace lm
