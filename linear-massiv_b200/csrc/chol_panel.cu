// One block column of the Cholesky factorisation (128 columns): the diagonal
// block, then the rows below it.
//
// potrf_block — Cholesky of one <= 128 x 128 diagonal block in shared memory, by
//   16-column panels (rawCholColumnSIMDFrom, K.hs:2137-2195, for a diagonal
//   panel).  One CTA and a chain of 128 columns, so what bounds it is the latency
//   of a column: shuffle, rsqrt, product, shuffle, multiply-add.  Only the 16 x 16
//   diagonal blocks are on that chain: one warp takes them in registers, the next
//   one while the other warps still apply the panel to the rest (DMMA).  Diagonal
//   blocks of 32 columns took twice the shuffles per column, and the update
//   waited for them: 60 to 66 us per block before, 29 us now.
// chol_rows — L21 = A21 L11^-T by substitution, 64 rows per CTA: 16 columns solved
//   by one thread per row, then applied to the columns right of them on the
//   tensor cores.  Half the arithmetic of a product with the inverse of L11, and
//   no inverse to wait for: per block column of n = 8192, on the 16 SMs
//   beside the trailing update, 32 us (inverse), 11 us (copy of A21) and 45 us
//   (product) on average before, 54 us now; up to 600 rows 54 and 14 us.
#include "common.cuh"
#include "internal.h"

namespace lm {

void count_launch(int n);

namespace {

constexpr int kCB = 128;       // block column
constexpr int kCW = 16;        // panel of it
constexpr int kCLd = kCB + 4;  // row stride: 16-byte rows, DMMA operand reads without conflicts
constexpr int kCThreads = 256;
constexpr int kCRows = 64;  // rows per CTA of chol_rows

// C -= X Y^T for the 16 x 16 block C by one warp, X and Y 16 x 16 (all in shared
// memory with row stride kCLd).
__device__ __forceinline__ void block16_update(double* C, const double* X, const double* Y) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double acc[2][4];
#pragma unroll
  for (int ni = 0; ni < 2; ++ni)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double2 v = *reinterpret_cast<const double2*>(C + (g + 8 * h) * kCLd + ni * 8 + 2 * t);
      acc[ni][2 * h] = v.x;
      acc[ni][2 * h + 1] = v.y;
    }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < kCW; k += 4) {
    const double a0 = -X[g * kCLd + k + t], a1 = -X[(g + 8) * kCLd + k + t];
#pragma unroll
    for (int ni = 0; ni < 2; ++ni) dmma_16x8x4(acc[ni], a0, a1, Y[(ni * 8 + g) * kCLd + k + t]);
  }
#pragma unroll
  for (int ni = 0; ni < 2; ++ni)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      *reinterpret_cast<double2*>(C + (g + 8 * h) * kCLd + ni * 8 + 2 * t) =
          make_double2(acc[ni][2 * h], acc[ni][2 * h + 1]);
}

// One row x of 16 entries (shared): x <- x L^-T with the 16 x 16 lower triangle L
// (row stride kCLd) and the reciprocals rd of its diagonal.
__device__ __forceinline__ void row16_solve(double* x, const double* L, const double* rd) {
  double a[kCW];
#pragma unroll
  for (int c = 0; c < kCW; c += 2) {
    const double2 v = *reinterpret_cast<const double2*>(x + c);
    a[c] = v.x;
    a[c + 1] = v.y;
  }
#pragma unroll
  for (int k = 0; k < kCW; ++k) {
    a[k] *= rd[k];
#pragma unroll
    for (int j = k + 1; j < kCW; ++j) a[j] = fma(-a[k], L[j * kCLd + k], a[j]);
  }
#pragma unroll
  for (int c = 0; c < kCW; c += 2) *reinterpret_cast<double2*>(x + c) = make_double2(a[c], a[c + 1]);
}

// Cholesky of the 16 x 16 block at D (row stride kCLd) by one warp, lane and lane
// + 16 holding the same row; the reciprocals of the diagonal to rd.  Returns the
// first column whose pivot is not positive, or -1 (the arithmetic continues,
// leaving the NaN the reference's would).  Entries above the diagonal are never
// used.
__device__ __forceinline__ int diag16(double* D, double* rd) {
  const int lane = threadIdx.x & 15;
  double d[kCW];
  double* row = D + lane * kCLd;
  __syncwarp();
#pragma unroll
  for (int c = 0; c < kCW; c += 2) {
    const double2 v = *reinterpret_cast<const double2*>(row + c);
    d[c] = v.x;
    d[c + 1] = v.y;
  }
  int bad = -1;
  double myr = 0.0;
#pragma unroll
  for (int k = 0; k < kCW; ++k) {
    const double p = __shfl_sync(0xffffffffu, d[k], k);
    bad = bad < 0 && !(p > 0.0) ? k : bad;
    const double r = rsqrt(p);
    const double l = d[k] * r;
    d[k] = lane >= k ? l : d[k];
    myr = lane == k ? r : myr;
#pragma unroll
    for (int j = k + 1; j < kCW; ++j) d[j] = fma(-l, __shfl_sync(0xffffffffu, l, j), d[j]);
  }
  if ((threadIdx.x & 31) < kCW) {
    rd[lane] = myr;
#pragma unroll
    for (int c = 0; c < kCW; ++c)
      if (c <= lane) row[c] = d[c];
  }
  __syncwarp();
  return bad;
}

constexpr size_t kPotrfSmem = sizeof(double) * (kCB * kCLd + kCB);

__global__ void __launch_bounds__(kCThreads) potrf_block_kernel(double* A, long long lda, int w, int base,
                                                               int* status) {
  extern __shared__ __align__(16) unsigned char pb_smem[];
  double* S = reinterpret_cast<double*>(pb_smem);  // kCB x kCLd
  double* rd = S + kCB * kCLd;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int np = (w + kCW - 1) / kCW, wp = np * kCW;  // padded with the identity
#pragma unroll 4
  for (int i = warp; i < wp; i += kCThreads / 32)
#pragma unroll
    for (int q = 0; q < kCB / 32; ++q) {
      const int j = q * 32 + lane;
      if (j < wp) S[i * kCLd + j] = j <= i && i < w ? A[(long long)i * lda + j] : (i == j ? 1.0 : 0.0);
    }
  __syncthreads();
  auto diag = [&](int c0) {  // warp 0
    const int bad = diag16(S + c0 * kCLd + c0, rd + c0);
    if (lane == 0 && bad >= 0 && c0 + bad < w) atomicCAS(status + 1, 0, base + c0 + bad + 1);
  };
  if (warp == 0) diag(0);
  __syncthreads();
#pragma unroll 1
  for (int c0 = 0; c0 + kCW < wp; c0 += kCW) {
    const int r0 = c0 + kCW, m = wp - r0;
    if (tid < m) row16_solve(S + (r0 + tid) * kCLd + c0, S + c0 * kCLd + c0, rd + c0);
    __syncthreads();
    // the lower triangle of the rest, 16 x 16 blocks; warp 0 takes the next
    // diagonal block and factors it
    auto block = [&](int bi, int bj) {
      block16_update(S + (r0 + bi * kCW) * kCLd + r0 + bj * kCW, S + (r0 + bi * kCW) * kCLd + c0,
                     S + (r0 + bj * kCW) * kCLd + c0);
    };
    if (warp == 0) {
      block(0, 0);
      diag(r0);
    } else {
      const int nb = m / kCW, blocks = nb * (nb + 1) / 2;
      int bi = 0, bj = warp;
      for (int t = warp; t < blocks; t += kCThreads / 32 - 1, bj += kCThreads / 32 - 1) {
        while (bj > bi) bj -= ++bi;
        block(bi, bj);
      }
    }
    __syncthreads();
  }
#pragma unroll 4
  for (int i = warp; i < w; i += kCThreads / 32)
#pragma unroll
    for (int q = 0; q < kCB / 32; ++q) {
      const int j = q * 32 + lane;
      if (j <= i) A[(long long)i * lda + j] = S[i * kCLd + j];
    }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

constexpr size_t kRowsSmem = sizeof(double) * ((kCB + kCRows) * kCLd + kCB);

// A21 (R x 128 below the factored diagonal block L11, same columns) <- A21 L11^-T.
__global__ void __launch_bounds__(kCThreads, 1) chol_rows_kernel(const double* L11, double* A21, long long lda, int R) {
  extern __shared__ __align__(16) unsigned char cr_smem[];
  double* L = reinterpret_cast<double*>(cr_smem);  // kCB x kCLd, lower triangle
  double* X = L + kCB * kCLd;                      // kCRows x kCLd
  double* rd = X + kCRows * kCLd;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* Ab = A21 + (long long)blockIdx.x * kCRows * lda;
  const int rows = min(kCRows, R - (int)blockIdx.x * kCRows);
#pragma unroll 4
  for (int i = warp; i < kCB; i += kCThreads / 32)
#pragma unroll
    for (int q = 0; q < kCB; q += 64) {
      const int j = q + 2 * lane;  // (up to the 16-column block of the diagonal)
      if (j <= (i | (kCW - 1))) cp_async16(L + i * kCLd + j, L11 + (long long)i * lda + j);
    }
#pragma unroll 4
  for (int i = warp; i < rows; i += kCThreads / 32)
#pragma unroll
    for (int q = 0; q < kCB; q += 64) cp_async16(X + i * kCLd + q + 2 * lane, Ab + (long long)i * lda + q + 2 * lane);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (tid < kCB) rd[tid] = 1.0 / L[tid * kCLd + tid];
  __syncthreads();
#pragma unroll 1
  for (int c0 = 0; c0 < kCB; c0 += kCW) {
    if (tid < rows) row16_solve(X + tid * kCLd + c0, L + c0 * kCLd + c0, rd + c0);
    __syncthreads();
    if (c0 + kCW == kCB) break;
    // columns right of it, 16 x 16 blocks (rows past `rows` hold nothing that is stored)
    const int nb = (kCB - c0) / kCW - 1, units = nb * ((rows + kCW - 1) / kCW);
    for (int u = warp; u < units; u += kCThreads / 32) {
      const int q0 = c0 + kCW + (u % nb) * kCW, r0 = (u / nb) * kCW;
      block16_update(X + r0 * kCLd + q0, X + r0 * kCLd + c0, L + q0 * kCLd + c0);
    }
    __syncthreads();
  }
#pragma unroll 4
  for (int i = warp; i < rows; i += kCThreads / 32)
#pragma unroll
    for (int q = 0; q < kCB; q += 64)
      *reinterpret_cast<double2*>(Ab + (long long)i * lda + q + 2 * lane) =
          *reinterpret_cast<const double2*>(X + i * kCLd + q + 2 * lane);
}

template <typename K>
int set_smem(K kern, bool (&done)[kMaxDevices], int dev, size_t bytes) {
  if (!done[dev]) {
    LM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    done[dev] = true;
  }
  return LM_OK;
}

}  // namespace

int potrf_block(Ctx& c, double* A, long long lda, int w, int base, cudaStream_t st) {
  if (w <= 0) return LM_OK;
  if (w > kCB) return LM_ERR_ARG;
  static bool attr_set[kMaxDevices] = {};
  LM_TRY(set_smem(potrf_block_kernel, attr_set, ctx_device(c), kPotrfSmem));
  potrf_block_kernel<<<1, kCThreads, kPotrfSmem, st>>>(A, lda, w, base, ctx_status(c));
  count_launch(1);
  LM_CUDA_TRY(cudaGetLastError());
  return LM_OK;
}

int chol_rows(Ctx& c, double* A11, long long lda, int R, cudaStream_t st) {
  if (R <= 0) return LM_OK;
  if ((reinterpret_cast<uintptr_t>(A11) & 15) || (lda & 1)) return LM_ERR_ARG;
  static bool attr_set[kMaxDevices] = {};
  LM_TRY(set_smem(chol_rows_kernel, attr_set, ctx_device(c), kRowsSmem));
  chol_rows_kernel<<<cdiv(R, kCRows), kCThreads, kRowsSmem, st>>>(A11, A11 + kCB * lda, lda, R);
  count_launch(1);
  LM_CUDA_TRY(cudaGetLastError());
  return LM_OK;
}

}  // namespace lm
