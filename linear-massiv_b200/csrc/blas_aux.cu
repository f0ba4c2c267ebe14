// Row interchanges, triangular block solves, copies and the FP64 residual.
//
// laswp_*    : applyPivotsForward (LU.hs:493-507) on right-hand sides, as one
//              composed permutation.
// trsm_left  : the diagonal blocks of the substitutions with several right-hand
//              sides (rawForwardSubUnitPackedSIMD, rawBackSubPackedSIMD,
//              rawForwardSubCholPackedSIMD and rawBackSubCholTPackedSIMD,
//              K.hs:2205-2430).
// dresidual  : r = b - A x in FP64, the GEMV of matvecP / rawGemv
//              (L2.hs:131-139, K.hs:119-134) on the refinement path.
#include <climits>

#include "common.cuh"
#include "internal.h"
#include "pivot.cuh"

namespace lm {

void count_launch(int n);

namespace {

// All interchanges ipiv[0..n) on a narrow block B (n x nrhs) at once:
// W(i, :) = B(sigma(i), :) with sigma(i) = tau_0(tau_1(... tau_{n-1}(i))),
// tau_k the transposition (k, ipiv[k]).  Thread i walks the swap list
// backwards (ipiv staged through shared memory, read as broadcasts), so the
// n sequential swaps of applyPivotsForward (LU.hs:493-507) become one
// parallel gather; an out-of-range pivot row records LM_DEVERR_BOUNDS.
template <typename T>
__global__ void __launch_bounds__(128) perm_gather_kernel(const T* __restrict__ B, long long ldb, int n, int nrhs,
                                                          const int* __restrict__ ipiv, T* W, long long ldw,
                                                          int* status) {
  constexpr int CH = 4096;
  __shared__ int sp[CH];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int r = i;
  bool bad = false;
  for (int c0 = ((n - 1) / CH) * CH; c0 >= 0; c0 -= CH) {
    const int cnt = min(CH, n - c0);
    __syncthreads();
    for (int e = threadIdx.x; e < cnt; e += blockDim.x) sp[e] = __ldg(ipiv + c0 + e);
    __syncthreads();
#pragma unroll 8
    for (int k = cnt - 1; k >= 0; --k) {
      const int p = sp[k];
      const int kk = c0 + k;
      r = (r == kk) ? p : ((r == p) ? kk : r);
    }
  }
  if (i < n) {
    if (r < 0 || r >= n) bad = true;
    if (bad) {
      atomicCAS(status, 0, LM_DEVERR_BOUNDS);
      r = i;
    }
    for (int c = 0; c < nrhs; ++c) W[(long long)i * ldw + c] = B[(long long)r * ldb + c];
  }
}

// sigma of the swap list ipiv[0..n) (as perm_gather_kernel walks it), once
// per factorisation: perm[i] = sigma(i), so that every later application of
// the interchanges to a right-hand side (applyPivotsForward, LU.hs:493-507)
// is a plain gather; an out-of-range pivot row records LM_DEVERR_BOUNDS and
// maps i to itself.
__global__ void __launch_bounds__(128) perm_from_swaps_kernel(const int* __restrict__ ipiv, int n, int* perm,
                                                              int* status) {
  constexpr int CH = 4096;
  __shared__ int sp[CH];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int r = i;
  for (int c0 = ((n - 1) / CH) * CH; c0 >= 0; c0 -= CH) {
    const int cnt = min(CH, n - c0);
    __syncthreads();
    for (int e = threadIdx.x; e < cnt; e += blockDim.x) sp[e] = __ldg(ipiv + c0 + e);
    __syncthreads();
#pragma unroll 8
    for (int k = cnt - 1; k >= 0; --k) {
      const int p = sp[k];
      const int kk = c0 + k;
      r = (r == kk) ? p : ((r == p) ? kk : r);
    }
  }
  if (i < n) {
    if (r < 0 || r >= n) {
      atomicCAS(status, 0, LM_DEVERR_BOUNDS);
      r = i;
    }
    perm[i] = r;
  }
}

// W(i, :) = B(perm[i], :) for a narrow block (n x nrhs).
template <typename T>
__global__ void gather_rows_kernel(const T* __restrict__ B, long long ldb, int n, int nrhs,
                                   const int* __restrict__ perm, T* W, long long ldw) {
  const long long total = (long long)n * nrhs;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e / nrhs), c = (int)(e % nrhs);
    W[(long long)i * ldw + c] = B[(long long)__ldg(perm + i) * ldb + c];
  }
}

// op(Tri) X = B for 8 columns of B per CTA (w <= 128): the block solves of the
// substitutions with more than a few right-hand sides.  One launch after the
// other, so latency bounds it: op(Tri) is staged whole (row stride 129, so that
// a warp reads a column of it without conflicts), a thread keeps its row of B
// (4 of the 8 columns) in registers, and the rows are solved in blocks of 32:
//   solve  : warp h takes column h of the block, lane = row (tri_sweep);
//   update : every thread applies the 32 solved entries to its row.
// w = 128 with 64 columns: 86 us before (16-row blocks solved by one warp that
// read every operand of its serial sums from shared memory), 17 us now, of which
// 3 us bring the triangle in (11 us when it came through registers); 33 us with a
// branch per step in the sweeps.
constexpr int kTrsmLd = 129, kTrsmCols = 8;
constexpr size_t kTrsmSmem = sizeof(double) * (128 * kTrsmLd + 128 + 2 * 32 * kTrsmCols);

__global__ void __launch_bounds__(256) trsm_left_kernel(const double* __restrict__ Tri, long long ldt, int w, int lower,
                                                        int unit, int trans, double* B, long long ldb, int ncols) {
  extern __shared__ __align__(16) unsigned char sm[];
  const bool upper_op = (lower == 0) != (trans != 0);
  double* Ts = reinterpret_cast<double*>(sm);
  double* dr = Ts + 128 * kTrsmLd;  // reciprocals of the diagonal
  double* Xs = dr + 128;            // [2][32][8] the block being solved, by parity
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c0 = blockIdx.x * kTrsmCols;
  const int nc = min(kTrsmCols, ncols - c0);
  const int row = tid & 127, cg = (tid >> 7) * 4;  // this thread's row and columns of B
  // every entry of the triangle on its way at once
  for (int r = warp; r < w; r += 8) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = q * 32 + lane;
      if (c < w && (lower ? c <= r : c >= r))
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                         smem_u32(Ts + (trans ? c * kTrsmLd + r : r * kTrsmLd + c))),
                     "l"(Tri + (long long)r * ldt + c)
                     : "memory");
    }
  }
  double x[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) x[c] = row < w && cg + c < nc ? B[(long long)row * ldb + c0 + cg + c] : 0.0;
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (!unit && tid < w) dr[tid] = 1.0 / Ts[tid * kTrsmLd + tid];  // (read after the next barrier)
  const int nb = (w + 31) / 32;
  for (int bi = 0; bi < nb; ++bi) {
    const int r0 = (upper_op ? nb - 1 - bi : bi) * 32, bw = min(32, w - r0);
    double* X = Xs + (bi & 1) * 32 * kTrsmCols;
    if (row >= r0 && row < r0 + 32) {  // uniform in the warp
#pragma unroll
      for (int c = 0; c < 4; ++c) X[(row - r0) * kTrsmCols + cg + c] = x[c];
    }
    __syncthreads();
    if (warp < nc) {
      double y = X[lane * kTrsmCols + warp];
      const bool in = lane < bw;
      const double* trow = Ts + (in ? r0 + lane : r0) * kTrsmLd + r0;
      const double d = unit || !in ? 1.0 : trow[lane], rd = unit || !in ? 1.0 : dr[r0 + lane];
      y = tri_sweep<double, 32>(y, trow, d, rd, lane, bw, !upper_op, unit != 0);
      if (in) X[lane * kTrsmCols + warp] = y;
    }
    __syncthreads();
    if (row >= r0 && row < r0 + 32) {
#pragma unroll
      for (int c = 0; c < 4; ++c) x[c] = X[(row - r0) * kTrsmCols + cg + c];
    } else if (row < w && (upper_op ? row < r0 : row > r0)) {
      const double* trow = Ts + row * kTrsmLd + r0;
#pragma unroll 8
      for (int k = 0; k < bw; ++k) {
        const double t = trow[k];
        const double2 a = *reinterpret_cast<const double2*>(X + k * kTrsmCols + cg);
        const double2 b = *reinterpret_cast<const double2*>(X + k * kTrsmCols + cg + 2);
        x[0] = fma(-t, a.x, x[0]);
        x[1] = fma(-t, a.y, x[1]);
        x[2] = fma(-t, b.x, x[2]);
        x[3] = fma(-t, b.y, x[3]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
    if (row < w && cg + c < nc) B[(long long)row * ldb + c0 + cg + c] = x[c];
}

template <typename T>
__global__ void copy2d_kernel(T* dst, long long ldd, const T* src, long long lds, int rows, int cols) {
  const long long total = (long long)rows * cols;
#pragma unroll 4
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / cols), c = (int)(i % cols);
    dst[(long long)r * ldd + c] = src[(long long)r * lds + c];
  }
}

template <typename T>
__global__ void zero_upper_kernel(T* A, long long lda, int n) {
  const long long total = (long long)n * n;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / n), c = (int)(i % n);
    if (c > r) A[(long long)r * lda + c] = T(0);
  }
}

// One warp per row: r_i = b_i - sum_j a_ij x_j for up to 8 right-hand sides.
template <int NR>
__global__ void residual_kernel(int n, int nrhs, const double* __restrict__ A, long long lda,
                                const double* __restrict__ X, long long ldx, const double* __restrict__ B,
                                long long ldb, double* R, long long ldr) {
  const int warps = blockDim.x >> 5;
  const int row = blockIdx.x * warps + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= n) return;
  double acc[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) acc[r] = 0.0;
  const double* arow = A + (long long)row * lda;
#pragma unroll 8
  for (int j = lane; j < n; j += 32) {
    const double a = arow[j];
#pragma unroll
    for (int r = 0; r < NR; ++r)
      if (r < nrhs) acc[r] = fma(a, X[(long long)j * ldx + r], acc[r]);
  }
  __syncwarp();  // lanes leave the strided loop at different trip counts
#pragma unroll
  for (int r = 0; r < NR; ++r)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
  if (lane == 0) {
#pragma unroll
    for (int r = 0; r < NR; ++r)
      if (r < nrhs) R[(long long)row * ldr + r] = B[(long long)row * ldb + r] - acc[r];
  }
}

int grid_for(long long total, int threads, int sms) {
  long long g = cdivll(total, threads);
  return (int)std::max<long long>(1, std::min<long long>(g, 8LL * sms > 0 ? 8LL * sms : 1184));
}

}  // namespace

int perm_from_swaps(const int* ipiv, int n, int* perm, int* status, cudaStream_t st) {
  if (n <= 0) return LM_OK;
  perm_from_swaps_kernel<<<cdiv(n, 128), 128, 0, st>>>(ipiv, n, perm, status);
  count_launch(1);
  LM_CUDA_TRY(cudaGetLastError());
  return LM_OK;
}

template <typename T>
int laswp_perm(T* B, long long ldb, int n, int nrhs, const int* perm, T* W, cudaStream_t st) {
  if (n <= 0 || nrhs <= 0) return LM_OK;
  const long long total = (long long)n * nrhs;
  gather_rows_kernel<T><<<(int)std::min<long long>((total + 255) / 256, 4096), 256, 0, st>>>(B, ldb, n, nrhs, perm,
                                                                                            W, nrhs);
  count_launch(1);
  LM_CUDA_TRY(cudaGetLastError());
  return copy2d<T>(B, ldb, W, nrhs, n, nrhs, st);
}

template <typename T>
int laswp_narrow(T* B, long long ldb, int n, int nrhs, const int* ipiv, T* W, int* status, cudaStream_t st) {
  if (n <= 0 || nrhs <= 0) return LM_OK;
  perm_gather_kernel<T><<<cdiv(n, 128), 128, 0, st>>>(B, ldb, n, nrhs, ipiv, W, nrhs, status);
  count_launch(1);
  LM_CUDA_TRY(cudaGetLastError());
  return copy2d<T>(B, ldb, W, nrhs, n, nrhs, st);
}

int trsm_left(const double* Tri, long long ldt, int w, bool lower, bool unit, bool trans, double* B, long long ldb,
              int ncols, cudaStream_t st) {
  if (w <= 0 || ncols <= 0) return LM_OK;
  if (w > 128) return LM_ERR_ARG;
  static bool attr_set[kMaxDevices] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev]) {
    LM_CUDA_TRY(cudaFuncSetAttribute(trsm_left_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrsmSmem));
    attr_set[dev] = true;
  }
  trsm_left_kernel<<<cdiv(ncols, kTrsmCols), 256, kTrsmSmem, st>>>(Tri, ldt, w, lower ? 1 : 0, unit ? 1 : 0,
                                                                   trans ? 1 : 0, B, ldb, ncols);
  count_launch(1);
  LM_CUDA_TRY(cudaGetLastError());
  return LM_OK;
}

template <typename T>
int copy2d(T* dst, long long ldd, const T* src, long long lds, int rows, int cols, cudaStream_t st) {
  if (rows <= 0 || cols <= 0) return LM_OK;
  copy2d_kernel<T><<<grid_for((long long)rows * cols, 256, 148), 256, 0, st>>>(dst, ldd, src, lds, rows, cols);
  count_launch(1);
  LM_CUDA_TRY(cudaGetLastError());
  return LM_OK;
}

template <typename T>
int zero_upper(T* A, long long lda, int n, cudaStream_t st) {
  if (n <= 1) return LM_OK;
  zero_upper_kernel<T><<<grid_for((long long)n * n, 256, 148), 256, 0, st>>>(A, lda, n);
  count_launch(1);
  LM_CUDA_TRY(cudaGetLastError());
  return LM_OK;
}

int dresidual(Ctx& c, int n, int nrhs, const double* A, long long lda, const double* X, long long ldx,
              const double* B, long long ldb, double* R, long long ldr, cudaStream_t st) {
  if (nrhs <= 8) {
    const int warps = 8;
    residual_kernel<8><<<cdiv(n, warps), warps * 32, 0, st>>>(n, nrhs, A, lda, X, ldx, B, ldb, R, ldr);
    count_launch(1);
    LM_CUDA_TRY(cudaGetLastError());
    return LM_OK;
  }
  // Wide right-hand sides: R = B, then R -= A X on the tensor cores.
  const bool ok = !((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(X)) & 15) && !(lda & 1) &&
                  !(ldx & 1);
  const double* A2 = A;
  const double* X2 = X;
  long long lda2 = lda, ldx2 = ldx;
  if (!ok) {
    lda2 = (n + 7) / 8 * 8;
    ldx2 = (nrhs + 7) / 8 * 8;
    void* ws = nullptr;
    LM_TRY(ctx_workspace(c, 1, sizeof(double) * ((size_t)n * lda2 + (size_t)n * ldx2), &ws));
    double* a = static_cast<double*>(ws);
    double* x = a + (size_t)n * lda2;
    LM_TRY(copy2d<double>(a, lda2, A, lda, n, n, st));
    LM_TRY(copy2d<double>(x, ldx2, X, ldx, n, nrhs, st));
    A2 = a;
    X2 = x;
  }
  LM_TRY(copy2d<double>(R, ldr, B, ldb, n, nrhs, st));
  GemmDesc d;
  d.m = n; d.n = nrhs; d.k = n; d.alpha = -1.0; d.beta = 1.0;
  d.A = A2; d.lda = lda2; d.B = X2; d.ldb = ldx2; d.C = R; d.ldc = ldr;
  return dgemm(c, d, st);
}

template int laswp_narrow<double>(double*, long long, int, int, const int*, double*, int*, cudaStream_t);
template int laswp_perm<double>(double*, long long, int, int, const int*, double*, cudaStream_t);
template int laswp_perm<float>(float*, long long, int, int, const int*, float*, cudaStream_t);
template int copy2d<double>(double*, long long, const double*, long long, int, int, cudaStream_t);
template int copy2d<float>(float*, long long, const float*, long long, int, int, cudaStream_t);
template int zero_upper<double>(double*, long long, int, cudaStream_t);
template int zero_upper<float>(float*, long long, int, cudaStream_t);

}  // namespace lm
