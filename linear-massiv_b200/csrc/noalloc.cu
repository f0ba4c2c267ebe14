// lm_dpotrf_noalloc: the Cholesky factorisation without any device allocation, for
// callers that cannot allocate device memory at call time — code running where
// cudaMalloc is unavailable or forbidden (inside a memory-pool-managed runtime
// that owns every allocation, a real-time loop with a no-allocation rule, a plugin
// host that hands out only pre-registered buffers).
//
// The factorisation itself needs no scratch; its two status words are a file-scope
// array of this library.  CUDA loads a library's device code lazily by default, so
// the array is reserved on a device when the first call there looks up its address
// (a call with n = 0 does only that).
#include <mutex>

#include "common.cuh"
#include "internal.h"

namespace {

// Largest n this entry point accepts.  No buffer is sized by it any more; it stays
// because refusing larger orders is part of the documented interface.
constexpr int kNoAllocMaxN = 4096;

static __device__ __align__(256) int g_noalloc_status[64];  // [0, 2): error, info

std::mutex g_setup_mu;
int* g_status_dev[lm::kMaxDevices] = {};  // device address of the array, per device
int g_num_sms[lm::kMaxDevices] = {};

// Once per device, with that device current: the array's device address.
// (In host code `g_noalloc_status` names a host-side stand-in, not device
// memory, so it must never be passed to a kernel directly.)
int setup(int dev) {
  std::lock_guard<std::mutex> lock(g_setup_mu);
  if (g_status_dev[dev]) return LM_OK;
  void* p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_status);
  if (e != cudaSuccess || !p) {
    lm::set_last_error(std::string("cudaGetSymbolAddress(g_noalloc_status) failed: ") + cudaGetErrorString(e));
    return LM_ERR_CUDA;
  }
  int sms = 0;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) {
    lm::set_last_error(std::string("cudaDeviceGetAttribute failed: ") + cudaGetErrorString(e));
    return LM_ERR_CUDA;
  }
  g_num_sms[dev] = sms;
  g_status_dev[dev] = static_cast<int*>(p);
  return LM_OK;
}

}  // namespace

extern "C" int lm_dpotrf_noalloc(void* stream, int n, double* A, int lda, int* info) {
  if (n < 0 || (n > 0 && (!A || lda < n))) return LM_ERR_ARG;
  if (n > kNoAllocMaxN) {
    lm::set_last_error("lm_dpotrf_noalloc: n = " + std::to_string(n) + " exceeds its limit of " +
                       std::to_string(kNoAllocMaxN));
    return LM_ERR_ARG;
  }
  if (n > 0 && ((reinterpret_cast<uintptr_t>(A) & 15) || (lda & 1))) {
    lm::set_last_error("lm_dpotrf_noalloc: A must be 16-byte aligned with an even leading dimension");
    return LM_ERR_UNSUPPORTED;
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= lm::kMaxDevices) return LM_ERR_CUDA;
  LM_TRY(setup(dev));  // also for n = 0: the warm-up call that reserves the array
  if (n == 0) {
    if (info) *info = 0;
    return LM_OK;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int* status = g_status_dev[dev];  // error word, info word; they must start at zero
  LM_CUDA_TRY(cudaMemsetAsync(status, 0, 2 * sizeof(int), st));
  LM_TRY(lm::dpotrf_borrowed(dev, g_num_sms[dev], st, n, A, lda, status));
  int h[2] = {0, 0};
  LM_CUDA_TRY(cudaMemcpyAsync(h, status, sizeof h, cudaMemcpyDeviceToHost, st));
  LM_CUDA_TRY(cudaStreamSynchronize(st));
  if (h[0] != 0) {
    lm::set_last_error("lm_dpotrf_noalloc: a bounded device-side wait timed out");
    return LM_ERR_TIMEOUT;
  }
  if (info) *info = h[1];
  return h[1];
}
