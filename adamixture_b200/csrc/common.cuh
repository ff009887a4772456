// Shared definitions for the adamixture_b200 CUDA library (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

#include "../../include/adamixture_b200.h"

#define ADX_CUDA_TRY(expr)                                    \
  do {                                                        \
    cudaError_t _e = (expr);                                  \
    if (_e != cudaSuccess) { adx_set_cuda_error(_e); return ADX_ERR_CUDA; } \
  } while (0)

#define ADX_LAUNCH_CHECK()                                    \
  do {                                                        \
    cudaError_t _e = cudaGetLastError();                      \
    if (_e != cudaSuccess) { adx_set_cuda_error(_e); return ADX_ERR_CUDA; } \
  } while (0)

// Last CUDA error seen by the library (thread-local), readable through adx_last_error().
void adx_set_cuda_error(cudaError_t e);
void adx_set_message(const char* msg);

namespace adx {

constexpr double E_CLAMP = 1e-5;    // E-step reconstruction clamp
constexpr double LL_CLAMP = 1e-10;  // log-likelihood clamp
constexpr double DOMAIN = 1e-5;     // P/Q domain clamp after a step

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Number of SMs of the current device (cached per device).
int sm_count();

// The 8 bytes at G + at of a matrix of `total` bytes, at any alignment, as the three aligned
// words that hold them; bytes past the matrix are 0xFF. Fetching and putting together are two
// steps, so that a fetch ahead of its use waits for nothing (a funnel shift right behind the
// loads cost the float32 log-likelihood a memory latency per packed quad: 11.3 against 9.7 ms).
struct Words8 {
  uint32_t w0, w1, w2, sh;
  __device__ __forceinline__ uint64_t bytes() const {
    return (uint64_t)__funnelshift_r(w0, w1, sh) | ((uint64_t)__funnelshift_r(w1, w2, sh) << 32);
  }
};
__device__ __forceinline__ Words8 fetch8(const uint8_t* __restrict__ G, int64_t total, int64_t at) {
  const uint8_t* p = G + at;
  Words8 w;
  w.sh = 8u * (uint32_t)(reinterpret_cast<uintptr_t>(p) & 3);
  const uint8_t* q = p - (w.sh >> 3);
  if (q >= G && at + 12 <= total) {
    w.w0 = __ldg(reinterpret_cast<const uint32_t*>(q));
    w.w1 = __ldg(reinterpret_cast<const uint32_t*>(q + 4));
    w.w2 = __ldg(reinterpret_cast<const uint32_t*>(q + 8));
  } else {
    uint64_t v = 0;
    for (int b = 0; b < 8; ++b) v |= (uint64_t)(at + b < total ? __ldg(p + b) : (uint8_t)0xFF) << (8 * b);
    w.w0 = (uint32_t)v;
    w.w1 = (uint32_t)(v >> 32);
    w.w2 = 0;
    w.sh = 0;
  }
  return w;
}

__device__ __forceinline__ unsigned genotype(uint32_t byte, int s) { return (byte >> (2 * s)) & 3u; }

}  // namespace adx
