// Product of the centred genotype matrix with a skinny float32 factor without a workspace:
//
//   rows:  Y[M][L] = Xc . B      (B [N][L])      svd_gpu.py:106, 138 (proj = X @ orth)
//
// Xc[j][i] = g_ji - 2 f_j, 0 where missing (adamixture/src/utils_c/cuda/pack2bit.cu:46-77).
// The entry point for callers that give no workspace; with one, the product runs on the
// integer tensor cores (rsvd_tc.cu), about 10 times as fast.
//
// 256 threads = 64 groups of OP SNPs (OP = 8 while L <= 32, else 4) x 4 groups of C = LP/4
// factor columns; each thread keeps an OP x C float32 tile of the output in registers and
// walks the samples in chunks staged in shared memory (factor rows of the chunk, decoded
// genotype block of 32 KB). A thread's own SNPs are OP/4 runs of 4 spaced 256 apart, so each
// 16-byte load of the decoded block covers 512 contiguous bytes across the warp (no bank
// conflicts); shared loads per FMA are about 1/C + 1/OP. L <= 80 (LP = L rounded up to 4).
#include "common.cuh"

namespace adx {
namespace rsvd {

constexpr int TPB = 256;
constexpr int OG = 64;        // own groups
constexpr int CG = 4;         // column groups
constexpr int LMAX = 80;
constexpr int XS_FLOATS = 8192;  // decoded block: 32 KB

// own indices per thread for C columns per thread
__host__ __device__ constexpr int own_per_thread(int C) { return C <= 8 ? 8 : 4; }

__device__ __forceinline__ float centred(uint32_t byte, int s, float two_f) {
  const uint32_t g = (byte >> (2 * s)) & 3u;
  return g == 3u ? 0.0f : (float)g - two_f;
}

// own index of (thread group og, run v, slot q)
__device__ __forceinline__ int own_of(int og, int v, int q) { return v * (OG * 4) + og * 4 + q; }

// Y[j][:] = sum_i Xc[j][i] B[i][:] for the OWN SNPs of this CTA.
template <int C>  // columns per thread = LP / 4
__global__ void __launch_bounds__(TPB) rows_kernel(const uint8_t* __restrict__ G, int64_t M, int64_t N,
                                                   const float* __restrict__ f, const float* __restrict__ B,
                                                   int L, float* __restrict__ Y) {
  constexpr int LP = C * CG, OP = own_per_thread(C), OWN = OG * OP, CHK = XS_FLOATS / OWN;
  __shared__ __align__(16) float xs[CHK][OWN];   // [sample][snp]
  __shared__ __align__(16) float bs[CHK][LP];
  __shared__ float tf[OWN];
  const int tid = threadIdx.x, og = tid & (OG - 1), cg = tid / OG;
  const int64_t j0 = (int64_t)blockIdx.x * OWN;
  for (int t = tid; t < OWN; t += TPB) {
    const int64_t j = j0 + t;
    tf[t] = j < M ? 2.0f * f[j] : 0.0f;
  }
  float acc[OP][C];
#pragma unroll
  for (int a = 0; a < OP; ++a)
#pragma unroll
    for (int c = 0; c < C; ++c) acc[a][c] = 0.0f;
  const int64_t rows = (M + 3) >> 2;
  for (int64_t i0 = 0; i0 < N; i0 += CHK) {
    __syncthreads();
    for (int e = tid; e < CHK * LP; e += TPB) {
      const int s = e / LP, l = e - s * LP;
      const int64_t i = i0 + s;
      bs[s][l] = (i < N && l < L) ? B[i * L + l] : 0.0f;
    }
    // OWN/4 packed rows x CHK samples: one byte gives 4 SNPs of one sample
    for (int e = tid; e < (OWN / 4) * CHK; e += TPB) {
      const int pr = e / CHK, s = e - pr * CHK;
      const int64_t row = (j0 >> 2) + pr, i = i0 + s;
      const uint32_t byte = (row < rows && i < N) ? (uint32_t)G[row * N + i] : 0xFFu;
#pragma unroll
      for (int q = 0; q < 4; ++q) xs[s][pr * 4 + q] = centred(byte, q, tf[pr * 4 + q]);
    }
    __syncthreads();
    const int smax = (int)min((int64_t)CHK, N - i0);
    for (int s = 0; s < smax; ++s) {
      float x[OP];
#pragma unroll
      for (int v = 0; v < OP / 4; ++v) {
        const float4 x4 = *reinterpret_cast<const float4*>(&xs[s][own_of(og, v, 0)]);
        x[4 * v] = x4.x; x[4 * v + 1] = x4.y; x[4 * v + 2] = x4.z; x[4 * v + 3] = x4.w;
      }
      float b[C];
#pragma unroll
      for (int c = 0; c < C; ++c) b[c] = bs[s][cg * C + c];
#pragma unroll
      for (int a = 0; a < OP; ++a)
#pragma unroll
        for (int c = 0; c < C; ++c) acc[a][c] = fmaf(x[a], b[c], acc[a][c]);
    }
  }
#pragma unroll
  for (int a = 0; a < OP; ++a) {
    const int64_t j = j0 + own_of(og, a >> 2, a & 3);
    if (j >= M) continue;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int l = cg * C + c;
      if (l < L) Y[j * L + l] = acc[a][c];
    }
  }
}

}  // namespace rsvd
}  // namespace adx

using namespace adx;

#define ADX_LP_SWITCH(L, X)                                                              \
  switch ((L + 3) / 4) {                                                                 \
    case 1: X(1) break;   case 2: X(2) break;   case 3: X(3) break;   case 4: X(4) break;   \
    case 5: X(5) break;   case 6: X(6) break;   case 7: X(7) break;   case 8: X(8) break;   \
    case 9: X(9) break;   case 10: X(10) break; case 11: X(11) break; case 12: X(12) break; \
    case 13: X(13) break; case 14: X(14) break; case 15: X(15) break; case 16: X(16) break; \
    case 17: X(17) break; case 18: X(18) break; case 19: X(19) break; default: X(20) break; \
  }

extern "C" int adx_rsvd_rows(const uint8_t* G, int64_t M, int64_t N, const float* f, const float* B, int L,
                             float* Y, void* stream) {
  if (!G || !f || !B || !Y || M <= 0 || N <= 0 || L < 1 || L > rsvd::LMAX) {
    adx_set_message("adx_rsvd_rows: bad argument");
    return ADX_ERR_ARG;
  }
  cudaStream_t st = as_stream(stream);
  const int64_t own = (int64_t)rsvd::OG * rsvd::own_per_thread((L + rsvd::CG - 1) / rsvd::CG);
  const unsigned blocks = (unsigned)ceil_div(M, own);
#define LAUNCH(C) rsvd::rows_kernel<C><<<blocks, rsvd::TPB, 0, st>>>(G, M, N, f, B, L, Y);
  ADX_LP_SWITCH(L, LAUNCH)
#undef LAUNCH
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}
