// Packed-genotype layout kernels: decode, centring, per-SNP frequencies, per-sample counts,
// PLINK BED ingestion (decode + flip) and the synthetic cohort sampler.
//
// Packed layout: G[ceil(M/4)][N] uint8, byte (j>>2)*N + i holds SNP j of sample i in bits
// 2*(j&3) (adamixture/src/utils_c/cython/snp_reader.pyx:76-120). Consecutive samples are
// consecutive bytes, so every kernel here reads rows of G with consecutive threads on
// consecutive samples (coalesced), 16 bytes per thread where the row alignment allows.
#include "common.cuh"

namespace adx {

// ---------------------------------------------------------------- decode (pack2bit.cu:15-77)

__global__ void unpack_u8_kernel(const uint8_t* __restrict__ G, int64_t N, int64_t M_total,
                                 int64_t m_start, int64_t count, int64_t byte_offset,
                                 uint8_t* __restrict__ out) {
  const int64_t total = count * N;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t lm = idx / N, i = idx - lm * N;
    const int64_t j = m_start + lm;
    uint8_t v = 3;
    if (j < M_total && (j >> 2) >= byte_offset)
      v = (uint8_t)genotype(G[((j >> 2) - byte_offset) * N + i], (int)(j & 3));
    out[idx] = v;
  }
}

__global__ void unpack_center_kernel(const uint8_t* __restrict__ G, int64_t N, int64_t M_total,
                                     int64_t m_start, int64_t count, int64_t byte_offset,
                                     const float* __restrict__ f, float* __restrict__ out) {
  const int64_t total = count * N;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t lm = idx / N, i = idx - lm * N;
    const int64_t j = m_start + lm;
    float v = 0.0f;
    if (j < M_total && (j >> 2) >= byte_offset) {
      const unsigned g = genotype(G[((j >> 2) - byte_offset) * N + i], (int)(j & 3));
      v = g == 3u ? 0.0f : ((float)g - 2.0f * f[j]);
    }
    out[idx] = v;
  }
}

// ---------------------------------------------------------------- loads at any alignment

// A matrix of bytes [begin, end): rows of real cohorts start at any address, so the kernels
// below read whole aligned words and shift or mask. A word that would leave the matrix (its
// first or last few bytes) is put together from the bytes inside, with `fill` elsewhere.
struct Bytes {
  const uint8_t* begin;
  const uint8_t* end;
  __device__ __forceinline__ uint32_t word(const uint8_t* p, uint32_t fill) const {  // p 4-byte aligned
    if (p >= begin && p + 4 <= end) return __ldg(reinterpret_cast<const uint32_t*>(p));
    uint32_t w = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) w |= (p + b >= begin && p + b < end ? (uint32_t)__ldg(p + b) : fill) << (8 * b);
    return w;
  }
  __device__ __forceinline__ uint4 quad(const uint8_t* p, uint32_t fill) const {     // p 16-byte aligned
    if (p >= begin && p + 16 <= end) return __ldg(reinterpret_cast<const uint4*>(p));
    return make_uint4(word(p, fill), word(p + 4, fill), word(p + 8, fill), word(p + 12, fill));
  }
};

// Bytes of a word that starts `at` bytes from a range [0, n): 0xFF inside, 0 outside.
__device__ __forceinline__ uint32_t inside_mask(int64_t at, int64_t n) {
  uint32_t m = 0xFFFFFFFFu;
  if (at < 0) m = at <= -4 ? 0u : m << (8 * (uint32_t)(-at));
  if (at + 4 > n) m = at >= n ? 0u : m & (0xFFFFFFFFu >> (8 * (uint32_t)(at + 4 - n)));
  return m;
}

// ---------------------------------------------------------------- per-SNP frequencies

constexpr int FREQ_TPB = 256;

// TPR threads per packed row (4 SNPs): per SNP, the sum of the 2-bit codes and the number of
// missing entries (code 3), summed 16 samples at a time in nibbles from 16-byte loads; the dosage sum is
// the code sum less 3 per missing entry, exact in integers. Memory-bound: 1.25 GB in 0.40 ms
// at N=50,003 x M=100,001 (byte loads and 64-bit sums took 1.9 ms).
template <int TPR>
__global__ void __launch_bounds__(FREQ_TPB) allele_freq_kernel(const uint8_t* __restrict__ G, int64_t M, int64_t N,
                                                               float* __restrict__ f) {
  constexpr int RPB = FREQ_TPB / TPR;
  __shared__ unsigned long long part[TPR > 32 ? TPR / 32 : 1][8];
  const int64_t rows = (M + 3) >> 2;
  const int t = threadIdx.x % TPR, lane = threadIdx.x & 31;
  const Bytes all{G, G + rows * N};
  for (int64_t r0 = (int64_t)blockIdx.x * RPB; r0 < rows; r0 += (int64_t)gridDim.x * RPB) {
    const int64_t r = r0 + threadIdx.x / TPR;
    uint32_t sum[4] = {0, 0, 0, 0}, mis[4] = {0, 0, 0, 0};
    unsigned long long tot[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (r < rows) {
      const uint8_t* row = G + r * N;
      const int64_t lead = (int64_t)(reinterpret_cast<uintptr_t>(row) & 15);
      const int64_t quads = (lead + N + 15) >> 4;
      int since = 0;
#pragma unroll 4
      for (int64_t q = t; q < quads; q += TPR) {
        const int64_t at = 16 * q - lead;   // first sample of the 16
        const uint4 v = all.quad(row + at, 0u);
        uint32_t w[4] = {v.x, v.y, v.z, v.w};
        if (at < 0 || at + 16 > N) {
#pragma unroll
          for (int c = 0; c < 4; ++c) w[c] &= inside_mask(at + 4 * c, N);   // code 0: adds nothing
        }
        // the four words' codes summed in nibbles (at most 12), SNPs 0 and 2 / 1 and 3; their
        // missing flags in pairs in the 2-bit fields, then in nibbles; dp4a adds the bytes
        uint32_t ce = 0, co = 0, m[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          ce += w[c] & 0x33333333u;
          co += (w[c] >> 2) & 0x33333333u;
          m[c] = w[c] & (w[c] >> 1) & 0x55555555u;
        }
        const uint32_t ma = m[0] + m[1], mb = m[2] + m[3];
        const uint32_t me = (ma & 0x33333333u) + (mb & 0x33333333u);
        const uint32_t mo = ((ma >> 2) & 0x33333333u) + ((mb >> 2) & 0x33333333u);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          sum[s] = __dp4a(((s & 1 ? co : ce) >> (2 * (s & 2))) & 0x0F0F0F0Fu, 0x01010101u, sum[s]);
          mis[s] = __dp4a(((s & 1 ? mo : me) >> (2 * (s & 2))) & 0x0F0F0F0Fu, 0x01010101u, mis[s]);
        }
        if (++since == (1 << 24)) {   // 48 per step and sum: far below 2^32
          since = 0;
#pragma unroll
          for (int s = 0; s < 4; ++s) { tot[s] += sum[s]; tot[4 + s] += mis[s]; sum[s] = mis[s] = 0; }
        }
      }
    }
#pragma unroll
    for (int s = 0; s < 4; ++s) { tot[s] += sum[s]; tot[4 + s] += mis[s]; }
    if (N < (1 << 28)) {   // a warp's sums fit 32 bits
#pragma unroll
      for (int v = 0; v < 8; ++v) tot[v] = __reduce_add_sync(0xffffffffu, (uint32_t)tot[v]);
    } else {
#pragma unroll
      for (int v = 0; v < 8; ++v)
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) tot[v] += __shfl_xor_sync(0xffffffffu, tot[v], o);
    }
    if constexpr (TPR > 32) {
      __syncthreads();   // the previous row's readers are done
      if (lane == 0) {
#pragma unroll
        for (int v = 0; v < 8; ++v) part[t >> 5][v] = tot[v];
      }
      __syncthreads();
      if (t < 4) {
        unsigned long long a = 0, b = 0;
        for (int w = 0; w < TPR / 32; ++w) { a += part[w][t]; b += part[w][4 + t]; }
        tot[0] = a;
        tot[4] = b;
      }
    } else if (lane < 4) {
      const unsigned long long a = lane == 0 ? tot[0] : lane == 1 ? tot[1] : lane == 2 ? tot[2] : tot[3];
      const unsigned long long b = lane == 0 ? tot[4] : lane == 1 ? tot[5] : lane == 2 ? tot[6] : tot[7];
      tot[0] = a;
      tot[4] = b;
    }
    const int64_t j = r * 4 + t;
    if (t < 4 && r < rows && j < M) {
      // utils.py:826-829: f = sum / (2 * count) where count > 0, else 0 (float32 math)
      const unsigned long long cnt = (unsigned long long)N - tot[4];
      const float s = (float)(tot[0] - 3ull * tot[4]), c = (float)cnt;
      f[j] = cnt ? s / (2.0f * c) : 0.0f;
    }
  }
}

// ---------------------------------------------------------------- per-sample counts

// Per-sample counts over the SNPs: missing entries (HET = false; q_bat_i = 2 * #observed) or
// heterozygous ones (HET = true). A thread owns 8 consecutive samples and walks the block's
// packed rows; a row's 8 bytes come from three aligned words and a funnel shift, at any
// alignment. A flag per 2-bit field (code 3: both bits; code 1: the low one) is summed in the
// fields (3 rows), nibbles (12 per 6 rows), bytes (24, 10 times) and 32-bit counters. Padding
// fields of the last row are code 0: neither missing nor heterozygous. Blocks on grid.y
// cover disjoint row ranges and add their integer counts with float64 atomics: integers
// below 2^53 add exactly, so the result does not depend on the order. Memory-bound: 1.25 GB
// in 0.38 ms at N=50,003 x M=100,001 (one byte per thread and row took 2.3 ms).
constexpr int COUNT_TPB = 128;
constexpr int COUNT_SPT = 8;    // samples per thread
constexpr int COUNT_ROWS = 6;   // rows summed in nibbles
constexpr int COUNT_GROUPS = 10; // nibble sums added in bytes

template <bool HET>
__global__ void __launch_bounds__(COUNT_TPB) count_kernel(const uint8_t* __restrict__ G, int64_t M, int64_t N,
                                                          int64_t rows_per_part, double* __restrict__ out) {
  const int64_t i = ((int64_t)blockIdx.x * COUNT_TPB + threadIdx.x) * COUNT_SPT;
  if (i >= N) return;
  const int64_t rows = (M + 3) >> 2;
  const int64_t r0 = (int64_t)blockIdx.y * rows_per_part;
  const int64_t r1 = min(rows, r0 + rows_per_part);
  if (r0 >= r1) return;
  const Bytes all{G, G + rows * N};
  uint32_t total[COUNT_SPT];
#pragma unroll
  for (int b = 0; b < COUNT_SPT; ++b) total[b] = 0;
  auto flags = [](uint32_t w) { return (HET ? w & ~(w >> 1) : w & (w >> 1)) & 0x55555555u; };
  for (int64_t r = r0; r < r1;) {
    uint32_t by[2] = {0, 0};
    for (int g = 0; g < COUNT_GROUPS && r < r1; ++g, r += COUNT_ROWS) {
      uint32_t nib[2] = {0, 0};
      if (r > 0 && r + COUNT_ROWS <= r1 && r + COUNT_ROWS < rows && N >= 12) {
        // neither the first nor the last row: the words (from at most 3 bytes before the
        // thread's first sample to at most 12 past it) cannot leave the matrix
        uint32_t w[COUNT_ROWS][2];
        const uint8_t* src = G + r * N + i;
#pragma unroll
        for (int u = 0; u < COUNT_ROWS; ++u, src += N) {
          const uint32_t sh = 8u * (uint32_t)(reinterpret_cast<uintptr_t>(src) & 3);
          const uint8_t* p = src - (sh >> 3);
          uint32_t v[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) v[c] = __ldg(reinterpret_cast<const uint32_t*>(p + 4 * c));
          w[u][0] = __funnelshift_r(v[0], v[1], sh);
          w[u][1] = __funnelshift_r(v[1], v[2], sh);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const uint32_t x = flags(w[0][c]) + flags(w[1][c]) + flags(w[2][c]);
          const uint32_t y = flags(w[3][c]) + flags(w[4][c]) + flags(w[5][c]);
          nib[c] = (x & 0x33333333u) + ((x >> 2) & 0x33333333u) + (y & 0x33333333u) + ((y >> 2) & 0x33333333u);
        }
      } else {
        for (int u = 0; u < COUNT_ROWS && r + u < r1; ++u) {
          const uint8_t* src = G + (r + u) * N + i;
          const uint32_t sh = 8u * (uint32_t)(reinterpret_cast<uintptr_t>(src) & 3);
          const uint8_t* p = src - (sh >> 3);
          const uint32_t w0 = all.word(p, 0u), w1 = all.word(p + 4, 0u), w2 = all.word(p + 8, 0u);
          const uint32_t w[2] = {__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh)};
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint32_t m = flags(w[c]);
            nib[c] += (m & 0x33333333u) + ((m >> 2) & 0x33333333u);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) by[c] += (nib[c] & 0x0F0F0F0Fu) + ((nib[c] >> 4) & 0x0F0F0F0Fu);
    }
#pragma unroll
    for (int b = 0; b < COUNT_SPT; ++b) total[b] += (by[b >> 2] >> (8 * (b & 3))) & 0xFFu;
  }
  const int64_t snps = min(M, r1 * 4) - r0 * 4;
#pragma unroll
  for (int b = 0; b < COUNT_SPT; ++b)
    if (i + b < N) atomicAdd(out + i + b, HET ? (double)total[b] : 2.0 * (double)(snps - (int64_t)total[b]));
}

// ---------------------------------------------------------------- synthetic sampler

__device__ __forceinline__ uint64_t splitmix64(uint64_t z) {
  z ^= z >> 30;
  z *= 0xBF58476D1CE4E5B9ull;
  z ^= z >> 27;
  z *= 0x94D049BB133111EBull;
  z ^= z >> 31;
  return z;
}

template <int KMAX>
__global__ void simulate_kernel(const uint32_t* __restrict__ Pq, const uint32_t* __restrict__ Qq,
                                int64_t M, int64_t N, int K, uint64_t key1, uint64_t key2,
                                uint32_t miss_q, uint8_t* __restrict__ G) {
  // one thread per sample, grid-stride over packed rows (blockIdx.y)
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  uint32_t q[KMAX];
#pragma unroll
  for (int k = 0; k < KMAX; ++k) q[k] = k < K ? Qq[i * K + k] : 0u;
  const int64_t rows = (M + 3) >> 2;
  for (int64_t r = blockIdx.y; r < rows; r += gridDim.y) {
    uint32_t byte = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int64_t j = r * 4 + s;
      if (j >= M) break;
      uint64_t hq = 0;
#pragma unroll
      for (int k = 0; k < KMAX; ++k)
        if (k < K) hq += (uint64_t)__ldg(Pq + j * K + k) * q[k];
      const uint64_t c = ((uint64_t)j * (uint64_t)N + (uint64_t)i) * 0x9E3779B97F4A7C15ull;
      const uint64_t z1 = splitmix64(c + key1);
      const uint64_t z2 = splitmix64(c + key2);
      uint32_t g = (uint32_t)((z1 & 0xFFFFFFFFull) < hq) + (uint32_t)((z1 >> 32) < hq);
      if ((uint32_t)(z2 & 0xFFFFFFFFull) < miss_q) g = 3u;
      byte |= g << (2 * s);
    }
    G[r * N + i] = (uint8_t)byte;
  }
}

// ---------------------------------------------------------------- PLINK BED -> packed

// A BED row holds a SNP's samples, 4 per byte; a packed row holds 4 SNPs, one byte per sample:
// decoding is a 4 x 4 transpose of 2-bit fields per 4 samples. One warp per packed row (rows
// over blockIdx.x, its 32-unit segments over blockIdx.y); a unit is 16 samples that start at
// a 16-byte boundary of the packed matrix, so the stores are whole and aligned at any N. The
// unit's fields of each SNP are 32 bits at any bit address: two aligned words and a funnel
// shift. Codes go through the LUT [2,3,1,0] (snp_reader.pyx:53-58) as bit operations: the
// high bit is inverted, the low one is the exclusive or of both. Also sums the dosages and
// the observed counts for the flip decision. 2.5 GB in 0.92 ms at N=50,003 x
// M=100,001 (one output byte per thread with byte loads and a 64-bit division took 7 ms).
// 72 % of the issue slots: the transposes and the flag sums.
constexpr int BED_TPB = 256;

__device__ __forceinline__ uint32_t transpose4x4(uint32_t v) {  // field (i, j): bits 8i + 2j
  uint32_t t = (v ^ (v >> 6)) & 0x00CC00CCu;
  v ^= t ^ (t << 6);
  t = (v ^ (v >> 12)) & 0x0000F0F0u;
  return v ^ t ^ (t << 12);
}

__global__ void __launch_bounds__(BED_TPB) bed_decode_kernel(const uint8_t* __restrict__ bed, int64_t M, int64_t N,
                                                             uint8_t* __restrict__ G,
                                                             unsigned long long* __restrict__ acc) {
  __shared__ unsigned long long sh[2];
  if (threadIdx.x < 2) sh[threadIdx.x] = 0;
  __syncthreads();
  const int64_t nb = (N + 3) >> 2;
  const int64_t rows = (M + 3) >> 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Bytes all{bed, bed + M * nb};
  unsigned long long s = 0, c = 0;
  for (int64_t r = (int64_t)blockIdx.x * (BED_TPB / 32) + warp; r < rows; r += (int64_t)gridDim.x * (BED_TPB / 32)) {
    uint8_t* dst = G + r * N;
    const int64_t lead = (int64_t)(reinterpret_cast<uintptr_t>(dst) & 15);
    const int64_t units = (lead + N + 15) >> 4;
    for (int64_t u = (int64_t)blockIdx.y * 32 + lane; u < units; u += (int64_t)gridDim.y * 32) {
      const int64_t s0 = 16 * u - lead;   // the unit's first sample (below 0 in a row's first unit)
      // fields of samples in [0, N)
      uint32_t valid = 0xFFFFFFFFu;
      if (s0 < 0) valid <<= 2 * (uint32_t)(-s0);
      if (s0 + 16 > N) valid &= 0xFFFFFFFFu >> (2 * (uint32_t)(s0 + 16 - N));
      const uint8_t* src = bed + 4 * r * nb + (s0 >> 2);   // floor division: s0 may be negative
      // the unit's words of all four SNPs are inside the matrix: no check per word
      const bool plain = src - 3 >= all.begin && src + 3 * nb + 8 <= all.end;
      uint32_t lo[4], hi[4], bit[4], g[4];
#pragma unroll
      for (int k = 0; k < 4; ++k, src += nb) {
        const uint32_t by = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 3);
        bit[k] = 8u * by + 2u * (uint32_t)(s0 & 3);
        const uint8_t* p = src - by;
        if (plain) {
          lo[k] = __ldg(reinterpret_cast<const uint32_t*>(p));
          hi[k] = __ldg(reinterpret_cast<const uint32_t*>(p + 4));
        } else {
          const bool in = 4 * r + k < M;
          lo[k] = in ? all.word(p, 0u) : 0u;
          hi[k] = in ? all.word(p + 4, 0u) : 0u;
        }
      }
      uint32_t hm[4], ht[4], ms[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t w = __funnelshift_r(lo[k], hi[k], bit[k]);
        const uint32_t v = plain || 4 * r + k < M ? valid : 0u;
        g[k] = ((~w & 0xAAAAAAAAu) | ((w ^ (w >> 1)) & 0x55555555u)) & v;
        const uint32_t l = g[k] & 0x55555555u, h = (g[k] >> 1) & 0x55555555u;
        hm[k] = h & ~l;
        ht[k] = l & ~h;
        ms[k] = (~(l & h)) & (v & 0x55555555u);
      }
      // two SNPs' flags per population count
      const uint32_t hom = __popc(hm[0] | (hm[1] << 1)) + __popc(hm[2] | (hm[3] << 1));
      const uint32_t het = __popc(ht[0] | (ht[1] << 1)) + __popc(ht[2] | (ht[3] << 1));
      const uint32_t seen = __popc(ms[0] | (ms[1] << 1)) + __popc(ms[2] | (ms[3] << 1));
      s += 2 * hom + het;
      c += 2 * seen;
      uint32_t o[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t lo = __byte_perm(g[0], g[1], q | ((4 + q) << 4));
        const uint32_t hi = __byte_perm(g[2], g[3], q | ((4 + q) << 4));
        o[q] = transpose4x4(__byte_perm(lo, hi, 0x5410));
      }
      if (s0 >= 0 && s0 + 16 <= N) {
        *reinterpret_cast<uint4*>(dst + s0) = make_uint4(o[0], o[1], o[2], o[3]);
      } else {
#pragma unroll
        for (int b = 0; b < 16; ++b)
          if (s0 + b >= 0 && s0 + b < N) dst[s0 + b] = (uint8_t)(o[b >> 2] >> (8 * (b & 3)));
      }
    }
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  if (lane == 0) {
    atomicAdd(&sh[0], s);  // integer sums: exact, order-independent
    atomicAdd(&sh[1], c);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(&acc[0], sh[0]);
    atomicAdd(&acc[1], sh[1]);
  }
}

// 0<->2 swap of every field when sum/count >= 0.5 (snp_reader.pyx:254-303); padding fields
// of the last row stay 0. Per field 0->2, 1->1, 2->0, 3->3: the high bit flips where the low
// one is 0. 16 bytes per thread from the first 16-byte boundary.
__global__ void bed_flip_kernel(const unsigned long long* __restrict__ acc, int64_t M, int64_t N,
                                uint8_t* __restrict__ G, int* __restrict__ flipped) {
  const unsigned long long s = acc[0], c = acc[1];
  const bool flip = c != 0 && (double)s / (double)c >= 0.5;
  const int64_t rows = (M + 3) >> 2;
  const int64_t total = rows * N;
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid == 0 && flipped) *flipped = flip ? 1 : 0;
  if (!flip) return;
  const int rem = (int)(M & 3);
  const uint32_t last_mask = (rem ? ((1u << (2 * rem)) - 1u) : 0xFFu) * 0x01010101u;
  const int64_t last = (rows - 1) * N;   // first byte of the last row
  const int64_t lead = (int64_t)(reinterpret_cast<uintptr_t>(G) & 15);
  for (int64_t q = gid; 16 * q - lead < total; q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t at = 16 * q - lead;
    auto swap = [](uint32_t b) { return b ^ ((~b & 0x55555555u) << 1); };
    if (at >= 0 && at + 16 <= last) {
      uint4* p = reinterpret_cast<uint4*>(G + at);
      const uint4 v = *p;
      *p = make_uint4(swap(v.x), swap(v.y), swap(v.z), swap(v.w));
    } else {
      for (int64_t b = max((int64_t)0, at); b < min(total, at + 16); ++b)
        G[b] = (uint8_t)(b >= last ? swap(G[b]) & last_mask : swap(G[b]));
    }
  }
}

}  // namespace adx

using namespace adx;

static unsigned grid_for(int64_t work, int threads) {
  const int64_t b = ceil_div(work, threads);
  const int64_t cap = (int64_t)sm_count() * 32;
  return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
}

extern "C" int adx_unpack_u8(const uint8_t* G, int64_t rows, int64_t N, int64_t M_total,
                             int64_t m_start, int64_t count, int64_t byte_offset, uint8_t* out,
                             void* stream) {
  if (N <= 0 || M_total < 0 || m_start < 0 || count < 0 || byte_offset < 0 || !G || (!out && count)) {
    adx_set_message("adx_unpack_u8: bad arguments");
    return ADX_ERR_ARG;
  }
  count = count < M_total - m_start ? count : M_total - m_start;
  if (count <= 0) return ADX_OK;
  const int64_t last_row = ((m_start + count - 1) >> 2) - byte_offset;
  if (last_row >= rows) { adx_set_message("adx_unpack_u8: chunk beyond the packed rows given"); return ADX_ERR_ARG; }
  unpack_u8_kernel<<<grid_for(count * N, 256), 256, 0, as_stream(stream)>>>(G, N, M_total, m_start, count, byte_offset, out);
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

extern "C" int adx_unpack_center_f32(const uint8_t* G, int64_t rows, int64_t N, int64_t M_total,
                                     int64_t m_start, int64_t count, int64_t byte_offset,
                                     const float* f, float* out, void* stream) {
  if (N <= 0 || M_total < 0 || m_start < 0 || count < 0 || byte_offset < 0 || !G || !f || (!out && count)) {
    adx_set_message("adx_unpack_center_f32: bad arguments");
    return ADX_ERR_ARG;
  }
  count = count < M_total - m_start ? count : M_total - m_start;
  if (count <= 0) return ADX_OK;
  const int64_t last_row = ((m_start + count - 1) >> 2) - byte_offset;
  if (last_row >= rows) { adx_set_message("adx_unpack_center_f32: chunk beyond the packed rows given"); return ADX_ERR_ARG; }
  unpack_center_kernel<<<grid_for(count * N, 256), 256, 0, as_stream(stream)>>>(G, N, M_total, m_start, count, byte_offset, f, out);
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

extern "C" int adx_allele_frequency(const uint8_t* G, int64_t M, int64_t N, float* f, void* stream) {
  if (M <= 0 || N <= 0 || !G || !f) { adx_set_message("adx_allele_frequency: bad arguments"); return ADX_ERR_ARG; }
  const int64_t rows = (M + 3) >> 2;
  // a warp per row while a row is a few loads per lane, a block per row beyond that
  if (N <= 4096) {
    allele_freq_kernel<32><<<grid_for(rows * 32, FREQ_TPB), FREQ_TPB, 0, as_stream(stream)>>>(G, M, N, f);
  } else {
    allele_freq_kernel<FREQ_TPB><<<grid_for(rows * FREQ_TPB, FREQ_TPB), FREQ_TPB, 0, as_stream(stream)>>>(G, M, N, f);
  }
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

template <bool HET>
static int launch_counts(const uint8_t* G, int64_t M, int64_t N, double* out, void* stream) {
  const int64_t rows = (M + 3) >> 2;
  const int64_t xblocks = ceil_div(N, (int64_t)COUNT_TPB * COUNT_SPT);
  // about 16 blocks per SM in all, each of at least a byte sum's rows
  int64_t parts = ceil_div((int64_t)sm_count() * 16, xblocks);
  const int64_t most = ceil_div(rows, COUNT_GROUPS * COUNT_ROWS);
  parts = parts < 1 ? 1 : (parts > most ? most : parts);
  parts = parts > 65535 ? 65535 : parts;
  const int64_t rpp = ceil_div(rows, parts);
  parts = ceil_div(rows, rpp);
  cudaStream_t st = as_stream(stream);
  ADX_CUDA_TRY(cudaMemsetAsync(out, 0, (size_t)N * sizeof(double), st));
  count_kernel<HET><<<dim3((unsigned)xblocks, (unsigned)parts), COUNT_TPB, 0, st>>>(G, M, N, rpp, out);
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

extern "C" int adx_sample_counts(const uint8_t* G, int64_t M, int64_t N, double* q_bat, void* stream) {
  if (M <= 0 || N <= 0 || !G || !q_bat) { adx_set_message("adx_sample_counts: bad arguments"); return ADX_ERR_ARG; }
  return launch_counts<false>(G, M, N, q_bat, stream);
}

extern "C" int adx_sample_het_counts(const uint8_t* G, int64_t M, int64_t N, double* het, void* stream) {
  if (M <= 0 || N <= 0 || !G || !het) { adx_set_message("adx_sample_het_counts: bad arguments"); return ADX_ERR_ARG; }
  return launch_counts<true>(G, M, N, het, stream);
}

extern "C" int adx_simulate_packed(const uint32_t* Pq, const uint32_t* Qq, int64_t M, int64_t N,
                                   int K, uint64_t key1, uint64_t key2, uint32_t miss_q, uint8_t* G,
                                   void* stream) {
  if (M <= 0 || N <= 0 || K < 1 || K > ADX_MAX_K || !Pq || !Qq || !G) {
    adx_set_message("adx_simulate_packed: bad arguments");
    return ADX_ERR_ARG;
  }
  const int threads = 128;
  const int64_t rows = (M + 3) >> 2;
  const unsigned gx = (unsigned)ceil_div(N, threads);
  int64_t gy = ceil_div((int64_t)sm_count() * 16, gx);
  gy = gy < 1 ? 1 : (gy > rows ? rows : gy);
  gy = gy > 65535 ? 65535 : gy;
  const dim3 grid(gx, (unsigned)gy);
  cudaStream_t st = as_stream(stream);
#define SIM(KM) simulate_kernel<KM><<<grid, threads, 0, st>>>(Pq, Qq, M, N, K, key1, key2, miss_q, G)
  if (K <= 4) SIM(4);
  else if (K <= 8) SIM(8);
  else if (K <= 16) SIM(16);
  else if (K <= 32) SIM(32);
  else SIM(64);
#undef SIM
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

extern "C" int adx_bed_workspace_bytes(int64_t M, int64_t N, size_t* bytes) {
  if (M <= 0 || N <= 0 || !bytes) { adx_set_message("adx_bed_workspace_bytes: bad arguments"); return ADX_ERR_ARG; }
  *bytes = 2 * sizeof(unsigned long long);
  return ADX_OK;
}

extern "C" int adx_bed_to_packed(const uint8_t* bed, int64_t M, int64_t N, uint8_t* G, int* flipped,
                                 void* workspace, size_t workspace_bytes, void* stream) {
  if (M <= 0 || N <= 0 || !bed || !G || !workspace) { adx_set_message("adx_bed_to_packed: bad arguments"); return ADX_ERR_ARG; }
  if (workspace_bytes < 2 * sizeof(unsigned long long)) { adx_set_message("adx_bed_to_packed: workspace too small"); return ADX_ERR_WORKSPACE; }
  cudaStream_t st = as_stream(stream);
  unsigned long long* acc = reinterpret_cast<unsigned long long*>(workspace);
  ADX_CUDA_TRY(cudaMemsetAsync(acc, 0, 2 * sizeof(unsigned long long), st));
  const int64_t rows = (M + 3) >> 2;
  const int64_t segs = ceil_div(N + 15, 512);   // 32 units of 16 samples
  const int64_t gx = ceil_div(rows, BED_TPB / 32), cap = (int64_t)sm_count() * 32;
  // rows first; where they leave SMs idle, a row's segments too
  const unsigned bx = (unsigned)(gx < cap ? gx : cap);
  int64_t gy = cap / bx;
  gy = gy < 1 ? 1 : (gy > segs ? segs : gy);
  bed_decode_kernel<<<dim3(bx, (unsigned)(gy < 65535 ? gy : 65535)), BED_TPB, 0, st>>>(bed, M, N, G, acc);
  ADX_LAUNCH_CHECK();
  bed_flip_kernel<<<grid_for(ceil_div(rows * N + 15, 16), 256), 256, 0, st>>>(acc, M, N, G, flipped);
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}
