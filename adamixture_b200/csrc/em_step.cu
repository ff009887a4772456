// Fused Adam-EM E-step for the ADMIXTURE binomial model on B200 (sm_100a), CUDA-core form.
//
// One sweep over the packed genotype matrix computes, for every entry (SNP j, sample i),
//   h = P_j . Q_i,  rec = clamp(h, 1e-5, 1-1e-5),  a = g/rec,  b = (2-g)/(1-rec)  (0 if missing)
// and accumulates both sides of the two-sided reduction
//   A_j = sum_i a Q_i,  B_j = sum_i b Q_i           (P side: reduce over samples)
//   T_i = sum_j (a-b) P_j + sum_j b                  (Q side: reduce over SNPs)
// (adamixture/model/em_adam_gpu.py:46-78). The reference materialises ~6 float64 C x N
// temporaries per 8192-SNP chunk and runs 4 DGEMMs; here G is read once, 2 bits per entry.
//
// Work decomposition (deterministic, no atomics):
//  - a block owns a SNP range [j0, j1) ("SNP block", multiple of CH SNPs, quad aligned) and a
//    residue class of sample sub-tiles ("split"); a sub-tile is TPB*SPT consecutive samples,
//    SPT per thread (their Q rows and T accumulators live in registers);
//  - per SNP, each thread forms its SPT samples' contributions to A_j/B_j, a warp
//    reduce-scatter folds the 2K values over 32 lanes, a cross-warp pass folds the 8 warps
//    and adds the block's partial into AB_part[split][j] (the block is the only writer of
//    those rows, and always the same thread adds the same element);
//  - after its SNP range, each thread writes T_part[snp_block][i] for its samples.
// A second kernel reduces AB_part over splits and T_part over SNP blocks in float64, in a
// fixed order, and either writes A/B/T or applies em_final_update + the Adam move directly.
#include "common.cuh"

#include <math.h>

namespace adx {

constexpr int TPB = 256;
constexpr int WARPS = TPB / 32;
// Block count of a sweep, at most (12 per SM on 148 SMs: whole waves at 1, 2, 3, 4 or 6
// resident blocks per SM, which covers every instance); fixed so the partition, hence the
// summation order, never depends on the GPU.
constexpr int PLAN_BLOCKS = 1776;

template <typename R, int KMAX>
struct EmCfg {
  static constexpr int SPT = (sizeof(R) == 4) ? (KMAX <= 16 ? 4 : (KMAX <= 32 ? 2 : 1))
                                              : (KMAX <= 8 ? 2 : 1);
  static constexpr int W = TPB * SPT;            // samples per sub-tile
  static constexpr int V = 2 * KMAX;             // A and B values per SNP
  static constexpr int VP = ((V + 31) / 32) * 32;
  static constexpr int NCH = VP / 32;
  static constexpr int CH_RAW = 40960 / (WARPS * VP * (int)sizeof(R));
  static constexpr int CH = CH_RAW >= 32 ? 32 : (CH_RAW / 4) * 4;  // SNPs staged per chunk
  static_assert(CH >= 4, "chunk must hold a packed quad");
};

struct EmPlan {
  int64_t M, N;
  int K, kmax, prec;
  int W, CH;
  int64_t n_stile;   // sample sub-tiles
  int n_split;       // sample splits (partials of A/B)
  int n_mblk;        // SNP blocks (partials of T)
  int64_t mb;        // SNPs per SNP block
  size_t ab_elems, t_elems, elem_size;
  // Workspace: a 256-byte header whose first word is the sweep's sticky status (the same
  // offset for every shape, so a shared grow-only buffer keeps it), then the partials.
  // The tensor-core sweep also keeps a 16-bit (FP16 or BF16) copy of Q after the partials.
  static constexpr size_t HEADER = 256;
  size_t extra_bytes = 0;
  size_t extra_offset() const { return (HEADER + (ab_elems + t_elems) * elem_size + 255) & ~size_t(255); }
  size_t bytes() const { return extra_offset() + extra_bytes; }
};

// ---------------------------------------------------------------- device helpers

__device__ __forceinline__ float clampr(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }
__device__ __forceinline__ double clampr(double x, double lo, double hi) { return fmin(fmax(x, lo), hi); }

// a = ga/rec, b = gb/(1-rec). Float: one correctly rounded reciprocal of rec*(1-rec).
// Double: two IEEE divisions, as the reference computes them.
__device__ __forceinline__ void ratios(float ga, float gb, float rec, float omr, float& a, float& b) {
  const float r = __frcp_rn(rec * omr);
  a = ga * (omr * r);
  b = gb * (rec * r);
}
__device__ __forceinline__ void ratios(double ga, double gb, double rec, double omr, double& a, double& b) {
  a = ga / rec;
  b = gb / omr;
}

// Warp reduce-scatter of 32 values: afterwards lane l holds sum over lanes of v[l].
template <typename R>
__device__ __forceinline__ R reduce_scatter32(R (&v)[32], int lane) {
#pragma unroll
  for (int h = 16; h >= 1; h >>= 1) {
    const bool up = (lane & h) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const R send = up ? v[i] : v[i + h];
      const R keep = up ? v[i + h] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
    }
  }
  return v[0];
}

// The same for VR (a power of two below 32) values per lane: the butterfly over the low
// log2(VR) lane bits leaves lane L with value L & (VR - 1) summed over its group of VR lanes,
// and a plain xor-sum across the 32 / VR groups completes it: (VR - 1) + log2(32 / VR)
// shuffles instead of 31 for a vector padded to 32.
template <int VR, typename R>
__device__ __forceinline__ R reduce_scatter_small(R (&v)[VR], int lane) {
#pragma unroll
  for (int h = VR / 2; h >= 1; h >>= 1) {
    const bool up = (lane & h) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const R send = up ? v[i] : v[i + h];
      const R keep = up ? v[i + h] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
    }
  }
#pragma unroll
  for (int h = VR; h < 32; h <<= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], h);
  return v[0];
}

// ---------------------------------------------------------------- E-step sweep

template <typename R, int KMAX>
__global__ void __launch_bounds__(TPB)
em_sweep_kernel(const uint8_t* __restrict__ G, const R* __restrict__ P, const R* __restrict__ Q,
                int64_t M, int64_t N, int K, int64_t n_stile, int n_split, int n_mblk, int64_t mb,
                R* __restrict__ ABp, R* __restrict__ Tp) {
  using C = EmCfg<R, KMAX>;
  constexpr int SPT = C::SPT, CH = C::CH, VP = C::VP, V = C::V;
  __shared__ R Ps[CH][KMAX];
  __shared__ R red[WARPS][CH][VP];

  const int mblk = blockIdx.x % n_mblk;
  const int split = blockIdx.x / n_mblk;
  const int64_t j0 = (int64_t)mblk * mb;
  const int64_t j1 = min(M, j0 + mb);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool aligned4 = (SPT == 4) && ((N & 3) == 0);
  const R ELO = (R)E_CLAMP, EHI = (R)(1.0 - E_CLAMP);

  bool first = true;
  for (int64_t st = split; st < n_stile; st += n_split) {
    const int64_t i0 = st * C::W + (int64_t)threadIdx.x * SPT;
    R q[SPT][KMAX], tab[SPT][KMAX], tb[SPT];
#pragma unroll
    for (int u = 0; u < SPT; ++u) {
      tb[u] = 0;
#pragma unroll
      for (int k = 0; k < KMAX; ++k) {
        tab[u][k] = 0;
        q[u][k] = (i0 + u < N && k < K) ? Q[(i0 + u) * K + k] : (R)0;
      }
    }

    for (int64_t c0 = j0; c0 < j1; c0 += CH) {
      const int cn = (int)min((int64_t)CH, j1 - c0);
      __syncthreads();
      for (int e = threadIdx.x; e < CH * KMAX; e += TPB) {
        const int jl = e / KMAX, k = e % KMAX;
        Ps[jl][k] = (jl < cn && k < K) ? P[(c0 + jl) * K + k] : (R)0;
      }
      __syncthreads();

      for (int qd = 0; qd < cn; qd += 4) {
        const int64_t row = (c0 + qd) >> 2;
        uint32_t bytes[SPT];
        if (aligned4 && i0 < N) {
          const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(G + row * N + i0));
#pragma unroll
          for (int u = 0; u < SPT; ++u) bytes[u] = (w >> (8 * u)) & 0xFFu;
        } else {
#pragma unroll
          for (int u = 0; u < SPT; ++u) bytes[u] = (i0 + u < N) ? (uint32_t)__ldg(G + row * N + i0 + u) : 0xFFu;
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int jl = qd + s;
          if (jl >= cn) break;  // uniform across the block
          R a[SPT], b[SPT], hh[SPT];
#pragma unroll
          for (int u = 0; u < SPT; ++u) {
            R h = 0;
#pragma unroll
            for (int k = 0; k < KMAX; ++k) h += Ps[jl][k] * q[u][k];
            hh[u] = h;
          }
#pragma unroll
          for (int u = 0; u < SPT; ++u) {
            const unsigned g = genotype(bytes[u], s);
            const R rec = clampr(hh[u], ELO, EHI);
            const R omr = (R)1 - rec;
            const R ga = (g == 3u) ? (R)0 : (R)g;
            const R gb = (g == 3u) ? (R)0 : (R)(2u - g);
            ratios(ga, gb, rec, omr, a[u], b[u]);
            const R d = a[u] - b[u];
#pragma unroll
            for (int k = 0; k < KMAX; ++k) tab[u][k] += d * Ps[jl][k];
            tb[u] += b[u];
          }
          // this thread's part of value v of the SNP: A column v (v < KMAX), else B column
          // v - KMAX, summed over its samples
          auto part_of = [&](int v) {
            R acc = 0;
            if (v < KMAX) {
#pragma unroll
              for (int u = 0; u < SPT; ++u) acc += a[u] * q[u][v < KMAX ? v : 0];
            } else if (v < V) {
#pragma unroll
              for (int u = 0; u < SPT; ++u) acc += b[u] * q[u][v >= KMAX && v < V ? v - KMAX : 0];
            }
            return acc;
          };
          if constexpr (V > 16 && V < 32 && ((V - 16) & (V - 17)) == 0) {
            // 16 + 4 or 16 + 8 values: two power-of-two vectors, 16 + 6 or 16 + 9 shuffle
            // steps instead of 31; lane l < 16 holds value l, lane 16 + i value 16 + i
            constexpr int VR2 = V - 16;
            R p1[16], p2[VR2];
#pragma unroll
            for (int v = 0; v < 16; ++v) p1[v] = part_of(v);
#pragma unroll
            for (int v = 0; v < VR2; ++v) p2[v] = part_of(16 + v);
            const R r1 = reduce_scatter_small<16>(p1, lane);
            const R r2 = reduce_scatter_small<VR2>(p2, lane);
            red[warp][jl][lane] = lane < 16 ? r1 : r2;
          } else {
#pragma unroll
            for (int c = 0; c < C::NCH; ++c) {
              R part[32];
#pragma unroll
              for (int l = 0; l < 32; ++l) part[l] = part_of(c * 32 + l);
              red[warp][jl][c * 32 + lane] = reduce_scatter32(part, lane);
            }
          }
        }
      }
      __syncthreads();
      const int nv = cn * V;
      for (int e = threadIdx.x; e < nv; e += TPB) {
        const int jl = e / V, v = e % V;
        const int k = v < KMAX ? v : v - KMAX;
        if (k >= K) continue;
        R sum = 0;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) sum += red[w][jl][v];
        R* dst = ABp + ((int64_t)split * M + (c0 + jl)) * (2 * K) + (v < KMAX ? k : K + k);
        *dst = first ? sum : *dst + sum;
      }
    }
#pragma unroll
    for (int u = 0; u < SPT; ++u) {
      if (i0 + u < N) {
        R* dst = Tp + ((int64_t)mblk * N + i0 + u) * K;
#pragma unroll
        for (int k = 0; k < KMAX; ++k)
          if (k < K) dst[k] = tab[u][k] + tb[u];
      }
    }
    first = false;
  }
}

// ---------------------------------------------------------------- float32 sweep, K <= 8
//
// The float32 sweep for the K whose default arithmetic it is. The same statistics, partition
// and partials as em_sweep_kernel<float>; what bounds both is instruction issue, so the work
// per entry is cut: a thread owns 8 consecutive samples and computes them as four packed
// float32 pairs (h, T, A and B are fma.rn.f32x2: the pairs run along the samples, so every
// product uses the same packed copy of Q), the 2K sums of a SNP over its 8 samples go to
// shared memory once per SNP as 16-byte stores, and after a packed quad of SNPs the warp sums
// them by columns (16-byte loads) -- about 2 instructions an entry where the butterfly over
// the lanes of 4 samples took 15. The reciprocal of rec (1 - rec) is the hardware
// approximation (1 ulp) refined by one Newton-Raphson step. N=20,000 x M=100,000, K=6: 5.8 ->
// 3.8 ms an iteration (36 instructions an entry, 54 % of the packed FMA rate).
namespace f32s {

constexpr int TPB = 128;
constexpr int WARPS = TPB / 32;
constexpr int C = 8;                 // samples per thread
constexpr int W = TPB * C;           // samples per sub-tile
constexpr int CH = 32;               // SNP blocks are whole multiples

using u64 = unsigned long long;
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
  u64 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
  u64 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64 pack2(float lo, float hi) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(u64 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ float rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

constexpr int ctas_per_sm(int K) { return K <= 2 ? 5 : K <= 4 ? 4 : K <= 6 ? 3 : 2; }   // registers without spills

template <int K>
struct Cfg {
  static constexpr int V = 2 * K;
  static constexpr int V4 = (V + 3) / 4;                        // 16-byte columns of a SNP's sums
  static constexpr int RS = V4 == 1 ? 4 : V4 <= 3 ? 12 : 20;    // floats per lane: 16-byte stores free of conflicts
  static constexpr int SS = 32 * RS + (V4 == 3 ? 12 : 0);       // floats per SNP: column loads likewise (nearly)
  static constexpr int COLS = 4 * V4;                           // columns of a quad of SNPs
  static constexpr int LPC = COLS == 4 ? 8 : COLS == 8 ? 4 : 2; // lanes that share a column
  static constexpr int KP = (K + 1) / 2 * 2;                    // P row of a SNP: pairs {p, p}, 16-byte loads
  static constexpr int OCC = ctas_per_sm(K);
  static constexpr int CHK = K <= 6 ? 32 : 16;                  // SNPs per staged chunk (48 KB of shared memory)
};

template <int K>
__global__ void __launch_bounds__(TPB, Cfg<K>::OCC)
em_sweep_f32_kernel(const uint8_t* __restrict__ G, const float* __restrict__ P, const float* __restrict__ Q, int64_t M,
                    int64_t N, int64_t n_stile, int n_split, int n_mblk, int64_t mb, float* __restrict__ ABp,
                    float* __restrict__ Tp) {
  using F = Cfg<K>;
  constexpr int CH = F::CHK, V = F::V, V4 = F::V4, RS = F::RS, SS = F::SS, LPC = F::LPC, KP = F::KP;
  __shared__ __align__(16) u64 Ps[CH][KP];
  __shared__ __align__(16) float part[WARPS][4 * SS];
  __shared__ __align__(16) float red[WARPS][CH][4 * V4];
  const int mblk = blockIdx.x % n_mblk;
  const int split = blockIdx.x / n_mblk;
  const int64_t j0 = (int64_t)mblk * mb;
  const int64_t j1 = min(M, j0 + mb);
  const int64_t total = ((M + 3) >> 2) * N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const u64 one2 = pack2(1.0f, 1.0f), mone2 = pack2(-1.0f, -1.0f);
  const float ELO = (float)E_CLAMP, EHI = (float)(1.0 - E_CLAMP);
  // weights as the high halves of float32 values by the 2-bit code (low halves 0), two per byte
  // permute: -g -> {-0, -1, -2, -0} (its product with -1/rec is a), 2 - g -> {2, 1, 0, 0}
  constexpr uint32_t GA_LO = 0xBF808000u, GA_HI = 0x8000C000u, GB_LO = 0x3F804000u, GB_HI = 0x00000000u;

  bool first = true;
  for (int64_t st = split; st < n_stile; st += n_split) {
    const int64_t i0 = st * W + (int64_t)threadIdx.x * C;
    u64 q[C / 2][K], tt[C / 2][K], tb[C / 2];
#pragma unroll
    for (int v = 0; v < C / 2; ++v) {
      tb[v] = 0ull;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        tt[v][k] = 0ull;
        q[v][k] = pack2(i0 + 2 * v < N ? Q[(i0 + 2 * v) * K + k] : 0.0f, i0 + 2 * v + 1 < N ? Q[(i0 + 2 * v + 1) * K + k] : 0.0f);
      }
    }
    // the 8 bytes of the thread's samples in the packed row of SNP j. Samples past N read the
    // next row's (or 0xFF): their Q is zero, so they add nothing, and their T is not written
    auto fetch = [&](int64_t j) { return i0 < N ? fetch8(G, total, (j >> 2) * N + i0) : Words8{~0u, ~0u, ~0u, 0u}; };
    Words8 next = fetch(j0);
    // a chunk's P values, loaded a chunk ahead of their use
    constexpr int PPT = (CH * KP + TPB - 1) / TPB;
    float pnext[PPT];
    auto load_p = [&](int64_t c0) {
#pragma unroll
      for (int u = 0; u < PPT; ++u) {
        const int e = threadIdx.x + u * TPB, jl = e / KP, k = e - jl * KP;
        pnext[u] = e < CH * KP && c0 + jl < j1 && k < K ? P[(c0 + jl) * K + k] : 0.0f;
      }
    };
    load_p(j0);
    for (int64_t c0 = j0; c0 < j1; c0 += CH) {
      const int cn = (int)min((int64_t)CH, j1 - c0);
      __syncthreads();
#pragma unroll
      for (int u = 0; u < PPT; ++u) {
        const int e = threadIdx.x + u * TPB;
        if (e < CH * KP) (&Ps[0][0])[e] = pack2(pnext[u], pnext[u]);
      }
      __syncthreads();
      if (c0 + CH < j1) load_p(c0 + CH);
      for (int qd = 0; qd < cn; qd += 4) {
        const uint64_t bytes = next.bytes();
        if (c0 + qd + 4 < j1) next = fetch(c0 + qd + 4);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int jl = qd + s;
          u64 p[KP];
#pragma unroll
          for (int k = 0; k < KP; k += 2) {
            const ulonglong2 pp = *reinterpret_cast<const ulonglong2*>(&Ps[jl][k]);
            p[k] = pp.x;
            p[k + 1] = pp.y;
          }
          u64 a[C / 2], b[C / 2];
#pragma unroll
          for (int v = 0; v < C / 2; ++v) {
            u64 h = mul2(p[0], q[v][0]);
#pragma unroll
            for (int k = 1; k < K; ++k) h = fma2(p[k], q[v][k], h);
            float h0, h1;
            unpack2(h, h0, h1);
            const u64 rec = pack2(fminf(fmaxf(h0, ELO), EHI), fminf(fmaxf(h1, ELO), EHI));
            const u64 nom = add2(rec, mone2);          // -(1 - rec)
            const u64 nx = mul2(rec, nom);             // -rec (1 - rec)
            float x0, x1;
            unpack2(nx, x0, x1);
            u64 r = pack2(rcp(-x0), rcp(-x1));
            r = fma2(r, fma2(nx, r, one2), r);
            // codes of the two samples (SNPs past the range: missing), then both weights of each
            uint32_t t2 = (uint32_t)(bytes >> (16 * v + 2 * s)) & 0x0303u;
            if (jl >= cn) t2 = 0x0303u;
            const uint32_t sel = t2 * 0x22u + 0x1010u;
            const uint32_t wa = __byte_perm(GA_LO, GA_HI, sel), wb = __byte_perm(GB_LO, GB_HI, sel);
            const u64 ga = ((u64)(wa & 0xFFFF0000u) << 32) | (wa << 16), gb = ((u64)(wb & 0xFFFF0000u) << 32) | (wb << 16);
            a[v] = mul2(ga, mul2(nom, r));
            b[v] = mul2(gb, mul2(rec, r));
            tb[v] = add2(tb[v], b[v]);
            const u64 d = fma2(b[v], mone2, a[v]);
#pragma unroll
            for (int k = 0; k < K; ++k) tt[v][k] = fma2(d, p[k], tt[v][k]);
          }
          float out[4 * V4];
#pragma unroll
          for (int k = 0; k < 4 * V4; ++k) {
            if (k >= V) { out[k] = 0.0f; continue; }
            const int kk = k < K ? k : k - K;
            u64 m = mul2(k < K ? a[0] : b[0], q[0][kk]);
#pragma unroll
            for (int v = 1; v < C / 2; ++v) m = fma2(k < K ? a[v] : b[v], q[v][kk], m);
            float lo, hi;
            unpack2(m, lo, hi);
            out[k] = lo + hi;
          }
          float4* dst = reinterpret_cast<float4*>(&part[warp][s * SS + lane * RS]);
#pragma unroll
          for (int c = 0; c < V4; ++c) dst[c] = make_float4(out[4 * c], out[4 * c + 1], out[4 * c + 2], out[4 * c + 3]);
        }
        __syncwarp();
        // column c = (SNP, 4 sums): LPC lanes add 32 / LPC rows each
        {
          const int c = min(lane / LPC, F::COLS - 1), hl = lane % LPC;
          const int s = c / V4, qq = c - s * V4;
          const float* src = &part[warp][s * SS + hl * RS + 4 * qq];
          float4 x = *reinterpret_cast<const float4*>(src);
          u64 lo = pack2(x.x, x.y), hi = pack2(x.z, x.w);
#pragma unroll
          for (int r = 1; r < 32 / LPC; ++r) {
            const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(src + r * LPC * RS);
            lo = add2(lo, y.x);
            hi = add2(hi, y.y);
          }
#pragma unroll
          for (int o = 1; o < LPC; o <<= 1) {
            lo = add2(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = add2(hi, __shfl_xor_sync(0xffffffffu, hi, o));
          }
          if (hl == 0 && lane / LPC < F::COLS)
            *reinterpret_cast<ulonglong2*>(&red[warp][qd + s][4 * qq]) = make_ulonglong2(lo, hi);
        }
        __syncwarp();
      }
      __syncthreads();
      for (int e = threadIdx.x; e < cn * V; e += TPB) {
        const int jl = e / V, v = e - jl * V;
        float sum = 0.0f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) sum += red[w][jl][v];
        // the block is the only writer of the element and this thread always adds it, so an
        // add in memory keeps the order, and nothing waits for the old value
        float* dst = ABp + ((int64_t)split * M + (c0 + jl)) * V + v;
        if (first) *dst = sum;
        else atomicAdd(dst, sum);
      }
    }
#pragma unroll
    for (int v = 0; v < C / 2; ++v) {
      float b0, b1;
      unpack2(tb[v], b0, b1);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int64_t i = i0 + 2 * v + u;
        if (i >= N) continue;
        float* dst = Tp + ((int64_t)mblk * N + i) * K;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          float t0, t1;
          unpack2(tt[v][k], t0, t1);
          dst[k] = (u ? t1 : t0) + (u ? b1 : b0);
        }
      }
    }
    first = false;
  }
}

constexpr int MAX_K = 8;

}  // namespace f32s

// ---------------------------------------------------------------- reduce / targets / Adam

struct AdamArgs {
  double t, lr, b1, b2, eps;
  // captured iterations: the step is *t_dev + t (t the iteration's offset in the replay)
  const double* t_dev = nullptr;
};

__device__ __forceinline__ double adam_step_no(const AdamArgs& ad) { return ad.t_dev ? *ad.t_dev + ad.t : ad.t; }

// Adds v over the warp's lanes (32 lanes a row) in a fixed order; every lane gets the sum.
template <int KMAX>
__device__ __forceinline__ void warp_sum(double (&v)[KMAX]) {
#pragma unroll
  for (int k = 0; k < KMAX; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
}

// mode 0: write A, B, T (float64 statistics). mode 1: EM targets + Adam move on P and Q.
// gp, gq: threads per P and Q row, 1 or 32. One adds a row's partials in turn; 32 add every
// 32nd and then each other's. The first p_blocks blocks do the P rows.
template <typename R, int KMAX>
__global__ void em_update_kernel(const R* __restrict__ ABp, const R* __restrict__ Tp, int64_t M,
                                 int64_t N, int K, int n_split, int n_mblk, int mode,
                                 double* __restrict__ outA, double* __restrict__ outB,
                                 double* __restrict__ outT, const double* __restrict__ q_bat,
                                 double* __restrict__ P, double* __restrict__ Q,
                                 float* __restrict__ P32, float* __restrict__ Q32,
                                 double* __restrict__ mP, double* __restrict__ vP,
                                 double* __restrict__ mQ, double* __restrict__ vQ, AdamArgs ad, unsigned p_blocks,
                                 int gp, int gq) {
  const bool p_side = blockIdx.x < p_blocks;
  const int g = p_side ? gp : gq;
  const int64_t idx = (int64_t)(p_side ? blockIdx.x : blockIdx.x - p_blocks) * blockDim.x + threadIdx.x;
  const int64_t row = g == 1 ? idx : idx >> 5;
  const int part0 = g == 1 ? 0 : (int)(idx & 31);
  if (row >= (p_side ? M : N)) return;   // whole warps when g = 32
  const double t = adam_step_no(ad);
  const double bc1 = 1.0 - pow(ad.b1, t);
  const double bc2 = 1.0 - pow(ad.b2, t);
  if (p_side) {
    const int64_t j = row;
    double A[KMAX], B[KMAX];
#pragma unroll
    for (int k = 0; k < KMAX; ++k) { A[k] = 0.0; B[k] = 0.0; }
    for (int s = part0; s < n_split; s += g) {
      const R* src = ABp + ((int64_t)s * M + j) * (2 * K);
#pragma unroll
      for (int k = 0; k < KMAX; ++k)
        if (k < K) { A[k] += (double)src[k]; B[k] += (double)src[K + k]; }
    }
    if (g > 1) {
      warp_sum(A);
      warp_sum(B);
      if (part0) return;
    }
    if (mode == 0) {
#pragma unroll
      for (int k = 0; k < KMAX; ++k)
        if (k < K) { outA[j * K + k] = A[k]; outB[j * K + k] = B[k]; }
      return;
    }
#pragma unroll
    for (int k = 0; k < KMAX; ++k) {
      if (k >= K) continue;
      const int64_t o = j * K + k;
      const double p = P[o];
      // em_final_update order: ((A-B)*P + B) -> clamp(min 1e-5) -> reciprocal -> *P -> *A
      const double den = fmax((A[k] - B[k]) * p + B[k], 1e-5);
      const double target = ((1.0 / den) * p) * A[k];
      const double delta = target - p;
      const double m = mP[o] * ad.b1 + (1.0 - ad.b1) * delta;
      const double v = vP[o] * ad.b2 + (1.0 - ad.b2) * (delta * delta);
      mP[o] = m;
      vP[o] = v;
      double np = p + (ad.lr * (m / bc1)) / (sqrt(v / bc2) + ad.eps);
      np = fmin(fmax(np, DOMAIN), 1.0 - DOMAIN);
      P[o] = np;
      if (P32) P32[o] = (float)np;
    }
    return;
  }
  const int64_t i = row;
  double T[KMAX];
#pragma unroll
  for (int k = 0; k < KMAX; ++k) T[k] = 0.0;
  for (int b = part0; b < n_mblk; b += g) {
    const R* src = Tp + ((int64_t)b * N + i) * K;
#pragma unroll
    for (int k = 0; k < KMAX; ++k)
      if (k < K) T[k] += (double)src[k];
  }
  if (g > 1) {
    warp_sum(T);
    if (part0) return;
  }
  if (mode == 0) {
#pragma unroll
    for (int k = 0; k < KMAX; ++k)
      if (k < K) outT[i * K + k] = T[k];
    return;
  }
  const double scale = 1.0 / fmax(q_bat[i], 1e-5);
  double qe[KMAX];
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < KMAX; ++k) {
    qe[k] = (k < K) ? (Q[i * K + k] * T[k]) * scale : 0.0;
    s += qe[k];
  }
  s = fmax(s, 1e-5);
  double tot = 0.0;
#pragma unroll
  for (int k = 0; k < KMAX; ++k) {
    if (k >= K) continue;
    const int64_t o = i * K + k;
    const double qv = Q[o];
    const double delta = qe[k] / s - qv;
    const double m = mQ[o] * ad.b1 + (1.0 - ad.b1) * delta;
    const double v = vQ[o] * ad.b2 + (1.0 - ad.b2) * (delta * delta);
    mQ[o] = m;
    vQ[o] = v;
    double nq = qv + (ad.lr * (m / bc1)) / (sqrt(v / bc2) + ad.eps);
    nq = fmin(fmax(nq, DOMAIN), 1.0 - DOMAIN);
    qe[k] = nq;
    tot += nq;
  }
#pragma unroll
  for (int k = 0; k < KMAX; ++k) {
    if (k >= K) continue;
    const double nq = qe[k] / tot;
    Q[i * K + k] = nq;
    if (Q32) Q32[i * K + k] = (float)nq;
  }
}

// The same for launches whose blocks are all on the chip at once (K <= 16, the rule stands at the
// launch): their time is the longest chain of one thread, not memory. So a P element, which
// depends on no other, has a thread of its own (blockDim.x / K rows a block); partials load in
// batches; the bias corrections are formed once a block, beside those loads; and the
// lanes that added a Q row's partials (gq = 32) take its elements, the sums that normalise it
// running over the lanes in the elements' order. A 20-iteration fit of 105 x 8,451, K=7 in
// float64: 1.33 -> 1.24 ms. Larger launches want the form above: 20,000 x 100,000, K=6 took
// 3.82 ms with this one against 3.80, and 10,007 x 200,003, K=8 1.96 against 1.92.
template <typename R, int KMAX>
__device__ __forceinline__ void add_partials(double (&v)[KMAX], const R* __restrict__ src, int64_t stride, int K,
                                             int part0, int n_parts, int step) {
  constexpr int REGS = KMAX * (int)(sizeof(R) / 4);   // of one part; a batch takes at most 48
  constexpr int BATCH = 4 * REGS <= 48 ? 4 : 2 * REGS <= 48 ? 2 : 1;
  int s = part0;
  for (; s + (BATCH - 1) * step < n_parts; s += BATCH * step) {
    R x[BATCH][KMAX];
#pragma unroll
    for (int u = 0; u < BATCH; ++u)
#pragma unroll
      for (int k = 0; k < KMAX; ++k)
        if (k < K) x[u][k] = src[(s + u * step) * stride + k];
#pragma unroll
    for (int u = 0; u < BATCH; ++u)
#pragma unroll
      for (int k = 0; k < KMAX; ++k)
        if (k < K) v[k] += (double)x[u][k];
  }
  for (; s < n_parts; s += step)
#pragma unroll
    for (int k = 0; k < KMAX; ++k)
      if (k < K) v[k] += (double)src[s * stride + k];
}

constexpr int RESIDENT_MAX_K = 16, RESIDENT_TPB = 128, RESIDENT_BLOCKS = 4;   // threads, blocks per SM

template <typename R, int KMAX>
__global__ void __launch_bounds__(RESIDENT_TPB, RESIDENT_BLOCKS) em_update_resident_kernel(
    const R* __restrict__ ABp, const R* __restrict__ Tp, int64_t M, int64_t N, int K, int n_split, int n_mblk,
    int mode, double* __restrict__ outA, double* __restrict__ outB, double* __restrict__ outT,
    const double* __restrict__ q_bat, double* __restrict__ P, double* __restrict__ Q, float* __restrict__ P32,
    float* __restrict__ Q32, double* __restrict__ mP, double* __restrict__ vP, double* __restrict__ mQ,
    double* __restrict__ vQ, AdamArgs ad, unsigned p_blocks, int gq) {
  __shared__ double bc[2];
  const int lane = threadIdx.x & 31;
  if (mode != 0 && lane == 0 && threadIdx.x < 64)
    bc[threadIdx.x >> 5] = 1.0 - pow(threadIdx.x ? ad.b2 : ad.b1, adam_step_no(ad));
  auto move = [&](double x, double target, double* m_, double* v_, int64_t o) {
    const double delta = target - x;
    const double m = m_[o] * ad.b1 + (1.0 - ad.b1) * delta;
    const double v = v_[o] * ad.b2 + (1.0 - ad.b2) * (delta * delta);
    m_[o] = m;
    v_[o] = v;
    const double nx = x + (ad.lr * (m / bc[0])) / (sqrt(v / bc[1]) + ad.eps);
    return fmin(fmax(nx, DOMAIN), 1.0 - DOMAIN);
  };
  if (blockIdx.x < p_blocks) {
    const int rows = blockDim.x / K, r = threadIdx.x / K, k = threadIdx.x - r * K;
    const int64_t j = (int64_t)blockIdx.x * rows + r, o = j * K + k;
    const bool mine = r < rows && j < M;
    double a[1] = {0.0}, b[1] = {0.0};
    if (mine) {
      const R* src = ABp + j * (2 * K) + k;
      add_partials(a, src, M * 2 * K, 1, 0, n_split, 1);
      add_partials(b, src + K, M * 2 * K, 1, 0, n_split, 1);
    }
    __syncthreads();
    if (!mine) return;
    if (mode == 0) {
      outA[o] = a[0];
      outB[o] = b[0];
      return;
    }
    const double p = P[o];
    const double den = fmax((a[0] - b[0]) * p + b[0], 1e-5);
    const double np = move(p, ((1.0 / den) * p) * a[0], mP, vP, o);
    P[o] = np;
    if (P32) P32[o] = (float)np;
    return;
  }
  const int64_t idx = (int64_t)(blockIdx.x - p_blocks) * blockDim.x + threadIdx.x;
  const int64_t i = gq == 1 ? idx : idx >> 5;
  const bool mine = i < N;   // whole warps when gq = 32
  double T[KMAX];
#pragma unroll
  for (int k = 0; k < KMAX; ++k) T[k] = 0.0;
  if (mine) {
    add_partials(T, Tp + i * K, N * K, K, gq == 1 ? 0 : lane, n_mblk, gq);
    if (gq > 1) warp_sum(T);
  }
  __syncthreads();
  if (!mine) return;
  if (mode == 0) {
    if (gq > 1 && lane) return;
#pragma unroll
    for (int k = 0; k < KMAX; ++k)
      if (k < K) outT[i * K + k] = T[k];
    return;
  }
  const double scale = 1.0 / fmax(q_bat[i], 1e-5);
  double s = 0.0, tot = 0.0;
  if (gq > 1) {   // lane k: element k
    const int64_t o = i * K + lane;
    const bool has = lane < K;
    double x = 0.0, e = 0.0, nq = 0.0;
#pragma unroll
    for (int k = 0; k < KMAX; ++k)
      if (lane == k) e = T[k];
    if (has) {
      x = Q[o];
      e = (x * e) * scale;
    }
#pragma unroll
    for (int k = 0; k < KMAX; ++k) s += __shfl_sync(0xffffffffu, e, k);   // 0 past K
    if (has) nq = move(x, e / fmax(s, 1e-5), mQ, vQ, o);
#pragma unroll
    for (int k = 0; k < KMAX; ++k) tot += __shfl_sync(0xffffffffu, nq, k);
    if (has) {
      nq /= tot;
      Q[o] = nq;
      if (Q32) Q32[o] = (float)nq;
    }
    return;
  }
  double qe[KMAX];
#pragma unroll
  for (int k = 0; k < KMAX; ++k) {
    qe[k] = (k < K) ? (Q[i * K + k] * T[k]) * scale : 0.0;
    s += qe[k];
  }
  s = fmax(s, 1e-5);
#pragma unroll
  for (int k = 0; k < KMAX; ++k) {
    if (k >= K) continue;
    const int64_t o = i * K + k;
    qe[k] = move(Q[o], qe[k] / s, mQ, vQ, o);
    tot += qe[k];
  }
#pragma unroll
  for (int k = 0; k < KMAX; ++k) {
    if (k >= K) continue;
    const double nq = qe[k] / tot;
    Q[i * K + k] = nq;
    if (Q32) Q32[i * K + k] = (float)nq;
  }
}

// ---------------------------------------------------------------- planning and dispatch

static const int KMAX_LIST[] = {2, 3, 4, 6, 8, 10, 12, 16, 24, 32, 48, 64};

int pick_kmax(int K) {
  for (int km : KMAX_LIST)
    if (K <= km) return km;
  return -1;
}

template <typename R, int KMAX>
static void cfg_of(int& W, int& CH) {
  W = EmCfg<R, KMAX>::W;
  CH = EmCfg<R, KMAX>::CH;
}

#define ADX_KMAX_SWITCH(kmax, MACRO)                                                   \
  switch (kmax) {                                                                      \
    case 2: MACRO(2); break;   case 3: MACRO(3); break;   case 4: MACRO(4); break;     \
    case 6: MACRO(6); break;   case 8: MACRO(8); break;   case 10: MACRO(10); break;   \
    case 12: MACRO(12); break; case 16: MACRO(16); break; case 24: MACRO(24); break;   \
    case 32: MACRO(32); break; case 48: MACRO(48); break; case 64: MACRO(64); break;   \
    default: break;                                                                    \
  }

int tc_plan(int64_t M, int64_t N, int K, int64_t& n_stile, int& n_split, int& n_mblk);
size_t tc_q_bytes(int64_t n_stile);
int tc_sweep(const uint8_t* G, const float* P, const float* Q, int64_t M, int64_t N, int K,
             int64_t n_stile, int n_split, int n_mblk, float* ABp, float* Tp, void* Qb, int* err,
             bool f16, cudaStream_t st);

int dmma_plan_width();
int dmma_plan_chunk();
int dmma_sweep(const uint8_t* G, const double* P, const double* Q, int64_t M, int64_t N, int K,
               int64_t n_stile, int n_split, int n_mblk, int64_t mb, double* ABp, double* Tp,
               cudaStream_t st, double* llp = nullptr, int b0 = 0, int b1 = 0);
// Float64 sweeps for K <= 16 run on the float64 tensor-core MMA (em_sweep_dmma.cu).
constexpr int DMMA_MAX_K = 16;

int em_plan(int64_t M, int64_t N, int K, int prec, EmPlan& pl) {
  if (M <= 0 || N <= 0 || K < 1 || K > ADX_MAX_K) return ADX_ERR_ARG;
  if (prec != ADX_F64 && prec != ADX_F32 && prec != ADX_BF16 && prec != ADX_F16) return ADX_ERR_UNSUPPORTED;
  pl.M = M; pl.N = N; pl.K = K; pl.prec = prec;
  pl.kmax = pick_kmax(K);
  if (prec == ADX_BF16 || prec == ADX_F16) {
    // tensor-core sweep: 896-SNP blocks x 128-sample tiles, float partials
    int64_t n_stile = 0;
    int n_split = 0, n_mblk = 0;
    const int rc = tc_plan(M, N, K, n_stile, n_split, n_mblk);
    if (rc) return rc;
    pl.W = 128; pl.CH = 0;
    pl.elem_size = sizeof(float);
    pl.n_stile = n_stile; pl.n_split = n_split; pl.n_mblk = n_mblk;
    pl.mb = 896;
    pl.ab_elems = (size_t)n_split * (size_t)M * 2 * K;
    pl.t_elems = (size_t)n_mblk * (size_t)N * K;
    pl.extra_bytes = tc_q_bytes(n_stile);
    return ADX_OK;
  }
  int W = 0, CH = 0;
#define CFG64(KM) cfg_of<double, KM>(W, CH)
#define CFG32(KM) cfg_of<float, KM>(W, CH)
  if (prec == ADX_F64) { ADX_KMAX_SWITCH(pl.kmax, CFG64) } else { ADX_KMAX_SWITCH(pl.kmax, CFG32) }
#undef CFG64
#undef CFG32
  if (prec == ADX_F64 && K <= DMMA_MAX_K) {
    W = dmma_plan_width();
    CH = dmma_plan_chunk();
  }
  if (prec == ADX_F32 && K <= f32s::MAX_K) {
    W = f32s::W;
    CH = f32s::CH;
  }
  pl.W = W; pl.CH = CH;
  pl.elem_size = prec == ADX_F64 ? sizeof(double) : sizeof(float);
  pl.n_stile = ceil_div(N, W);
  // minimise split*2MK + mblk*NK with split*mblk ~ PLAN_BLOCKS
  double s = sqrt((double)PLAN_BLOCKS * (double)N / (2.0 * (double)M));
  int64_t n_split = (int64_t)llround(s);
  n_split = n_split < 1 ? 1 : n_split;
  n_split = n_split > pl.n_stile ? pl.n_stile : n_split;
  n_split = n_split > PLAN_BLOCKS ? PLAN_BLOCKS : n_split;  // the grid stays within PLAN_BLOCKS
  int64_t max_mblk = ceil_div(M, CH);
  int64_t n_mblk = 0, mb = 0;
  auto blocks_of = [&](int64_t blocks) {   // the grid stays within `blocks`
    n_mblk = blocks / n_split;
    n_mblk = n_mblk < 1 ? 1 : (n_mblk > max_mblk ? max_mblk : n_mblk);
    mb = ceil_div(ceil_div(M, n_mblk), CH) * CH;
    n_mblk = ceil_div(M, mb);
  };
  blocks_of(PLAN_BLOCKS);
  // Small cohorts: with PLAN_BLOCKS a CTA has one or a few chunks of SNPs, less than what its Q
  // tile, its T partials and the pipeline's start cost (about 4 chunks of the float64 MMA form, 1
  // of the float32 pairs). Of 1 to 12 CTAs per SM (148, a constant, as above), the count whose
  // CTAs finish first, as many at a time as the registers allow (float64: 1). At N=105 x
  // M=8,451, K=7 in float64: 133 CTAs of 4 chunks in one round instead of 529 of one chunk in four.
  // An iteration with PLAN_BLOCKS and with this rule: float64 K=10, 1,000 x 20,000 185 and 136 us,
  // 2,504 x 20,003 359 and 321; but the float64 log-likelihood has the sweep's partition (its
  // partials are the same), runs two CTAs per SM and loses from about 2,000 samples on (2,000 x
  // 12,000 56 and 60 us, 2,504 x 20,003 95 and 117), so the line is at 2,048. Float32 K=8, 5,000 x 30,000 527 and 402 us, 18,000 x 5,000 318 and 255;
  // with K <= 4, whose chunks are short, 5,000 x 30,000 181 and 187, 16,000 x 30,000 536 and 517: no
  // gain to speak of above 2,048 samples.
  const bool mma64 = prec == ADX_F64 && K <= DMMA_MAX_K, pairs32 = prec == ADX_F32 && K <= f32s::MAX_K;
  const int64_t own_tiles = ceil_div(pl.n_stile, n_split);
  const int64_t most = mma64 || K <= 4 ? 2048 : 19999;
  if ((mma64 || pairs32) && N <= most && own_tiles * (mb / CH) < 16) {
    const int64_t slots = mma64 ? 148 : 148 * f32s::ctas_per_sm(K), start = mma64 ? 4 : 1;
    auto rounds = [&]() { return ceil_div(n_split * n_mblk, slots) * own_tiles * (mb / CH + start); };
    int64_t best = rounds(), best_blocks = PLAN_BLOCKS;
    for (int64_t blocks = PLAN_BLOCKS / slots * slots; blocks >= slots; blocks -= slots) {
      blocks_of(blocks);
      if (rounds() < best) { best = rounds(); best_blocks = blocks; }
    }
    blocks_of(best_blocks);
  }
  pl.n_split = (int)n_split;
  pl.n_mblk = (int)n_mblk;
  pl.mb = mb;
  pl.ab_elems = (size_t)n_split * (size_t)M * 2 * K;
  pl.t_elems = (size_t)n_mblk * (size_t)N * K;
  // the float64 tensor-core sweep can also leave one log-likelihood partial per CTA
  if (prec == ADX_F64 && K <= DMMA_MAX_K) pl.extra_bytes = (size_t)n_split * (size_t)n_mblk * sizeof(double);
  return ADX_OK;
}

template <typename R>
static int launch_sweep(const EmPlan& pl, const uint8_t* G, const void* P, const void* Q, void* ws,
                        cudaStream_t st) {
  R* ABp = reinterpret_cast<R*>(reinterpret_cast<uint8_t*>(ws) + EmPlan::HEADER);
  R* Tp = ABp + pl.ab_elems;
  const dim3 grid((unsigned)(pl.n_split * pl.n_mblk));
  if constexpr (sizeof(R) == 4) {
#define ADX_F32_CASE(KK)                                                                                           \
  case KK:                                                                                                         \
    f32s::em_sweep_f32_kernel<KK><<<grid, f32s::TPB, 0, st>>>(G, (const float*)P, (const float*)Q, pl.M, pl.N,       \
                                                              pl.n_stile, pl.n_split, pl.n_mblk, pl.mb, ABp, Tp);  \
    ADX_LAUNCH_CHECK();                                                                                            \
    return ADX_OK;
    switch (pl.K) {
      ADX_F32_CASE(1) ADX_F32_CASE(2) ADX_F32_CASE(3) ADX_F32_CASE(4)
      ADX_F32_CASE(5) ADX_F32_CASE(6) ADX_F32_CASE(7) ADX_F32_CASE(8)
      default: break;
    }
#undef ADX_F32_CASE
  }
  // float32 above K = 8, float64 above K = 16 (the float64 MMA form)
#define LAUNCH(KM)                                                                              \
  em_sweep_kernel<R, KM><<<grid, TPB, 0, st>>>(G, (const R*)P, (const R*)Q, pl.M, pl.N, pl.K,   \
                                               pl.n_stile, pl.n_split, pl.n_mblk, pl.mb, ABp, Tp)
  switch (pl.kmax) {
    case 10: if constexpr (sizeof(R) == 4) { LAUNCH(10); } break;
    case 12: if constexpr (sizeof(R) == 4) { LAUNCH(12); } break;
    case 16: if constexpr (sizeof(R) == 4) { LAUNCH(16); } break;
    case 24: LAUNCH(24); break;
    case 32: LAUNCH(32); break;
    case 48: LAUNCH(48); break;
    case 64: LAUNCH(64); break;
    default: break;
  }
#undef LAUNCH
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

template <typename R>
static int launch_update_from(const EmPlan& pl, const R* ABp, const R* Tp, int mode, double* A, double* B,
                              double* T, const double* q_bat, double* P, double* Q, float* P32, float* Q32,
                              double* mP, double* vP, double* mQ, double* vQ, AdamArgs ad, cudaStream_t st) {
  const int threads = 128;
  // A warp per row where one thread's walk over the partials would be the launch's time: few
  // rows, many partials. One thread per sample took 130 us of a 150 us iteration at N=105 x
  // M=8,451, K=7 (529 partials), and 2.70 -> 2.64 ms at N=10,007 (224 partials); with fewer
  // partials or more rows the threads' neighbouring rows make up for it: at N=15,912 x M=9,908,
  // K=16 (45 and 38 partials) 1.18 ms against 1.21, at N=20,000 (136) 3.97 against 4.02.
  auto lanes = [](int64_t rows, int parts) {
    return (rows <= 4096 && parts >= 32) || (rows < 16384 && parts >= 128) ? 32 : 1;
  };
  const int gp = lanes(pl.M, pl.n_split), gq = lanes(pl.N, pl.n_mblk);
  // every block of the launch on the chip at once (148 SMs, a constant): see the resident kernel
  const int64_t resident_p = pl.K <= RESIDENT_MAX_K ? ceil_div(pl.M, RESIDENT_TPB / pl.K) : 0;
  const int64_t resident = resident_p + ceil_div(pl.N * gq, RESIDENT_TPB);
  if (pl.K <= RESIDENT_MAX_K && gp == 1 && resident <= 148 * RESIDENT_BLOCKS) {
    const unsigned pb = (unsigned)resident_p, blocks = (unsigned)resident;
#define LAUNCH(KM)                                                                                            \
  if constexpr (KM <= RESIDENT_MAX_K)                                                                         \
    em_update_resident_kernel<R, KM><<<blocks, RESIDENT_TPB, 0, st>>>(                                        \
        ABp, Tp, pl.M, pl.N, pl.K, pl.n_split, pl.n_mblk, mode, A, B, T, q_bat, P, Q, P32, Q32, mP, vP, mQ,   \
        vQ, ad, pb, gq);
    ADX_KMAX_SWITCH(pl.kmax, LAUNCH)
#undef LAUNCH
    ADX_LAUNCH_CHECK();
    return ADX_OK;
  }
  const unsigned p_blocks = (unsigned)ceil_div(pl.M * gp, threads);
  const dim3 grid(p_blocks + (unsigned)ceil_div(pl.N * gq, threads));
#define LAUNCH(KM)                                                                          \
  em_update_kernel<R, KM><<<grid, threads, 0, st>>>(ABp, Tp, pl.M, pl.N, pl.K, pl.n_split,  \
                                                    pl.n_mblk, mode, A, B, T, q_bat, P, Q,  \
                                                    P32, Q32, mP, vP, mQ, vQ, ad, p_blocks, gp, gq)
  ADX_KMAX_SWITCH(pl.kmax, LAUNCH)
#undef LAUNCH
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

template <typename R>
static int launch_update(const EmPlan& pl, void* ws, int mode, double* A, double* B, double* T,
                         const double* q_bat, double* P, double* Q, float* P32, float* Q32,
                         double* mP, double* vP, double* mQ, double* vQ, AdamArgs ad,
                         cudaStream_t st) {
  const R* ABp = reinterpret_cast<const R*>(reinterpret_cast<const uint8_t*>(ws) + EmPlan::HEADER);
  return launch_update_from<R>(pl, ABp, ABp + pl.ab_elems, mode, A, B, T, q_bat, P, Q, P32, Q32, mP, vP, mQ,
                               vQ, ad, st);
}

int em_sweep(const EmPlan& pl, const uint8_t* G, const void* P, const void* Q, void* ws,
             cudaStream_t st) {
  if (pl.prec == ADX_BF16 || pl.prec == ADX_F16) {
    float* ABp = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(ws) + EmPlan::HEADER);
    int* err = reinterpret_cast<int*>(ws);
    void* Qb = reinterpret_cast<uint8_t*>(ws) + pl.extra_offset();
    return tc_sweep(G, (const float*)P, (const float*)Q, pl.M, pl.N, pl.K, pl.n_stile, pl.n_split,
                    pl.n_mblk, ABp, ABp + pl.ab_elems, Qb, err, pl.prec == ADX_F16, st);
  }
  if (pl.prec == ADX_F64 && pl.K <= DMMA_MAX_K) {
    double* ABp = reinterpret_cast<double*>(reinterpret_cast<uint8_t*>(ws) + EmPlan::HEADER);
    return dmma_sweep(G, (const double*)P, (const double*)Q, pl.M, pl.N, pl.K, pl.n_stile, pl.n_split,
                      pl.n_mblk, pl.mb, ABp, ABp + pl.ab_elems, st);
  }
  return pl.prec == ADX_F64 ? launch_sweep<double>(pl, G, P, Q, ws, st)
                            : launch_sweep<float>(pl, G, P, Q, ws, st);
}

int em_update(const EmPlan& pl, void* ws, int mode, double* A, double* B, double* T,
              const double* q_bat, double* P, double* Q, float* P32, float* Q32, double* mP,
              double* vP, double* mQ, double* vQ, AdamArgs ad, cudaStream_t st) {
  return pl.prec == ADX_F64
             ? launch_update<double>(pl, ws, mode, A, B, T, q_bat, P, Q, P32, Q32, mP, vP, mQ, vQ, ad, st)
             : launch_update<float>(pl, ws, mode, A, B, T, q_bat, P, Q, P32, Q32, mP, vP, mQ, vQ, ad, st);
}

// Elementwise kernels for the unfused API (em_final_update and step as separate calls).
__global__ void em_targets_kernel(const double* __restrict__ P, const double* __restrict__ Q,
                                  const double* __restrict__ A, const double* __restrict__ B,
                                  const double* __restrict__ T, const double* __restrict__ q_bat,
                                  int64_t M, int64_t N, int K, double* __restrict__ P_EM,
                                  double* __restrict__ Q_EM) {
  const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (row < M) {
    for (int k = 0; k < K; ++k) {
      const int64_t o = row * K + k;
      const double den = fmax((A[o] - B[o]) * P[o] + B[o], 1e-5);
      P_EM[o] = ((1.0 / den) * P[o]) * A[o];
    }
  } else if (row < M + N) {
    const int64_t i = row - M;
    const double scale = 1.0 / fmax(q_bat[i], 1e-5);
    double s = 0.0;
    for (int k = 0; k < K; ++k) s += (Q[i * K + k] * T[i * K + k]) * scale;
    s = fmax(s, 1e-5);
    for (int k = 0; k < K; ++k) Q_EM[i * K + k] = ((Q[i * K + k] * T[i * K + k]) * scale) / s;
  }
}

__global__ void adam_step_kernel(double* __restrict__ P, double* __restrict__ Q,
                                 const double* __restrict__ P_EM, const double* __restrict__ Q_EM,
                                 double* __restrict__ mP, double* __restrict__ vP,
                                 double* __restrict__ mQ, double* __restrict__ vQ, int64_t M,
                                 int64_t N, int K, AdamArgs ad, float* __restrict__ P32,
                                 float* __restrict__ Q32) {
  const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= M + N) return;
  const double t = adam_step_no(ad);
  const double bc1 = 1.0 - pow(ad.b1, t);
  const double bc2 = 1.0 - pow(ad.b2, t);
  const bool isP = row < M;
  const int64_t r = isP ? row : row - M;
  double* X = isP ? P : Q;
  const double* Xt = isP ? P_EM : Q_EM;
  double* m = isP ? mP : mQ;
  double* v = isP ? vP : vQ;
  float* X32 = isP ? P32 : Q32;
  double tot = 0.0;
  for (int k = 0; k < K; ++k) {
    const int64_t o = r * K + k;
    const double x = X[o];
    const double delta = Xt[o] - x;
    const double mm = m[o] * ad.b1 + (1.0 - ad.b1) * delta;
    const double vv = v[o] * ad.b2 + (1.0 - ad.b2) * (delta * delta);
    m[o] = mm;
    v[o] = vv;
    double nx = x + (ad.lr * (mm / bc1)) / (sqrt(vv / bc2) + ad.eps);
    nx = fmin(fmax(nx, DOMAIN), 1.0 - DOMAIN);
    X[o] = nx;
    tot += nx;
  }
  for (int k = 0; k < K; ++k) {
    const int64_t o = r * K + k;
    if (!isP) X[o] = X[o] / tot;
    if (X32) X32[o] = (float)X[o];
  }
}

}  // namespace adx

using namespace adx;

extern "C" int adx_em_workspace_bytes(int64_t M, int64_t N, int K, int precision, size_t* bytes) {
  if (!bytes) return ADX_ERR_ARG;
  EmPlan pl;
  const int rc = em_plan(M, N, K, precision, pl);
  if (rc) { adx_set_message("adx_em_workspace_bytes: bad shape or precision"); return rc; }
  *bytes = pl.bytes();
  return ADX_OK;
}

extern "C" int adx_em_status(void* workspace, size_t workspace_bytes, int64_t M, int64_t N, int K,
                             int precision, int* status, void* stream) {
  EmPlan pl;
  int rc = em_plan(M, N, K, precision, pl);
  if (rc) { adx_set_message("adx_em_status: bad shape or precision"); return rc; }
  if (!workspace || !status) { adx_set_message("adx_em_status: null pointer"); return ADX_ERR_ARG; }
  if (workspace_bytes < pl.bytes()) { adx_set_message("adx_em_status: workspace too small"); return ADX_ERR_WORKSPACE; }
  cudaStream_t st = as_stream(stream);
  int* word = reinterpret_cast<int*>(workspace);
  ADX_CUDA_TRY(cudaMemcpyAsync(status, word, sizeof(int), cudaMemcpyDeviceToHost, st));
  ADX_CUDA_TRY(cudaStreamSynchronize(st));
  ADX_CUDA_TRY(cudaMemsetAsync(word, 0, sizeof(int), st));
  return ADX_OK;
}

extern "C" int adx_em_stats(const uint8_t* G, int64_t M, int64_t N, int K, int precision,
                            const void* P, const void* Q, double* A, double* B, double* T,
                            void* workspace, size_t workspace_bytes, void* stream) {
  EmPlan pl;
  int rc = em_plan(M, N, K, precision, pl);
  if (rc) { adx_set_message("adx_em_stats: bad shape or precision"); return rc; }
  if (!G || !P || !Q || !A || !B || !T || !workspace) { adx_set_message("adx_em_stats: null pointer"); return ADX_ERR_ARG; }
  if (workspace_bytes < pl.bytes()) { adx_set_message("adx_em_stats: workspace too small"); return ADX_ERR_WORKSPACE; }
  cudaStream_t st = as_stream(stream);
  rc = em_sweep(pl, G, P, Q, workspace, st);
  if (rc) return rc;
  return em_update(pl, workspace, 0, A, B, T, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                   nullptr, nullptr, nullptr, AdamArgs{1, 0, 0, 0, 0}, st);
}

extern "C" int adx_em_sweep(const uint8_t* G, int64_t M, int64_t N, int K, int precision,
                            const void* P, const void* Q, void* workspace, size_t workspace_bytes,
                            void* stream) {
  EmPlan pl;
  int rc = em_plan(M, N, K, precision, pl);
  if (rc) { adx_set_message("adx_em_sweep: bad shape or precision"); return rc; }
  if (!G || !P || !Q || !workspace) { adx_set_message("adx_em_sweep: null pointer"); return ADX_ERR_ARG; }
  if (workspace_bytes < pl.bytes()) { adx_set_message("adx_em_sweep: workspace too small"); return ADX_ERR_WORKSPACE; }
  return em_sweep(pl, G, P, Q, workspace, as_stream(stream));
}

extern "C" int adx_em_targets(const double* P, const double* Q, const double* A, const double* B,
                              const double* T, const double* q_bat, int64_t M, int64_t N, int K,
                              double* P_EM, double* Q_EM, void* stream) {
  if (M <= 0 || N <= 0 || K < 1 || K > ADX_MAX_K) { adx_set_message("adx_em_targets: bad shape"); return ADX_ERR_ARG; }
  const int threads = 128;
  em_targets_kernel<<<(unsigned)ceil_div(M + N, threads), threads, 0, as_stream(stream)>>>(
      P, Q, A, B, T, q_bat, M, N, K, P_EM, Q_EM);
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

extern "C" int adx_adam_step(double* P, double* Q, const double* P_EM, const double* Q_EM,
                             double* mP, double* vP, double* mQ, double* vQ, int64_t M, int64_t N,
                             int K, double t, double lr, double beta1, double beta2, double eps,
                             float* P32, float* Q32, void* stream) {
  if (M <= 0 || N <= 0 || K < 1 || K > ADX_MAX_K || t < 1) { adx_set_message("adx_adam_step: bad arguments"); return ADX_ERR_ARG; }
  const int threads = 128;
  adam_step_kernel<<<(unsigned)ceil_div(M + N, threads), threads, 0, as_stream(stream)>>>(
      P, Q, P_EM, Q_EM, mP, vP, mQ, vQ, M, N, K, AdamArgs{t, lr, beta1, beta2, eps}, P32, Q32);
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

extern "C" int adx_em_adam_iteration(const uint8_t* G, int64_t M, int64_t N, int K, int precision,
                                     double* P, double* Q, float* P32, float* Q32, double* mP,
                                     double* vP, double* mQ, double* vQ, const double* q_bat,
                                     double t, double lr, double beta1, double beta2, double eps,
                                     void* workspace, size_t workspace_bytes, void* stream) {
  EmPlan pl;
  int rc = em_plan(M, N, K, precision, pl);
  if (rc) { adx_set_message("adx_em_adam_iteration: bad shape or precision"); return rc; }
  if (!G || !P || !Q || !mP || !vP || !mQ || !vQ || !q_bat || !workspace || t < 1) {
    adx_set_message("adx_em_adam_iteration: bad arguments");
    return ADX_ERR_ARG;
  }
  if (precision != ADX_F64 && (!P32 || !Q32)) { adx_set_message("adx_em_adam_iteration: P32/Q32 required"); return ADX_ERR_ARG; }
  if (workspace_bytes < pl.bytes()) { adx_set_message("adx_em_adam_iteration: workspace too small"); return ADX_ERR_WORKSPACE; }
  cudaStream_t st = as_stream(stream);
  const void* Pin = precision == ADX_F64 ? (const void*)P : (const void*)P32;
  const void* Qin = precision == ADX_F64 ? (const void*)Q : (const void*)Q32;
  rc = em_sweep(pl, G, Pin, Qin, workspace, st);
  if (rc) return rc;
  return em_update(pl, workspace, 1, nullptr, nullptr, nullptr, q_bat, P, Q, P32, Q32, mP, vP, mQ,
                   vQ, AdamArgs{t, lr, beta1, beta2, eps}, st);
}

// ---------------------------------------------------------------- captured iterations
//
// n fused Adam-EM iterations (adx_em_adam_iteration) captured once into a CUDA graph and
// replayed with one launch: 2n kernel launches and their host-side cost become one graph
// launch, which matters when an iteration takes tens of microseconds (small cohorts). The
// Adam step of the replay's iteration i (1..n) is *step_counter + i; adx_em_graph_launch
// first sets the counter to the steps already taken, so a replay computes exactly the n
// eager iterations t0+1..t0+n. Pointers, shapes and the learning rate are fixed at capture;
// the caller keeps every buffer alive, at the same address, for the graph's lifetime.

namespace adx {
__global__ void set_counter_kernel(double* c, double v) { *c = v; }
}  // namespace adx

struct AdxEmGraph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  double* counter = nullptr;
  int n = 0;
};

extern "C" int adx_em_graph_create(const uint8_t* G, int64_t M, int64_t N, int K, int precision, double* P,
                                   double* Q, float* P32, float* Q32, double* mP, double* vP, double* mQ,
                                   double* vQ, const double* q_bat, int n_iters, double lr, double beta1,
                                   double beta2, double eps, double* step_counter, void* workspace,
                                   size_t workspace_bytes, void** graph) {
  EmPlan pl;
  int rc = em_plan(M, N, K, precision, pl);
  if (rc) { adx_set_message("adx_em_graph_create: bad shape or precision"); return rc; }
  if (!G || !P || !Q || !mP || !vP || !mQ || !vQ || !q_bat || !workspace || !step_counter || !graph ||
      n_iters < 1 || n_iters > 4096) {
    adx_set_message("adx_em_graph_create: bad arguments (1 <= n_iters <= 4096, non-null buffers)");
    return ADX_ERR_ARG;
  }
  if (precision != ADX_F64 && (!P32 || !Q32)) { adx_set_message("adx_em_graph_create: P32/Q32 required"); return ADX_ERR_ARG; }
  if (workspace_bytes < pl.bytes()) { adx_set_message("adx_em_graph_create: workspace too small"); return ADX_ERR_WORKSPACE; }
  *graph = nullptr;
  const void* Pin = precision == ADX_F64 ? (const void*)P : (const void*)P32;
  const void* Qin = precision == ADX_F64 ? (const void*)Q : (const void*)Q32;
  // capture on a private stream (the caller's may be the legacy default stream, which cannot
  // be captured); relaxed mode, so a kernel's first-use attribute setup may run inside
  cudaStream_t cs = nullptr;
  ADX_CUDA_TRY(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
  cudaError_t ce = cudaStreamBeginCapture(cs, cudaStreamCaptureModeRelaxed);
  if (ce != cudaSuccess) {
    cudaStreamDestroy(cs);
    adx_set_cuda_error(ce);
    return ADX_ERR_CUDA;
  }
  for (int i = 1; i <= n_iters && !rc; ++i) {
    rc = em_sweep(pl, G, Pin, Qin, workspace, cs);
    if (!rc)
      rc = em_update(pl, workspace, 1, nullptr, nullptr, nullptr, q_bat, P, Q, P32, Q32, mP, vP, mQ, vQ,
                     AdamArgs{(double)i, lr, beta1, beta2, eps, step_counter}, cs);
  }
  cudaGraph_t g = nullptr;
  ce = cudaStreamEndCapture(cs, &g);
  cudaStreamDestroy(cs);
  if (rc || ce != cudaSuccess || !g) {
    if (g) cudaGraphDestroy(g);
    if (!rc) {
      adx_set_cuda_error(ce != cudaSuccess ? ce : cudaErrorStreamCaptureInvalidated);
      rc = ADX_ERR_CUDA;
    }
    cudaGetLastError();
    return rc;
  }
  cudaGraphExec_t ex = nullptr;
  ce = cudaGraphInstantiate(&ex, g, 0ULL);
  if (ce != cudaSuccess) {
    cudaGraphDestroy(g);
    adx_set_cuda_error(ce);
    return ADX_ERR_CUDA;
  }
  *graph = new AdxEmGraph{g, ex, step_counter, n_iters};
  return ADX_OK;
}

extern "C" int adx_em_graph_launch(void* graph, double t0, void* stream) {
  auto* h = static_cast<AdxEmGraph*>(graph);
  if (!h || t0 < 0) { adx_set_message("adx_em_graph_launch: bad arguments"); return ADX_ERR_ARG; }
  cudaStream_t st = as_stream(stream);
  adx::set_counter_kernel<<<1, 1, 0, st>>>(h->counter, t0);
  ADX_LAUNCH_CHECK();
  ADX_CUDA_TRY(cudaGraphLaunch(h->exec, st));
  return ADX_OK;
}

extern "C" int adx_em_graph_iterations(void* graph, int* n_iters) {
  auto* h = static_cast<AdxEmGraph*>(graph);
  if (!h || !n_iters) { adx_set_message("adx_em_graph_iterations: bad arguments"); return ADX_ERR_ARG; }
  *n_iters = h->n;
  return ADX_OK;
}

extern "C" int adx_em_graph_destroy(void* graph) {
  auto* h = static_cast<AdxEmGraph*>(graph);
  if (!h) return ADX_OK;
  if (h->exec) cudaGraphExecDestroy(h->exec);
  if (h->graph) cudaGraphDestroy(h->graph);
  delete h;
  return ADX_OK;
}

// ---------------------------------------------------------------- sweep + log-likelihood
//
// The reference checks the log-likelihood of (P, Q) after an iteration's Adam move, and the
// next iteration's E-step sweeps the same (P, Q). adx_em_sweep_loglik is that sweep with the
// check folded in (float64, K <= 16): the same partials as adx_em_sweep plus the log-
// likelihood of its input, bit-identical to adx_loglik's float64 form; the optimiser reads
// it (adx_em_loglik_from_sweep), takes its decisions, then applies the move
// (adx_em_adam_update), so a check costs no pass of its own.

namespace adx {
// The partials' sum in the order adx_loglik's final sum uses (256 strided sums, then a tree),
// so the two log-likelihoods are bit-identical.
__global__ void ll_sum_kernel(const double* __restrict__ partial, int n, double* __restrict__ out) {
  __shared__ double sh[256];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += partial[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w >= 1; w >>= 1) {
    if ((int)threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
}
}  // namespace adx

static int ll_layout(const EmPlan& pl, void* ws, double** llp) {
  if (pl.prec != ADX_F64 || pl.K > DMMA_MAX_K) return ADX_ERR_UNSUPPORTED;
  *llp = reinterpret_cast<double*>(static_cast<uint8_t*>(ws) + pl.extra_offset());
  return ADX_OK;
}

extern "C" int adx_em_sweep_loglik(const uint8_t* G, int64_t M, int64_t N, int K, int precision, const void* P,
                                   const void* Q, void* workspace, size_t workspace_bytes, void* stream) {
  EmPlan pl;
  int rc = em_plan(M, N, K, precision, pl);
  if (rc) { adx_set_message("adx_em_sweep_loglik: bad shape or precision"); return rc; }
  if (!G || !P || !Q || !workspace) { adx_set_message("adx_em_sweep_loglik: null pointer"); return ADX_ERR_ARG; }
  if (workspace_bytes < pl.bytes()) { adx_set_message("adx_em_sweep_loglik: workspace too small"); return ADX_ERR_WORKSPACE; }
  double* llp = nullptr;
  if (ll_layout(pl, workspace, &llp)) {
    adx_set_message("adx_em_sweep_loglik: float64 with K <= 16 only");
    return ADX_ERR_UNSUPPORTED;
  }
  double* ABp = reinterpret_cast<double*>(static_cast<uint8_t*>(workspace) + EmPlan::HEADER);
  return dmma_sweep(G, (const double*)P, (const double*)Q, M, N, K, pl.n_stile, pl.n_split, pl.n_mblk, pl.mb, ABp,
                    ABp + pl.ab_elems, as_stream(stream), llp);
}

extern "C" int adx_em_loglik_from_sweep(void* workspace, size_t workspace_bytes, int64_t M, int64_t N, int K,
                                        int precision, double* out, void* stream) {
  EmPlan pl;
  int rc = em_plan(M, N, K, precision, pl);
  if (rc) { adx_set_message("adx_em_loglik_from_sweep: bad shape or precision"); return rc; }
  if (!workspace || !out) { adx_set_message("adx_em_loglik_from_sweep: null pointer"); return ADX_ERR_ARG; }
  if (workspace_bytes < pl.bytes()) { adx_set_message("adx_em_loglik_from_sweep: workspace too small"); return ADX_ERR_WORKSPACE; }
  double* llp = nullptr;
  if (ll_layout(pl, workspace, &llp)) {
    adx_set_message("adx_em_loglik_from_sweep: float64 with K <= 16 only");
    return ADX_ERR_UNSUPPORTED;
  }
  ll_sum_kernel<<<1, 256, 0, as_stream(stream)>>>(llp, pl.n_split * pl.n_mblk, out);
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

extern "C" int adx_em_adam_update(int64_t M, int64_t N, int K, int precision, double* P, double* Q, float* P32,
                                  float* Q32, double* mP, double* vP, double* mQ, double* vQ, const double* q_bat,
                                  double t, double lr, double beta1, double beta2, double eps, void* workspace,
                                  size_t workspace_bytes, void* stream) {
  EmPlan pl;
  int rc = em_plan(M, N, K, precision, pl);
  if (rc) { adx_set_message("adx_em_adam_update: bad shape or precision"); return rc; }
  if (!P || !Q || !mP || !vP || !mQ || !vQ || !q_bat || !workspace || t < 1) {
    adx_set_message("adx_em_adam_update: bad arguments");
    return ADX_ERR_ARG;
  }
  if (workspace_bytes < pl.bytes()) { adx_set_message("adx_em_adam_update: workspace too small"); return ADX_ERR_WORKSPACE; }
  return em_update(pl, workspace, 1, nullptr, nullptr, nullptr, q_bat, P, Q, P32, Q32, mP, vP, mQ, vQ,
                   AdamArgs{t, lr, beta1, beta2, eps}, as_stream(stream));
}

// ---------------------------------------------------------------- block-range sweeps
//
// The float64 sweep (K <= 16) over a range of its SNP blocks, for callers that upload the
// packed matrix in pieces and sweep each piece as it lands: the partition is the full
// sweep's, each block's partial sums depend on that block alone, so the ranges of one
// workspace add up to exactly the full sweep.

extern "C" int adx_em_sweep_blocks_info(int64_t M, int64_t N, int K, int precision, int64_t* snps_per_block,
                                        int* n_blocks, int* ctas_per_block) {
  EmPlan pl;
  const int rc = em_plan(M, N, K, precision, pl);
  if (rc || !snps_per_block || !n_blocks || !ctas_per_block) { adx_set_message("adx_em_sweep_blocks_info: bad arguments"); return rc ? rc : ADX_ERR_ARG; }
  if (precision != ADX_F64 || K > DMMA_MAX_K) {
    adx_set_message("adx_em_sweep_blocks_info: float64 with K <= 16 only");
    return ADX_ERR_UNSUPPORTED;
  }
  *snps_per_block = pl.mb;
  *n_blocks = pl.n_mblk;
  *ctas_per_block = pl.n_split;
  return ADX_OK;
}

extern "C" int adx_em_sweep_blocks(const uint8_t* G, int64_t M, int64_t N, int K, int precision, const void* P,
                                   const void* Q, int b0, int b1, void* workspace, size_t workspace_bytes,
                                   void* stream) {
  EmPlan pl;
  int rc = em_plan(M, N, K, precision, pl);
  if (rc) { adx_set_message("adx_em_sweep_blocks: bad shape or precision"); return rc; }
  if (precision != ADX_F64 || K > DMMA_MAX_K) {
    adx_set_message("adx_em_sweep_blocks: float64 with K <= 16 only");
    return ADX_ERR_UNSUPPORTED;
  }
  if (!G || !P || !Q || !workspace || b0 < 0 || b1 > pl.n_mblk || b0 >= b1) {
    adx_set_message("adx_em_sweep_blocks: bad arguments (0 <= b0 < b1 <= n_blocks)");
    return ADX_ERR_ARG;
  }
  if (workspace_bytes < pl.bytes()) { adx_set_message("adx_em_sweep_blocks: workspace too small"); return ADX_ERR_WORKSPACE; }
  double* ABp = reinterpret_cast<double*>(static_cast<uint8_t*>(workspace) + EmPlan::HEADER);
  return dmma_sweep(G, (const double*)P, (const double*)Q, M, N, K, pl.n_stile, pl.n_split, pl.n_mblk, pl.mb, ABp,
                    ABp + pl.ab_elems, as_stream(stream), nullptr, b0, b1);
}

// The float64 log-likelihood on the float64 MMA (em_sweep_dmma.cu) uses the float64 sweep's
// partition; ADX_ERR_UNSUPPORTED when K > 16.
namespace adx {
int dmma_loglik_plan(int64_t M, int64_t N, int K, int64_t& n_stile, int& n_split, int& n_mblk, int64_t& mb) {
  if (K > DMMA_MAX_K) return ADX_ERR_UNSUPPORTED;
  EmPlan pl;
  const int rc = em_plan(M, N, K, ADX_F64, pl);
  if (rc) return rc;
  n_stile = pl.n_stile;
  n_split = pl.n_split;
  n_mblk = pl.n_mblk;
  mb = pl.mb;
  return ADX_OK;
}
}  // namespace adx

// ---------------------------------------------------------------- batched float64 E-step
//
// Several E-step problems on one cohort (K <= 16 each; e.g. the K sweep and its cross-
// validation folds) in one launch of the float64 tensor-core sweep. All of them share the
// float64 sweep's partition (it does not depend on K), so each problem's partial sums, and
// hence its statistics, are bit-identical to a single-problem sweep of the same P, Q and
// (fold-masked) genotypes. Workspace: a 256-byte header, then per problem its A/B partials
// and T partials, each 256-byte aligned.

namespace adx {
int dmma_sweep_batch(int64_t M, int64_t N, int n, const int* K, const uint8_t* const* G, const double* const* P,
                     const double* const* Q, double* const* ABp, double* const* Tp, int64_t n_stile, int n_split,
                     int n_mblk, int64_t mb, cudaStream_t st);
}

static int batch_layout(int64_t M, int64_t N, int n, const int* K, EmPlan& pl, size_t* offs, size_t* total) {
  if (n < 1 || n > 64 || !K) return ADX_ERR_ARG;
  for (int p = 0; p < n; ++p)
    if (K[p] < 1 || K[p] > DMMA_MAX_K) return ADX_ERR_ARG;
  const int rc = em_plan(M, N, K[0], ADX_F64, pl);
  if (rc) return rc;
  size_t off = EmPlan::HEADER;
  for (int p = 0; p < n; ++p) {
    if (offs) offs[p] = off;
    const size_t ab = (size_t)pl.n_split * (size_t)M * 2 * K[p], tt = (size_t)pl.n_mblk * (size_t)N * K[p];
    off = (off + (ab + tt) * sizeof(double) + 255) & ~size_t(255);
  }
  *total = off;
  return ADX_OK;
}

extern "C" int adx_em_batch_workspace_bytes(int64_t M, int64_t N, int n, const int* K, size_t* bytes) {
  EmPlan pl;
  if (!bytes) return ADX_ERR_ARG;
  const int rc = batch_layout(M, N, n, K, pl, nullptr, bytes);
  if (rc) adx_set_message("adx_em_batch_workspace_bytes: bad shape or K (1 <= n <= 64 problems, 1 <= K <= 16)");
  return rc;
}

extern "C" int adx_em_sweep_batch(int64_t M, int64_t N, int n, const int* K, const uint8_t* const* G,
                                  const double* const* P, const double* const* Q, void* workspace,
                                  size_t workspace_bytes, void* stream) {
  EmPlan pl;
  size_t offs[64], total = 0;
  int rc = batch_layout(M, N, n, K, pl, offs, &total);
  if (rc || !G || !P || !Q || !workspace) {
    adx_set_message("adx_em_sweep_batch: bad argument (1 <= n <= 64 problems, 1 <= K <= 16)");
    return rc ? rc : ADX_ERR_ARG;
  }
  if (workspace_bytes < total) { adx_set_message("adx_em_sweep_batch: workspace too small"); return ADX_ERR_WORKSPACE; }
  double* ABp[64];
  double* Tp[64];
  for (int p = 0; p < n; ++p) {
    if (!G[p] || !P[p] || !Q[p]) { adx_set_message("adx_em_sweep_batch: null pointer"); return ADX_ERR_ARG; }
    ABp[p] = reinterpret_cast<double*>(static_cast<uint8_t*>(workspace) + offs[p]);
    Tp[p] = ABp[p] + (size_t)pl.n_split * (size_t)M * 2 * K[p];
  }
  return dmma_sweep_batch(M, N, n, K, G, P, Q, ABp, Tp, pl.n_stile, pl.n_split, pl.n_mblk, pl.mb,
                          as_stream(stream));
}

extern "C" int adx_em_batch_apply(int64_t M, int64_t N, int n, const int* K, int p, int mode, double* A, double* B,
                                  double* T, const double* q_bat, double* P, double* Q, double* mP, double* vP,
                                  double* mQ, double* vQ, double t, double lr, double beta1, double beta2,
                                  double eps, void* workspace, size_t workspace_bytes, void* stream) {
  EmPlan pl;
  size_t offs[64], total = 0;
  const int rc = batch_layout(M, N, n, K, pl, offs, &total);
  if (rc || p < 0 || p >= n || !workspace || (mode != 0 && mode != 1)) {
    adx_set_message("adx_em_batch_apply: bad argument");
    return rc ? rc : ADX_ERR_ARG;
  }
  if (workspace_bytes < total) { adx_set_message("adx_em_batch_apply: workspace too small"); return ADX_ERR_WORKSPACE; }
  if (mode == 0 ? (!A || !B || !T) : (!q_bat || !P || !Q || !mP || !vP || !mQ || !vQ || t < 1)) {
    adx_set_message("adx_em_batch_apply: bad argument");
    return ADX_ERR_ARG;
  }
  EmPlan pp;
  em_plan(M, N, K[p], ADX_F64, pp);
  const double* ABp = reinterpret_cast<const double*>(static_cast<const uint8_t*>(workspace) + offs[p]);
  const double* Tp = ABp + (size_t)pl.n_split * (size_t)M * 2 * K[p];
  return launch_update_from<double>(pp, ABp, Tp, mode, A, B, T, q_bat, P, Q, nullptr, nullptr, mP, vP, mQ, vQ,
                                    AdamArgs{t, lr, beta1, beta2, eps}, as_stream(stream));
}
