// Tensor-core (tcgen05, sm_100a) form of the E-step sweep: BF16 or FP16 operands, FP32
// accumulation in tensor memory. Same statistics and the same partial-sum layout as
// em_sweep_kernel (adamixture/model/em_adam_gpu.py:46-78), for 1 <= K <= 16 (K padded to 16
// in the MMAs).
//
// Operand formats (one kind::f16 MMA takes both operands in the same format):
//   BF16: 8-bit significand, values as they are.
//   FP16: 11-bit significand (8x finer rounding at the same MMA rate), with power-of-two
//         scalings that keep every operand in FP16's normal range: P, 1-P and Q are stored
//         x8 (values >= 1e-5 become >= 8e-5; the smallest normal is 6.1e-5). H then holds
//         64 h, so the ratio step's 1/H and 1/Hc are a/64 and b/64 with no extra operation
//         (from 1/64 up to 2/(64 * 1e-5) = 3125, inside FP16's normal range), and A/B/T
//         accumulate 1/8 of their value: the partial-sum writes multiply by 8.
//
// Per CTA: R = 7 SNP tiles of 128 SNPs (896 SNPs) and a residue class of 128-sample tiles.
// For each step (sample tile s, SNP tile r), in two half-steps of 64 samples:
//   H  = P_r  . Q_s^T      (tcgen05.mma M=128 SNPs, N=64 samples, K=16)         -> TMEM
//   Hc = (1-P_r) . Q_s^T   (the complement, so 1-h stays accurate when h -> 1)  -> TMEM
//   consumer warps read H/Hc rows from TMEM and form, per entry (one reciprocal each),
//     a = g / max(h,1e-5),  b = (2-g) / max(1-h,1e-5)   (0 where missing)
//   as BF16/FP16 tiles in shared memory; after both halves
//   A_r += a . Q_s, B_r += b . Q_s   (M=128 SNPs, N=16, K=128 samples; TMEM, all sample tiles)
//   T   += a^T . P_r + b^T . (1-P_r) (M=128 samples, N=16, K=128 SNPs; TMEM, all SNP tiles)
// After the R SNP tiles of a sample tile, T (over the CTA's 896 SNPs) goes to the T partials;
// after the last sample tile, A_r/B_r go to the A/B partials of the CTA's split.
//
// Warp specialisation: HALF_WGS warpgroups form the ratios of the first 64 samples of every
// step and as many those of the second 64 (each warpgroup a block of WG_COLS samples). One
// warp streams the G tiles (a ring of NG stages) and the converted Q tiles (NQ buffers) into
// shared memory with cp.async. Three warps issue the MMAs from precomputed shared-memory
// descriptors (one 64-bit add per operand): H, A/B and T. H/Hc live in two TMEM buffers (one per
// half) and the a/b tiles in two shared-memory buffers (one per step parity), so while the
// warpgroups form the ratios of a step the tensor pipe runs the next step's H and the A/B/T
// MMAs of the previous one. There is no block-wide barrier in the loop: the warps meet only at
// mbarriers, and loop counters advance incrementally (no division).
//
// TMEM (512 columns, one CTA per SM): H/Hc buffer b at [128b, 128b+128) (H first 64, Hc
// last 64) | T [256,272) and [496,512) (even and odd sample tiles) | A_r,B_r [272+32r, 304+32r)
// for r < 7.
// Shared-memory operands use the no-swizzle canonical layout (8-row x 16-byte core
// matrices). One copy of each tile serves both of its MMA views: P_r is the K-major A of H
// and the MN-major B of T; Q_s is the K-major B of H and the MN-major B of A/B; the a/b
// tiles are the K-major A of A/B and the MN-major A of T.
//
// Synchronisation (mbarriers): hfull (tcgen05.commit: a step's H is done), hfree (an arrival
// per consumer warp: it holds its H in registers, the buffers are free), abready[step parity]
// (an arrival per consumer warp: its a/b columns are written; two barriers, so that no phase can
// pass unseen by an issuer that is a step behind), abfree[step parity] (two commits: the step's
// A/B and T are done), gfull[g] and qfull[q] (32 cp.async arrivals: G stage g / Q buffer q is
// loaded), gfree[g] (an arrival per consumer warp) and qfree[q] (a commit). The consumers take
// their whole block of H at once and free the buffer before the arithmetic, so the next step's
// H is there when they come back for it. T has two buffers and is read two steps later, when
// abfree says that its last batch is done.
//
// N=200,000 x M=500,000, K=10: 75.1 ms (330 GB/s of algorithmic bytes, 106 TFLOP/s). An MMA of the
// A/B and T batches (M=128, N=16) runs for about 100 cycles beside the consumers and holds its
// issuer for as long, and a wait of the issuer drains the pipe for some 450 cycles: with one warp
// that loads and issues everything a step takes 5,200 cycles instead of 3,450 (113.9 ms).
// Every wait is bounded and also watches a shared abort word; on a timeout the kernel
// records ADX_ERR_TIMEOUT in the status word, all warps leave their loops, it waits (bounded)
// for its MMAs in flight, frees its TMEM and returns.
#include <algorithm>
#include <functional>
#include <queue>
#include <vector>

#include "tcgen05.cuh"

#ifndef ADX_TC_HALF_WGS
#define ADX_TC_HALF_WGS 2
#endif

namespace adx {
namespace tc {

constexpr int TILE = 128;      // SNPs per SNP tile, samples per sample tile
constexpr int KP = 16;         // padded K
constexpr int R = 7;           // SNP tiles per CTA
constexpr int SNP_BLOCK = R * TILE;
constexpr int HALF = TILE / 2;                          // samples per half-step
constexpr int HALF_WGS = ADX_TC_HALF_WGS;               // consumer warpgroups per half
constexpr int WG_COLS = HALF / HALF_WGS;                // samples per warpgroup and half-step
constexpr int CONSUMER_WARPS = 2 * 4 * HALF_WGS;
constexpr int LOAD_WARP = CONSUMER_WARPS, H_WARP = LOAD_WARP + 1, AB_WARP = LOAD_WARP + 2, T_WARP = LOAD_WARP + 3;
constexpr int TPB = CONSUMER_WARPS * 32 + 128;
constexpr int NG = 4;          // G stages
constexpr int NQ = 3;          // Q buffers
static_assert(WG_COLS % 16 == 0, "warpgroup column blocks are whole 16-column TMEM loads");

// shared-memory map (bytes)
constexpr int P_TILE_BYTES = TILE * KP * 2;             // 4096 (also one Q tile)
constexpr int G_ROW = TILE + 16;                        // padded packed row of a G tile
constexpr int G_TILE_BYTES = (TILE / 4) * G_ROW;        // 32 packed rows
constexpr int AB_TILE_BYTES = TILE * TILE * 2;          // 32768
constexpr int OFF_P = 0;                                // R x (P, 1-P)
constexpr int OFF_Q = OFF_P + R * 2 * P_TILE_BYTES;     // NQ buffers
constexpr int OFF_G = OFF_Q + NQ * P_TILE_BYTES;        // NG stages
constexpr int OFF_A = OFF_G + NG * G_TILE_BYTES;        // 2 buffers
constexpr int OFF_B = OFF_A + 2 * AB_TILE_BYTES;        // 2 buffers
constexpr int OFF_BAR = OFF_B + 2 * AB_TILE_BYTES;      // mbarriers
constexpr int N_BARS = 9 + 2 * NG + 2 * NQ;
constexpr int OFF_TMEM = OFF_BAR + 8 * N_BARS;          // TMEM address, then the abort word
constexpr int SMEM_BYTES = OFF_TMEM + 16;
constexpr int SMEM_ALLOC = SMEM_BYTES + 1024;           // room to align the base to 1024
static_assert(SMEM_ALLOC <= 227 * 1024, "shared memory budget");
static_assert(OFF_G % 16 == 0 && G_TILE_BYTES % 16 == 0 && G_ROW % 16 == 0, "cp.async alignment");
// descriptor start addresses are 14-bit fields of 16-byte units: offsets added to a base
// descriptor never carry out of the field while the whole map stays below 256 KiB
static_assert(SMEM_ALLOC < 256 * 1024, "descriptor start field");

// TMEM columns
constexpr uint32_t COL_AB = 272;
__device__ __forceinline__ uint32_t col_t(int sidx) { return (sidx & 1) ? 496u : 256u; }  // T of the CTA's sample tile sidx

// ---------------------------------------------------------------- descriptors

// Instruction descriptor, kind::f16: A/B format fmt (0 = FP16, 1 = BF16) for both, FP32 D,
// M = 128.
__host__ __device__ constexpr uint32_t idesc(int N, int a_mn, int b_mn, uint32_t fmt) {
  return (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
         ((uint32_t)(N >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
}

// Byte offsets inside the tiles (element size 2).
// P / Q tiles: (row, k), rows of 8 form core matrices of 128 B; k halves 128 B apart.
__device__ __forceinline__ uint32_t off_pq(int row, int k) {
  return (uint32_t)((row >> 3) * 256 + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2);
}
// a / b tiles: (snp j, sample i): sample groups of 8 are 128 B apart, SNP groups 2048 B.
__device__ __forceinline__ uint32_t off_ab(int j, int i) {
  return (uint32_t)((i >> 3) * 128 + (j >> 3) * 2048 + (j & 7) * 16 + (i & 7) * 2);
}

// ---------------------------------------------------------------- PTX wrappers

__device__ __forceinline__ void mma_f16kind(uint32_t tmem_d, uint64_t ad, uint64_t bd, uint32_t id,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
      :
      : "r"(tmem_d), "l"(ad), "l"(bd), "r"(id), "r"(accumulate));
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// Packed float32 pairs: mul.rn.f32x2 multiplies both lanes as two scalar IEEE multiplies do.
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

// Operand format traits. GA/GB: the genotype weights g -> {0, 1, 2, 0} (a) and
// g -> {2, 1, 0, 0} (b) as 16-bit pairs, looked up with one byte permute per pair (entry g
// at bytes 2g..2g+1 of {hi:lo}). PQ_SCALE: factor on stored P, 1-P and Q; H_UNITS: h in
// H's units (the 1e-5 clamp is applied there); OUT_SCALE: factor that takes the
// accumulated A/B/T back to their values.
template <bool F16>
struct Fmt;
template <>
struct Fmt<false> {
  static constexpr uint32_t CODE = 1;  // BF16
  static constexpr uint32_t GA_LO = 0x3F800000u, GA_HI = 0x00004000u;
  static constexpr uint32_t GB_LO = 0x3F804000u, GB_HI = 0x00000000u;
  static constexpr float PQ_SCALE = 1.0f, H_UNITS = 1.0f, OUT_SCALE = 1.0f;
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
  }
  static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
  }
};
template <>
struct Fmt<true> {
  static constexpr uint32_t CODE = 0;  // FP16
  static constexpr uint32_t GA_LO = 0x3C000000u, GA_HI = 0x00004000u;
  static constexpr uint32_t GB_LO = 0x3C004000u, GB_HI = 0x00000000u;
  static constexpr float PQ_SCALE = 8.0f, H_UNITS = 64.0f, OUT_SCALE = 8.0f;
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
  }
  static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
  }
};

// ---------------------------------------------------------------- kernel

struct Args {
  const uint8_t* G;
  const float* P;     // [M][K] float32
  const uint8_t* Qb;  // converted Q tiles [n_stile][4096 B], shared-memory layout
  int64_t M, N;
  int K;
  int64_t n_stile;    // sample tiles
  int n_split;
  int n_mblk;         // SNP blocks of 896
  float* ABp;         // [n_split][M][2K]
  float* Tp;          // [n_mblk][N][K]
  int* err;
};

// Q (float32 [N][K]) -> operand-format tiles (x PQ_SCALE) of 128 samples x 16 in the
// shared-memory layout of a Q tile (rows past N and columns past K are zero), so the
// producer copies them verbatim.
template <bool F16>
__global__ void q_to_tiles_kernel(const float* __restrict__ Q, int64_t N, int K, int64_t n_stile,
                                  uint8_t* __restrict__ Qb) {
  using F = Fmt<F16>;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_stile * TILE * 2) return;
  const int64_t tile = e / (TILE * 2);
  const int row = (int)((e >> 1) % TILE), kh = (int)(e & 1) * 8;
  const int64_t i = tile * TILE + row;
  float f[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int k = kh + q;
    f[q] = (i < N && k < K) ? __ldg(Q + i * K + k) * F::PQ_SCALE : 0.0f;
  }
  *reinterpret_cast<uint4*>(Qb + tile * P_TILE_BYTES + off_pq(row, kh)) =
      make_uint4(F::pack(f[0], f[1]), F::pack(f[2], f[3]), F::pack(f[4], f[5]), F::pack(f[6], f[7]));
}

// G tile (32 packed rows x 128 samples) into a shared-memory stage by the producer warp: lane
// l copies row l as whole 16-byte chunks by cp.async, and the lane's arrival on `bar` fires
// when they land. AL: every packed row starts 16-byte aligned (N % 16 == 0 and G aligned), 8
// chunks. Otherwise the 9 chunks from the 16-byte boundary at or below the row's first byte
// (they cover the 128 samples at any offset); the consumers apply the offset, which is a
// constant of the row within the tile (row_offset). A sample count that is not a multiple of
// 16 is what real cohorts have: N=10,007 x M=200,003, K=8 takes 1.9 ms, as the aligned shape
// (loaded byte by byte through one warp: 15 ms).
// Chunks that would leave the matrix (the last row or two) take byte loads; bytes past the
// matrix are 0xFF (missing). Samples past N read the next row's bytes or 0xFF: their Q rows
// are zero, so they add nothing to A and B, and their T is not written. Rows past the matrix
// are not loaded: the consumers count them as missing.
template <bool AL>
__device__ __forceinline__ void producer_load_g(const Args& a, int64_t row0, int64_t i0, uint8_t* gs, uint32_t bar) {
  constexpr int CHUNKS = AL ? TILE / 16 : TILE / 16 + 1;
  static_assert(16 * CHUNKS <= G_ROW, "the chunks fit the padded row");
  const int l = threadIdx.x & 31;
  const int64_t row = row0 + l;
  const int64_t rows = (a.M + 3) >> 2;
  uint8_t* dst = gs + l * G_ROW;
  if (row >= rows) {
    mbar_arrive(bar);
    return;
  }
  const uint8_t* src = a.G + row * a.N + i0;
  if constexpr (!AL) src -= reinterpret_cast<uintptr_t>(src) & 15;
  const uint8_t* end = a.G + rows * a.N;
  if (src >= a.G && src + 16 * CHUNKS <= end) {
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) cp_async16(smem_u32(dst + 16 * c), src + 16 * c);
    cp_async_arrive(bar);
  } else {
    for (int c = 0; c < 4 * CHUNKS; ++c) {
      uint32_t x = 0;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const uint8_t* p = src + c * 4 + b;
        x |= (p >= a.G && p < end ? (uint32_t)__ldg(p) : 0xFFu) << (8 * b);
      }
      *reinterpret_cast<uint32_t*>(dst + 4 * c) = x;
    }
    mbar_arrive(bar);
  }
}

// Offset (bytes) of a tile's first sample in row `lr` (0..31) of an unaligned G stage: tiles
// start at packed rows and samples that are multiples of 16, so it is the same in every tile.
static_assert(TILE % 64 == 0 && SNP_BLOCK % 64 == 0, "tiles start at packed rows that are multiples of 16");
__device__ __forceinline__ uint32_t row_offset(const Args& a, int lr) {
  return ((uint32_t)(reinterpret_cast<uintptr_t>(a.G) & 15) + (uint32_t)lr * (uint32_t)(a.N & 15)) & 15u;
}

// Converted Q tile (4096 B) into a shared-memory buffer by the producer warp: lane l copies
// bytes [128 l, 128 l + 128).
__device__ __forceinline__ void producer_load_q(const Args& a, int64_t tile, uint8_t* qs, uint32_t bar) {
  const int l = threadIdx.x & 31;
  const uint8_t* src = a.Qb + tile * P_TILE_BYTES + l * 128;
#pragma unroll
  for (int c = 0; c < 8; ++c) cp_async16(smem_u32(qs + l * 128 + 16 * c), src + 16 * c);
  cp_async_arrive(bar);
}

template <bool F16, bool AL>
__global__ void __launch_bounds__(TPB, 1) em_sweep_tc_kernel(Args a) {
  using F = Fmt<F16>;
  constexpr uint32_t ID_H = idesc(HALF, 0, 0, F::CODE);   // A = P (K-major), B = Q half (K-major)
  constexpr uint32_t ID_AB = idesc(KP, 0, 1, F::CODE);    // A = a (K-major), B = Q (MN-major)
  constexpr uint32_t ID_T = idesc(KP, 1, 1, F::CODE);     // A = a^T (MN-major), B = P (MN-major)
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(sm + OFF_TMEM);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_TMEM + 4);
  const uint32_t bars = smem_u32(sm + OFF_BAR);
  const uint32_t HFULL = bars, HFREE = bars + 8u;
  auto ABREADY = [&](int st) { return bars + 16u + 8u * (uint32_t)(st & 1); };
  auto ABFREE = [&](int st) { return bars + 32u + 8u * (uint32_t)(st & 1); };
  auto GFULL = [&](int g) { return bars + 48u + 8u * (uint32_t)g; };
  auto GFREE = [&](int g) { return bars + 48u + 8u * (uint32_t)(NG + g); };
  auto QFULL = [&](int q) { return bars + 48u + 8u * (uint32_t)(2 * NG + q); };
  auto QFREE = [&](int q) { return bars + 48u + 8u * (uint32_t)(2 * NG + NQ + q); };
  auto DRAIN = [&](int w) { return bars + 48u + 8u * (uint32_t)(2 * NG + 2 * NQ + w - H_WARP); };
  // all lanes of a warp leave a wait with the same answer
  auto warp_wait = [](uint32_t bar, uint32_t parity, volatile int* flag) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, flag));
  };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const int mblk = blockIdx.x % a.n_mblk;
  const int split = blockIdx.x / a.n_mblk;
  const int64_t jb = (int64_t)mblk * SNP_BLOCK;
  const int r_eff = (int)min((int64_t)R, (a.M - jb + TILE - 1) / TILE);
  const int64_t s_first = split;
  const int n_my = (int)((a.n_stile - split + a.n_split - 1) / a.n_split);  // sample tiles of this CTA
  const int nsteps = n_my * r_eff;

  // ---- prologue: TMEM (H warp), barriers, P tiles (all threads)
  if (warp == H_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_holder)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    *abort_flag = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(HFULL));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(HFREE), "r"(CONSUMER_WARPS));
    for (int b = 0; b < 2; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(ABREADY(b)), "r"(CONSUMER_WARPS));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(ABFREE(b)));   // A/B and T
    }
    for (int w = H_WARP; w <= T_WARP; ++w) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(DRAIN(w)));
    for (int g = 0; g < NG; ++g) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 32;" ::"r"(GFULL(g)));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(GFREE(g)), "r"(CONSUMER_WARPS));
    }
    for (int q = 0; q < NQ; ++q) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 32;" ::"r"(QFULL(q)));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(QFREE(q)));
    }
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  for (int e = tid; e < r_eff * TILE * 2; e += TPB) {
    const int r = e / (TILE * 2), row = (e / 2) % TILE, kh = (e & 1) * 8;
    const int64_t j = jb + (int64_t)r * TILE + row;
    float p[8], c[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int k = kh + q;
      const bool ok = j < a.M && k < a.K;
      const float v = ok ? __ldg(a.P + j * a.K + k) : 0.0f;
      p[q] = v * F::PQ_SCALE;
      c[q] = ok ? (1.0f - v) * F::PQ_SCALE : 0.0f;
    }
    uint8_t* pt = sm + OFF_P + r * 2 * P_TILE_BYTES;
    *reinterpret_cast<uint4*>(pt + off_pq(row, kh)) =
        make_uint4(F::pack(p[0], p[1]), F::pack(p[2], p[3]), F::pack(p[4], p[5]), F::pack(p[6], p[7]));
    *reinterpret_cast<uint4*>(pt + P_TILE_BYTES + off_pq(row, kh)) =
        make_uint4(F::pack(c[0], c[1]), F::pack(c[2], c[3]), F::pack(c[4], c[5]), F::pack(c[6], c[7]));
  }
  fence_async_smem();
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_holder;
  const float ELO = (float)E_CLAMP * F::H_UNITS;

  // Base descriptors; the offsets added below are in 16-byte units.
  const uint32_t s_p = smem_u32(sm + OFF_P), s_q = smem_u32(sm + OFF_Q), s_a = smem_u32(sm + OFF_A);
  const uint64_t dPK = sdesc(s_p, 128, 256);    // P_r K-major (A of H): + 512 r; 1-P: + 256
  const uint64_t dQK = sdesc(s_q, 128, 256);    // Q K-major (B of H): + 256 qb + 128 half
  const uint64_t dQM = sdesc(s_q, 256, 128);    // Q MN-major (B of A/B): + 256 qb + 32 ks
  const uint64_t dAK = sdesc(s_a, 128, 2048);   // a K-major (A of A/B): + 2048 buf + 16 ks; b: + 4096
  const uint64_t dAM = sdesc(s_a, 2048, 128);   // a MN-major (A of T): + 2048 buf + 256 ks; b: + 4096
  const uint64_t dPM = sdesc(s_p, 256, 128);    // P_r MN-major (B of T): + 512 r + 32 ks; 1-P: + 256
  constexpr uint64_t B_OFF = (uint64_t)(OFF_B - OFF_A) >> 4;

  // H/Hc of both halves of a step on SNP tile r and Q buffer qb
  auto issue_h = [&](int r, int qb) {
    const uint64_t ap = dPK + (uint64_t)(r * 512);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint64_t bq = dQK + (uint64_t)(qb * 256 + h * 128);
      const uint32_t col = tmem + (uint32_t)h * 128;
      mma_f16kind(col, ap, bq, ID_H, 0);
      mma_f16kind(col + HALF, ap + 256, bq, ID_H, 0);
    }
  };
  // A/B MMAs of a step on SNP tile r, Q buffer qb, a/b buffer buf, of the CTA's sample tile sidx
  auto issue_ab = [&](int r, int qb, int buf, int sidx) {
    const uint64_t qm = dQM + (uint64_t)(qb * 256);
    const uint64_t ak = dAK + (uint64_t)(buf * 2048);
    const uint32_t tab = tmem + COL_AB + 32u * (uint32_t)r;
#pragma unroll
    for (int ks = 0; ks < TILE / 16; ++ks) {
      const uint32_t acc = (sidx > 0 || ks > 0) ? 1u : 0u;
      mma_f16kind(tab, ak + 16 * ks, qm + 32 * ks, ID_AB, acc);
      mma_f16kind(tab + 16, ak + B_OFF + 16 * ks, qm + 32 * ks, ID_AB, acc);
    }
  };
  // its T MMAs
  auto issue_t = [&](int r, int buf, int sidx) {
    const uint32_t tt = tmem + col_t(sidx);
    const uint64_t am = dAM + (uint64_t)(buf * 2048);
    const uint64_t pm = dPM + (uint64_t)(r * 512);
#pragma unroll
    for (int ks = 0; ks < TILE / 16; ++ks) {
      const uint32_t acc = (r > 0 || ks > 0) ? 1u : 0u;
      mma_f16kind(tt, am + 256 * ks, pm + 32 * ks, ID_T, acc);
      mma_f16kind(tt, am + B_OFF + 256 * ks, pm + 256 + 32 * ks, ID_T, 1u);
    }
  };
  auto write_t = [&](int sidx) {  // one warpgroup: T rows (samples) of the CTA's sample tile sidx
    const int64_t s = s_first + (int64_t)sidx * a.n_split;
    uint32_t v[16];
    tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + col_t(sidx), v);
    tmem_wait_ld();
    const int64_t i = s * TILE + (warp & 3) * 32 + lane;
    if (i < a.N) {
      float* dst = a.Tp + ((int64_t)mblk * a.N + i) * a.K;
#pragma unroll
      for (int k = 0; k < KP; ++k)
        if (k < a.K) dst[k] = __uint_as_float(v[k]) * F::OUT_SCALE;
    }
  };

  bool aborted = false;
  if (warp == LOAD_WARP) {
    // ---------------------------------------------------------------- loads
    // G of step m goes to stage m % NG; with the first step of the CTA's sample tile t, its Q tile
    // goes to buffer t % NQ. Both wait for the previous fill's readers.
    int mr = 0, t = 0, gstage = 0, qbuf = 0;
    uint32_t gfill = 0, qfill = 0;
    for (int m = 0; m < nsteps; ++m) {
      if (mr == 0) {
        if (qfill > 0 && !warp_wait(QFREE(qbuf), (qfill - 1) & 1u, abort_flag)) { aborted = true; break; }
        producer_load_q(a, s_first + (int64_t)t * a.n_split, sm + OFF_Q + qbuf * P_TILE_BYTES, QFULL(qbuf));
        if (++qbuf == NQ) { qbuf = 0; ++qfill; }
      }
      if (gfill > 0 && !warp_wait(GFREE(gstage), (gfill - 1) & 1u, abort_flag)) { aborted = true; break; }
      producer_load_g<AL>(a, (jb + (int64_t)mr * TILE) >> 2, (s_first + (int64_t)t * a.n_split) * TILE,
                          sm + OFF_G + gstage * G_TILE_BYTES, GFULL(gstage));
      if (++mr == r_eff) { mr = 0; ++t; }
      if (++gstage == NG) { gstage = 0; ++gfill; }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp >= H_WARP) {
    // ---------------------------------------------------------------- MMAs
    // Three warps issue: H, A/B and T, each from one lane (an accumulator's MMAs come from one
    // thread, which keeps their order). The issue of a batch holds its thread about as long as
    // the batch runs, and a wait behind it costs some 450 cycles before the next batch starts, in
    // which a single issuer leaves the tensor pipe idle (5,200 cycles a step for 3,400 of MMAs);
    // here the other batches run meanwhile.
    if (lane == 0) {
      auto wait = [&](uint32_t bar, uint32_t parity) {
        if (!aborted && !mbar_wait(bar, parity, abort_flag)) aborted = true;
      };
      int r = 0, sidx = 0, qb = 0;   // the step's SNP tile, sample tile, Q buffer
      uint32_t qpar = 0u;            // parity of the Q buffer's fill for that sample tile
      for (int st = 0; st < nsteps; ++st) {
        if (warp == H_WARP) {
          if (st > 0) wait(HFREE, (uint32_t)(st - 1) & 1u);
          if (r == 0) {
            wait(QFULL(qb), qpar);
            fence_async_smem();
          }
        } else {
          wait(ABREADY(st), (uint32_t)(st >> 1) & 1u);
        }
        if (aborted) break;
        fence_after();
        if (warp == H_WARP) {
          issue_h(r, qb);
          mma_commit(HFULL);
        } else if (warp == AB_WARP) {
          issue_ab(r, qb, st & 1, sidx);
          mma_commit(ABFREE(st));
          if (r + 1 == r_eff) mma_commit(QFREE(qb));   // the tile's last batch; its H's were done before
        } else {
          issue_t(r, st & 1, sidx);
          mma_commit(ABFREE(st));
        }
        if (++r == r_eff) {
          r = 0;
          ++sidx;
          if (++qb == NQ) { qb = 0; qpar ^= 1u; }
        }
      }
    }
    __syncwarp();
  } else {
    // ---------------------------------------------------------------- consumers
    const int hw = warp / (4 * HALF_WGS);       // half of every step
    const int sub = (warp >> 2) % HALF_WGS;     // column block inside the half
    const int wq = warp & 3;                    // TMEM lane quarter
    const int jl = wq * 32 + lane;              // SNP row within the tile
    const int colb = hw * HALF + sub * WG_COLS; // first sample column inside the step's tile
    const uint32_t trow = tmem + ((uint32_t)(wq * 32) << 16) + (uint32_t)(hw * 128 + sub * WG_COLS);
    // bit shift of the SNP's field in a sample's byte; unaligned rows are read as words from
    // the word at or below the thread's first sample, and one funnel shift takes off both
    // the byte offset in the word and the field's position (at most 24 + 6 bits)
    const uint32_t goff = AL ? 0u : row_offset(a, jl >> 2);
    const uint32_t sh = 2u * (uint32_t)(jl & 3) + 8u * (goff & 3u);
    int r = 0, sidx = 0, gstage = 0, rprev = 0, sprev = 0;
    uint32_t gph = 0u;
    for (int st = 0; st < nsteps; ++st) {
      if (!warp_wait(HFULL, (uint32_t)st & 1u, abort_flag)) { aborted = true; break; }
      if (!warp_wait(GFULL(gstage), gph, abort_flag)) { aborted = true; break; }
      fence_after();
      const int64_t jglob = jb + (int64_t)r * TILE + jl;
      const uint8_t* gs = sm + OFF_G + gstage * G_TILE_BYTES + (jl >> 2) * G_ROW + colb + (goff & ~3u);
      uint8_t* ta = sm + OFF_A + (st & 1) * AB_TILE_BYTES;
      uint8_t* tb = sm + OFF_B + (st & 1) * AB_TILE_BYTES;
      // all of the warpgroup's H and Hc, then the buffer is free for the next step's
      constexpr int NCH = WG_COLS / 16;
      static_assert(NCH == 2, "the whole block of columns is held in registers");
      uint32_t hv[NCH][16], cv[NCH][16];
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        tmem_ld16(trow + 16 * c, hv[c]);
        tmem_ld16(trow + HALF + 16 * c, cv[c]);
      }
      tmem_wait_ld();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(HFREE);
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        const int cur = c;
        const int col0 = colb + 16 * c;
        uint32_t words[5];
        if constexpr (AL) {
          const uint4 gw = *reinterpret_cast<const uint4*>(gs + 16 * c);
          words[0] = gw.x; words[1] = gw.y; words[2] = gw.z; words[3] = gw.w; words[4] = 0;
        } else {
#pragma unroll
          for (int q = 0; q < 5; ++q) words[q] = *reinterpret_cast<const uint32_t*>(gs + 16 * c + 4 * q);
        }
        uint32_t ap[8], bp[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t tq = (AL ? words[q] >> sh : __funnelshift_r(words[q], words[q + 1], sh)) & 0x03030303u;
          if (jglob >= a.M) tq = 0x03030303u;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const int e = q * 4 + half * 2;
            const uint32_t x = half ? (tq >> 16) : (tq & 0x0303u);
            const uint32_t sel = x * 0x22u + 0x1010u;
            const float rec0 = fmaxf(__uint_as_float(hv[cur][e]), ELO);
            const float rec1 = fmaxf(__uint_as_float(hv[cur][e + 1]), ELO);
            const float omr0 = fmaxf(__uint_as_float(cv[cur][e]), ELO);
            const float omr1 = fmaxf(__uint_as_float(cv[cur][e + 1]), ELO);
            // the pair's products as packed float32 multiplies (each lane the scalar product)
            const uint64_t rr = pack_f32x2(rec0, rec1), oo = pack_f32x2(omr0, omr1);
            float x0, x1;
            unpack_f32x2(mul_f32x2(rr, oo), x0, x1);
            const uint64_t rp = pack_f32x2(rcp_approx(x0), rcp_approx(x1));
            float y0, y1, z0, z1;
            unpack_f32x2(mul_f32x2(oo, rp), y0, y1);
            unpack_f32x2(mul_f32x2(rr, rp), z0, z1);
            const uint32_t ypair = F::pack(y0, y1);  // 1/rec (FP16: 1/(64 rec))
            const uint32_t xpair = F::pack(z0, z1);  // 1/(1-rec)
            ap[e >> 1] = F::mul(prmt(F::GA_LO, F::GA_HI, sel), ypair);
            bp[e >> 1] = F::mul(prmt(F::GB_LO, F::GB_HI, sel), xpair);
          }
        }
        if (c == 0 && st > 1) {
          // the a/b buffer's last batch, of step st - 2, is done
          if (!warp_wait(ABFREE(st), (uint32_t)((st >> 1) - 1) & 1u, abort_flag)) { aborted = true; break; }
          // ... and with it T of a sample tile that ended there (T alternates between two
          // buffers: the current tile's is the other one or, with one SNP tile per CTA, the same
          // one, whose next batch waits for this warpgroup's arrival below)
          if (hw == 1 && sub == 0 && rprev == 0 && sprev > 0) {
            fence_after();
            write_t(sprev - 1);
            fence_before();
          }
        }
        *reinterpret_cast<uint4*>(ta + off_ab(jl, col0)) = make_uint4(ap[0], ap[1], ap[2], ap[3]);
        *reinterpret_cast<uint4*>(ta + off_ab(jl, col0 + 8)) = make_uint4(ap[4], ap[5], ap[6], ap[7]);
        *reinterpret_cast<uint4*>(tb + off_ab(jl, col0)) = make_uint4(bp[0], bp[1], bp[2], bp[3]);
        *reinterpret_cast<uint4*>(tb + off_ab(jl, col0 + 8)) = make_uint4(bp[4], bp[5], bp[6], bp[7]);
      }
      if (aborted) break;
      rprev = r;
      sprev = sidx;
      fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(ABREADY(st));
        mbar_arrive(GFREE(gstage));
      }
      if (++r == r_eff) { r = 0; ++sidx; }
      if (++gstage == NG) { gstage = 0; gph ^= 1u; }
    }
  }

  // ---- epilogue: wait for the last MMAs (the last step's commit covers everything)
  if (!aborted && warp != LOAD_WARP) {
    if (!mbar_wait(ABFREE(nsteps - 1), (uint32_t)((nsteps - 1) >> 1) & 1u, abort_flag)) aborted = true;
  }
  if (__syncthreads_or(aborted)) {
    if (tid == 0) atomicExch(a.err, ADX_ERR_TIMEOUT);
    if (warp >= H_WARP) {
      // MMAs may still be in flight: one more commit and a bounded wait before TMEM is freed
      volatile int never = 0;
      if (lane == 0) mma_commit(DRAIN(warp));
      (void)mbar_wait(DRAIN(warp), 0u, &never);
    }
  } else {
    fence_after();
    // the last tiles' T: the last one's, and with one SNP tile per CTA the one before it
    if (warp >= 4 * HALF_WGS && warp < 4 * HALF_WGS + 4) {
      if (r_eff == 1 && n_my > 1) write_t(n_my - 2);
      write_t(n_my - 1);
    }
    if (warp < 8) {
      // A/B of every SNP tile: warps 0-3 read A, warps 4-7 read B
      const int wg = warp >> 2, wq = warp & 3;
      for (int r = 0; r < r_eff; ++r) {
        uint32_t v[16];
        tmem_ld16(tmem + ((uint32_t)(wq * 32) << 16) + COL_AB + 32 * r + 16 * wg, v);
        tmem_wait_ld();
        const int64_t j = jb + (int64_t)r * TILE + wq * 32 + lane;
        if (j < a.M) {
          float* dst = a.ABp + ((int64_t)split * a.M + j) * (2 * a.K) + wg * a.K;
#pragma unroll
          for (int k = 0; k < KP; ++k)
            if (k < a.K) dst[k] = __uint_as_float(v[k]) * F::OUT_SCALE;
        }
      }
    }
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == H_WARP) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  }
}

// Self-test of the bounded wait above: one mbarrier expecting one arrival. With arrive = 0
// nothing arrives, so thread 0's wait gives up after `limit` polls, reports ADX_ERR_TIMEOUT
// and raises the abort word, and a second warp's wait on the same barrier must then leave
// at once; with arrive = 1 both waits complete. status[0..2]: the first wait's result, the
// abort word, the second wait's result.
__global__ void wait_selftest_kernel(int arrive, uint32_t limit, int* status) {
  __shared__ __align__(8) uint64_t bar_word;
  __shared__ int abort_word;
  const uint32_t bar = smem_u32(&bar_word);
  if (threadIdx.x == 0) {
    abort_word = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (arrive) mbar_arrive(bar);
    const bool ok = mbar_wait(bar, 0u, &abort_word, limit);
    status[0] = ok ? ADX_OK : ADX_ERR_TIMEOUT;
    status[1] = abort_word;
  }
  __syncthreads();
  if (threadIdx.x == 32) status[2] = mbar_wait(bar, 0u, &abort_word, limit) ? ADX_OK : ADX_ERR_TIMEOUT;
}

}  // namespace tc

namespace {

constexpr int NUM_SMS = 148;          // one CTA per SM (tensor memory and shared memory)
constexpr int64_t CTA_OVERHEAD = 3;   // prologue, pipeline fill and drain, in steps

// Finish time, in steps, of the grid (blockIdx = split * n_mblk + mblk) dispatched in
// blockIdx order onto NUM_SMS SMs, each CTA starting when an SM frees up. A CTA runs
// n_my(split) x r_eff(mblk) steps.
int64_t tc_makespan(int64_t M, int64_t n_stile, int n_split, int n_mblk) {
  std::priority_queue<int64_t, std::vector<int64_t>, std::greater<int64_t>> free_at;
  for (int i = 0; i < NUM_SMS; ++i) free_at.push(0);
  const int64_t m_tiles = ceil_div(M, tc::TILE);
  int64_t end = 0;
  for (int s = 0; s < n_split; ++s) {
    const int64_t n_my = (n_stile - s + n_split - 1) / n_split;
    for (int b = 0; b < n_mblk; ++b) {
      const int64_t r_eff = std::min<int64_t>(tc::R, m_tiles - (int64_t)b * tc::R);
      const int64_t t = free_at.top() + n_my * r_eff + CTA_OVERHEAD;
      free_at.pop();
      free_at.push(t);
      end = std::max(end, t);
    }
  }
  return end;
}

// Sample splits: the count, around the one that gives about 8 waves, whose grid finishes
// first (a smaller count unless a larger one is at least 0.2 % faster). The last wave of
// a fixed 8-wave rule can be mostly idle: at M=500,000 it ran a third full. The search
// costs about 3 ms of host time at N=200,000 x M=500,000 and up to about 60 ms at extreme
// aspect ratios (M=896 x N=10^7, M=10^8 x N=1000), once per shape: the last 4 shapes are
// cached per thread.
int tc_pick_split(int64_t M, int64_t n_stile, int n_mblk) {
  struct Entry { int64_t M, n_stile; int n_split; };
  thread_local Entry cache[4] = {};
  thread_local int next = 0;
  for (const Entry& e : cache)
    if (e.n_split > 0 && e.M == M && e.n_stile == n_stile) return e.n_split;
  const int64_t lo = std::max<int64_t>(1, std::min<int64_t>(n_stile, ceil_div(8 * NUM_SMS, n_mblk)));
  const int64_t hi = std::min<int64_t>(n_stile, 2 * lo + 8);
  int64_t best_t = -1, best_n = lo;
  for (int64_t n = std::max<int64_t>(1, lo / 2); n <= hi; ++n) {
    const int64_t t = tc_makespan(M, n_stile, (int)n, n_mblk);
    if (best_t < 0 || 1000 * t < 998 * best_t) { best_t = t; best_n = n; }
  }
  cache[next] = Entry{M, n_stile, (int)best_n};
  next = (next + 1) % 4;
  return (int)best_n;
}

}  // namespace

int tc_plan(int64_t M, int64_t N, int K, int64_t& n_stile, int& n_split, int& n_mblk) {
  if (M <= 0 || N <= 0 || K < 1 || K > tc::KP) return ADX_ERR_UNSUPPORTED;
  n_stile = ceil_div(N, tc::TILE);
  n_mblk = (int)ceil_div(M, tc::SNP_BLOCK);
  n_split = tc_pick_split(M, n_stile, n_mblk);
  return ADX_OK;
}

size_t tc_q_bytes(int64_t n_stile) { return (size_t)n_stile * tc::P_TILE_BYTES; }

template <bool F16, bool AL>
static int tc_launch(const tc::Args& a, int64_t n_stile, uint8_t* qb, const float* Q, cudaStream_t st) {
  static bool attr_set[64] = {false};
  int dev = 0;
  ADX_CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    ADX_CUDA_TRY(cudaFuncSetAttribute(tc::em_sweep_tc_kernel<F16, AL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      tc::SMEM_ALLOC));
    attr_set[dev] = true;
  }
  tc::q_to_tiles_kernel<F16><<<(unsigned)ceil_div(n_stile * tc::TILE * 2, 256), 256, 0, st>>>(Q, a.N, a.K,
                                                                                                n_stile, qb);
  ADX_LAUNCH_CHECK();
  tc::em_sweep_tc_kernel<F16, AL><<<(unsigned)(a.n_split * a.n_mblk), tc::TPB, tc::SMEM_ALLOC, st>>>(a);
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

extern "C" int adx_tc_wait_selftest(int arrive, uint32_t limit, int* status, void* stream) {
  if (!status || limit < 1) {
    adx_set_message("adx_tc_wait_selftest: bad argument");
    return ADX_ERR_ARG;
  }
  tc::wait_selftest_kernel<<<1, 64, 0, as_stream(stream)>>>(arrive, limit, status);
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

int tc_sweep(const uint8_t* G, const float* P, const float* Q, int64_t M, int64_t N, int K,
             int64_t n_stile, int n_split, int n_mblk, float* ABp, float* Tp, void* Qb, int* err,
             bool f16, cudaStream_t st) {
  uint8_t* qb = static_cast<uint8_t*>(Qb);
  const tc::Args a{G, P, qb, M, N, K, n_stile, n_split, n_mblk, ABp, Tp, err};
  // aligned rows need one 16-byte shared load per 16 samples instead of five 4-byte ones
  const bool al = (N & 15) == 0 && (reinterpret_cast<uintptr_t>(G) & 15) == 0;
  if (f16) return al ? tc_launch<true, true>(a, n_stile, qb, Q, st) : tc_launch<true, false>(a, n_stile, qb, Q, st);
  return al ? tc_launch<false, true>(a, n_stile, qb, Q, st) : tc_launch<false, false>(a, n_stile, qb, Q, st);
}

}  // namespace adx
