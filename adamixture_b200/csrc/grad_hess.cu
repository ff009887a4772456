// Gradient and Hessian passes of the original ADMIXTURE (BR-QN) algorithm in float64,
// straight from the packed genotypes:
//
//   Q side (per sample i):  Xtz_q[i] = sum_j a_ji P_j + b_ji (1 - P_j)
//                           XtX_q[i] = sum_j (a_ji / h_ji) P_j P_j' + (b_ji / (1-h_ji)) (1-P_j)(1-P_j)'
//   P side (per SNP j):     Xtz_p[j] = sum_i (a_ji - b_ji) Q_i
//                           XtX_p[j] = sum_i (a_ji / h_ji + b_ji / (1-h_ji)) Q_i Q_i'
//
// with h = clamp(P_j . Q_i, 1e-10, 1 - 1e-10), a = g / h, b = (2 - g) / (1 - h), missing
// entries skipped. adamixture/model/br_qn_gpu.py:67-214 (the reference materialises the
// coefficient matrices per 8192-SNP chunk and contracts them with einsum); the per-entry
// arithmetic follows adamixture/src/utils_c/cython/sqp.pyx:258-328.
//
// Each pass is a GEMM with a fused prologue. The Hessian of a row (sample for Q, SNP for P)
// is a weighted sum over the other axis of per-entry pair products -- P_jk P_jl (and the
// complement's) for the Q side, Q_ik Q_il for the P side -- and those products do not depend
// on the row. Everything is float64 MMAs (mma.sync .f64); what bounds it is the float64 pipe,
// which the MMAs share with the scalar operations, so the work is kept to the K at hand.
//
// K <= 16 (grad_hess_mma_kernel, instantiated per K): a CTA of 4 warps owns 64 rows and walks
// a range of the other axis ("reduced") in chunks of 32. Per chunk the CTA stages the factor
// rows and forms the pair products of the (k <= l) pairs, rounded up to 8 columns, and the
// gradient's columns, in shared memory. A warp owns 16 rows: per 8 reduced entries it forms
// h with MMAs, turns each h into its coefficients in place, and feeds them to the Hessian's
// and the gradient's MMAs from registers: the accumulator layout of h is the A layout of
// those once column 2t + e of the h tile is k-slot t + 4e. So no coefficient goes through
// shared memory and no barrier stands between the two contractions.
// Reduced entry 8t + 2nt + e of a chunk is column 2t + e of h tile nt: a thread's 8 entries of a row
// are 8 consecutive genotypes (two packed bytes on the Q side, 8 bytes on the P side).
// Measured at N=20,000 x M=50,000, K=10: Q side 17.4 -> 11.4 ms, P side 12.4 -> 7.2 ms; at
// N=2,504 x M=100,003, K=7: 3.8 -> 1.9 and 2.8 -> 1.2 ms (before: 64-row x 64-pair tiles with the
// coefficients staged in shared memory, K = 7's 28 pairs padded to 64).
//
// K > 16 (grad_hess_kernel): a CTA owns 64 rows and 64 pairs and walks the other axis in
// chunks of 32: per chunk it stages the factor rows, forms the 32 x 64 pair products and the
// 64 x 32 coefficients (h, then a/h and b/(1-h)) once in shared memory, and each warp owns
// 32 rows x 16 pairs as 2 x 2 MMA tiles (m16n8k4), loading its fragments from shared memory
// whose rows are padded by 4 doubles so a fragment load is conflict-free.
//
// Every chunk enters the MMAs whole: entries past the reduced axis have zero coefficients.
// Ranges of the reduced axis are split across CTAs when the row tiles alone do not fill the
// GPU; their sums meet in float64 atomics on the zeroed outputs.
#include "common.cuh"

namespace adx {
namespace gh {

constexpr int TR = 64;       // rows per tile
constexpr int TP = 64;       // pairs per tile
constexpr int CJ = 32;       // reduced-axis entries per chunk
constexpr int TPB = 256;     // 8 warps: 2 row blocks of 32 x 4 pair blocks of 16
constexpr int CSTR = TR + 4; // padded row stride of the coefficient tiles (doubles)
constexpr int PSTR = TP + 4; // padded row stride of the pair-product tiles (doubles)

struct Args {
  const uint8_t* G;
  const double* P;   // [M][K]
  const double* Q;   // [N][K]
  int64_t M, N;
  int K;
  double* XtX;       // [rows][K][K]
  double* Xtz;       // [rows][K]
  int n_pblk;        // pair blocks
  int n_split;       // splits of the reduced axis
  int64_t chunks_per_split;
};

// d (4 doubles: rows g, g, g+8, g+8; columns 2t, 2t+1, 2t, 2t+1 of a 16 x 8 tile) +=
// A (16 x 4: a0 row g, a1 row g+8, column t) . B (4 x 8: b0 row t, column g), float64
// tensor-core MMA; g = lane / 4, t = lane % 4.
__device__ __forceinline__ void mma_f64(double (&d)[4], double a0, double a1, double b0) {
  asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
               : "d"(a0), "d"(a1), "d"(b0));
}

// shared-memory layout (doubles unless noted)
struct Smem {
  double *own, *fac, *coef, *zc, *pp;
  uint8_t *pk, *pl;
  static __host__ size_t bytes(int K, int nt) {
    return sizeof(double) * ((size_t)(TR + CJ) * K + (size_t)nt * CJ * 2 * CSTR + (size_t)nt * CJ * PSTR) + 2 * TP;
  }
  __device__ Smem(uint8_t* base, int K, int nt) {
    double* d = reinterpret_cast<double*>(base);
    own = d; d += TR * K;            // [TR][K] factors of the tile's rows
    fac = d; d += CJ * K;            // [CJ][K] factors of the chunk's reduced entries
    coef = d; d += nt * CJ * CSTR;   // [nt][CJ][CSTR] Hessian coefficients
    zc = d; d += nt * CJ * CSTR;     // [nt][CJ][CSTR] gradient coefficients
    pp = d; d += nt * CJ * PSTR;     // [nt][CJ][PSTR] pair products
    pk = reinterpret_cast<uint8_t*>(d);
    pl = pk + TP;
  }
};

// Any K up to 64: the gradient's MMA tiles are 64 rows x 8 column tiles of 8 over 8 warps.
template <bool QSIDE>
__global__ void __launch_bounds__(TPB) grad_hess_kernel(Args a) {
  constexpr int NTG = (ADX_MAX_K + 7) / 8;   // gradient column tiles
  constexpr int GT = (4 * NTG + 7) / 8;      // gradient tiles per warp
  constexpr int NT = QSIDE ? 2 : 1;   // coefficient terms
  extern __shared__ __align__(16) uint8_t smem[];
  const int K = a.K;
  Smem s(smem, K, NT);
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int fg = lane >> 2, ft = lane & 3;   // MMA fragment group and thread in group
  const int wr = warp & 1, wp = warp >> 1;   // the warp's row block (32) and pair block (16)
  const int64_t n_rows = QSIDE ? a.N : a.M;
  const int64_t n_red = QSIDE ? a.M : a.N;
  const double* ownF = QSIDE ? a.Q : a.P;
  const double* redF = QSIDE ? a.P : a.Q;

  int64_t b = blockIdx.x;
  const int pblk = (int)(b % a.n_pblk); b /= a.n_pblk;
  const int split = (int)(b % a.n_split); b /= a.n_split;
  const int64_t row0 = b * TR;
  const int n_pairs = K * (K + 1) / 2;
  const bool do_grad = pblk == 0;

  // pair table: pairs pblk*TP + t in row-major order of the upper triangle
  for (int t = tid; t < TP; t += TPB) {
    int p = pblk * TP + t, k = 0;
    if (p < n_pairs) {
      while (p >= K - k) { p -= K - k; ++k; }
      s.pk[t] = (uint8_t)k;
      s.pl[t] = (uint8_t)(k + p);
    } else {
      s.pk[t] = 0xFF;
      s.pl[t] = 0xFF;
    }
  }
  for (int e = tid; e < TR * K; e += TPB) {
    const int r = e / K, k = e - r * K;
    const int64_t row = row0 + r;
    s.own[e] = row < n_rows ? ownF[row * K + k] : 0.0;
  }

  double acc[2][2][4];   // [row tile][pair tile][fragment]
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[i][j][v] = 0.0;
  // gradient: 4 row tiles x NTG column tiles of 16 x 8; warp w owns tiles w, w + 8, ...
  double gacc[GT][4];
#pragma unroll
  for (int q = 0; q < GT; ++q)
#pragma unroll
    for (int v = 0; v < 4; ++v) gacc[q][v] = 0.0;

  const int64_t n_chunks = (n_red + CJ - 1) / CJ;
  const int64_t ch0 = (int64_t)split * a.chunks_per_split;
  const int64_t ch1 = min(n_chunks, ch0 + a.chunks_per_split);
  for (int64_t ch = ch0; ch < ch1; ++ch) {
    const int64_t red0 = ch * CJ;
    __syncthreads();  // the previous chunk's readers are done
    {
      // the chunk's factor rows are contiguous: a flat copy, zeros past the reduced axis
      const int64_t base = red0 * K, end = n_red * K;
      for (int e = tid; e < CJ * K; e += TPB) s.fac[e] = base + e < end ? redF[base + e] : 0.0;
    }
    __syncthreads();
    // pair products of the chunk's entries (shared by every row); TPB is a multiple of
    // TP, so a thread's entries all have pair t = tid % TP
    {
      static_assert(TPB % TP == 0, "one pair per thread");
      const int t = tid & (TP - 1);
      const int k = s.pk[t], l = s.pl[t];
      for (int c = tid / TP; c < CJ; c += TPB / TP) {
        double v0 = 0.0, v1 = 0.0;
        if (k != 0xFF) {
          const double fk = s.fac[c * K + k], fl = s.fac[c * K + l];
          v0 = fk * fl;
          if (QSIDE) v1 = (1.0 - fk) * (1.0 - fl);
        }
        s.pp[c * PSTR + t] = v0;
        if (QSIDE) s.pp[CJ * PSTR + c * PSTR + t] = v1;
      }
    }
    // coefficients of the TR x CJ entries; lanes walk the sample axis of G.
    // A thread's 8 entries run along the SNP axis -- Q side: chunk entries 8 (tid >> 6) + n
    // of row tid & 63; P side: rows 8 (tid >> 5) + n of chunk entry tid & 31 -- so they come
    // from two packed genotype bytes (SNPs snp0 .. snp0 + 7 of one sample).
    const int fixed = QSIDE ? (tid & (TR - 1)) : (tid & (CJ - 1));
    const int first = QSIDE ? 8 * (tid >> 6) : 8 * (tid >> 5);
    const int64_t smp = (QSIDE ? row0 : red0) + fixed;
    const int64_t snp0 = (QSIDE ? red0 : row0) + first;   // a multiple of 8
    uint32_t gbytes = 0xFFFFu;                              // all missing outside the matrix
    if (smp < a.N) {
      if (snp0 < a.M) gbytes = (gbytes & 0xFF00u) | (uint32_t)a.G[(snp0 >> 2) * a.N + smp];
      if (snp0 + 4 < a.M) gbytes = (gbytes & 0x00FFu) | ((uint32_t)a.G[((snp0 >> 2) + 1) * a.N + smp] << 8);
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int r = QSIDE ? fixed : first + n;
      const int c = QSIDE ? first + n : fixed;
      const int64_t row = row0 + r, red = red0 + c;
      double w1 = 0.0, w2 = 0.0, z1 = 0.0, z2 = 0.0;
      if (row < n_rows && red < n_red) {
        const unsigned g = (gbytes >> (2 * n)) & 3u;   // SNP snp0 + n
        if (g != 3u) {
          double h = 0.0;
          for (int k = 0; k < K; ++k) h += s.own[r * K + k] * s.fac[c * K + k];
          h = fmax(fmin(h, 1.0 - 1e-10), 1e-10);
          const double gd = (double)g, om = 1.0 - h;
          // 1/h and 1/(1-h) from one reciprocal of x = h(1-h) in [1e-10, 0.25]: the hardware
          // approximation refined by two Newton-Raphson steps r <- r (2 - x r), each of which
          // squares the relative error (within a unit or two of the last place after both)
          const double x = h * om;
          double rr;
          asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(rr) : "d"(x));
          rr = fma(rr, fma(-x, rr, 1.0), rr);
          rr = fma(rr, fma(-x, rr, 1.0), rr);
          const double ih = om * rr, iom = h * rr;
          z1 = gd * ih;
          z2 = (2.0 - gd) * iom;
          w1 = z1 * ih;
          w2 = z2 * iom;
        }
      }
      if (QSIDE) {
        s.coef[c * CSTR + r] = w1;
        s.coef[CJ * CSTR + c * CSTR + r] = w2;
        s.zc[c * CSTR + r] = z1;
        s.zc[CJ * CSTR + c * CSTR + r] = z2;
      } else {
        s.coef[c * CSTR + r] = w1 + w2;
        s.zc[c * CSTR + r] = z1 - z2;
      }
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      // A (rows x chunk entries) = coef^T, B (chunk entries x pairs) = pp: fragment
      // element (row fg [+8], entry ft) of A, (entry ft, pair fg) of B
      const double* cf = s.coef + t * CJ * CSTR + wr * 32 + fg;
      const double* pr = s.pp + t * CJ * PSTR + wp * 16 + fg;
#pragma unroll
      for (int c0 = 0; c0 < CJ; c0 += 4) {
        const double* ca = cf + (c0 + ft) * CSTR;
        const double* pb = pr + (c0 + ft) * PSTR;
        const double a00 = ca[0], a01 = ca[8], a10 = ca[16], a11 = ca[24];
        const double b0 = pb[0], b1 = pb[8];
        mma_f64(acc[0][0], a00, a01, b0);
        mma_f64(acc[0][1], a00, a01, b1);
        mma_f64(acc[1][0], a10, a11, b0);
        mma_f64(acc[1][1], a10, a11, b1);
      }
    }
    if (do_grad) {
      // Xtz += z1' fac (+ z2' (1 - fac) on the Q side): A = z (rows x chunk entries),
      // B = the chunk's factor rows, columns k >= K fed zeros
#pragma unroll
      for (int q = 0; q < GT; ++q) {
        const int tix = warp + 8 * q;
        if (tix >= 4 * NTG) break;   // warp-uniform
        const int mt = tix & 3, k = (tix >> 2) * 8 + fg;
        const bool kin = k < K;
        const double* z = s.zc + mt * 16 + fg;
#pragma unroll
        for (int c0 = 0; c0 < CJ; c0 += 4) {
          const int c = c0 + ft;
          const double f = kin ? s.fac[c * K + k] : 0.0;
          mma_f64(gacc[q], z[c * CSTR], z[c * CSTR + 8], f);
          if (QSIDE) mma_f64(gacc[q], z[(CJ + c) * CSTR], z[(CJ + c) * CSTR + 8], kin ? 1.0 - f : 0.0);
        }
      }
    }
  }

  // scatter: both halves of the symmetric Hessian; accumulator v of tile (i, j) is row
  // fg (+8 for v >= 2), pair 2 ft + (v & 1) of the tile
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int64_t row = row0 + wr * 32 + i * 16 + fg + (v >> 1) * 8;
      if (row >= n_rows) continue;
      double* H = a.XtX + row * K * K;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int t = wp * 16 + j * 8 + 2 * ft + (v & 1);
        const int k = s.pk[t];
        if (k == 0xFF) continue;
        const int l = s.pl[t];
        atomicAdd(H + k * K + l, acc[i][j][v]);
        if (l != k) atomicAdd(H + l * K + k, acc[i][j][v]);
      }
    }
  if (do_grad) {
#pragma unroll
    for (int q = 0; q < GT; ++q) {
      const int tix = warp + 8 * q;
      if (tix >= 4 * NTG) break;
      const int mt = tix & 3, nt = tix >> 2;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int64_t row = row0 + mt * 16 + fg + (v >> 1) * 8;
        const int k = nt * 8 + 2 * ft + (v & 1);
        if (row < n_rows && k < K) atomicAdd(a.Xtz + row * K + k, gacc[q][v]);
      }
    }
  }
}

// ---------------------------------------------------------------- K <= 16

constexpr int RW = 16;        // rows per warp
constexpr int MWARPS = 4;     // warps per CTA
static_assert(MWARPS * RW == TR, "row tiles");

__device__ __forceinline__ void mma_f64_k8(double (&d)[4], double a0, double a1, double a2, double a3, double b0,
                                           double b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
               : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

// Pair blocks of at most 10 column tiles, column tiles of a pair block, and the CTAs per SM that
// their accumulators' registers allow: for the kernels and for the host's choice of splits.
__host__ __device__ constexpr int pair_blocks(int K) { return (K * (K + 1) / 2 + 79) / 80; }
__host__ __device__ constexpr int pair_tiles(int K) { return ((K * (K + 1) / 2 + pair_blocks(K) - 1) / pair_blocks(K) + 7) / 8; }
__host__ __device__ constexpr int ctas_per_sm(int K) { return pair_tiles(K) <= 4 ? 4 : pair_tiles(K) <= 7 ? 3 : 2; }

template <bool QSIDE, int K>
struct Shape {
  static constexpr int KS = (K + 3) / 4;                       // h's k-steps of 4
  static constexpr int NTG = (K + 7) / 8;                      // gradient column tiles
  static constexpr int PAIRS = K * (K + 1) / 2;
  static constexpr int NPB = pair_blocks(K);
  static constexpr int NP = pair_tiles(K);
  static constexpr int TPC = 8 * NP;
  static constexpr int COLS = TPC + 8 * NTG;                   // pairs, then the gradient's columns
  static constexpr int CS = COLS + 2;                          // = 2 mod 8: 16-byte fragment loads free of conflicts
  static constexpr int NT = QSIDE ? 2 : 1;
  static constexpr int FS = K <= 4 ? 4 : (K <= 12 ? 12 : 20);  // factor row stride: 4 or 12 mod 16, conflict-free
  static constexpr int OCC = ctas_per_sm(K);
  static constexpr size_t SMEM = sizeof(double) * (CJ * FS + NT * CJ * CS);
};

// x * w for a genotype weight w = 0, 1 or 2, by the exponent (the float64 pipe is the bound)
__device__ __forceinline__ double times_weight(double x, bool zero, bool two) {
  const int hi = __double2hiint(x) + (two ? 0x00100000 : 0);
  return zero ? 0.0 : __hiloint2double(hi, __double2loint(x));
}

template <bool QSIDE, int K>
__global__ void __launch_bounds__(32 * MWARPS, Shape<QSIDE, K>::OCC) grad_hess_mma_kernel(Args a) {
  using S = Shape<QSIDE, K>;
  constexpr int KS = S::KS, NTG = S::NTG, NP = S::NP, NT = S::NT, CS = S::CS, FS = S::FS, TPC = S::TPC, COLS = S::COLS;
  extern __shared__ __align__(16) uint8_t smem[];
  double* fac = reinterpret_cast<double*>(smem);    // [CJ][FS] factor rows of the chunk, by column of the h tiles
  double* pp = fac + CJ * FS;                       // [NT][CJ / 2][CS][2] products of two reduced entries
  __shared__ uint8_t pk[TPC], pl[TPC];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int64_t n_rows = QSIDE ? a.N : a.M;
  const int64_t n_red = QSIDE ? a.M : a.N;
  const int64_t prows = (a.M + 3) >> 2;
  const double* ownF = QSIDE ? a.Q : a.P;
  const double* redF = QSIDE ? a.P : a.Q;

  int64_t b = blockIdx.x;
  const int pblk = S::NPB == 1 ? 0 : (int)(b % S::NPB);
  b /= S::NPB;
  const int split = (int)(b % a.n_split);
  const int64_t row0 = b / a.n_split * TR + warp * RW;   // the warp's first row

  for (int c = tid; c < TPC; c += 32 * MWARPS) {   // pairs in row-major order of the upper triangle
    int p = pblk * TPC + c, k = 0;
    const bool in = p < S::PAIRS;
    while (in && p >= K - k) { p -= K - k; ++k; }
    pk[c] = in ? (uint8_t)k : 0xFF;
    pl[c] = in ? (uint8_t)(k + p) : 0xFF;
  }
  for (int e = tid; e < CJ * FS; e += 32 * MWARPS) fac[e] = 0.0;

  double own[KS][2];   // h's A operand: rows g, g + 8, columns 4 ks + t
#pragma unroll
  for (int ks = 0; ks < KS; ++ks)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int64_t row = row0 + g + 8 * r;
      const int k = 4 * ks + t;
      own[ks][r] = row < n_rows && k < K ? ownF[row * K + k] : 0.0;
    }

  // The 2-bit codes of the thread's 8 reduced entries of rows g and g + 8 of a chunk: two packed
  // bytes on the Q side, 8 bytes on the P side. Loaded a chunk ahead, put together at use; rows
  // and entries outside the matrix are 3 (missing) or are masked by the caller.
  struct Codes {
    Words8 p[QSIDE ? 1 : 2];
    uint32_t q[2][2];
  };
  auto load_codes = [&](int64_t red0, Codes& c) {
    const int64_t first = red0 + 8 * t;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int64_t row = row0 + g + 8 * r;
      if constexpr (QSIDE) {
        const int64_t pr = first >> 2;   // first is a multiple of 8
        c.q[r][0] = row < a.N && pr < prows ? (uint32_t)__ldg(a.G + pr * a.N + row) : 0xFFu;
        c.q[r][1] = row < a.N && pr + 1 < prows ? (uint32_t)__ldg(a.G + (pr + 1) * a.N + row) : 0xFFu;
      } else {
        c.p[r] = row < a.M && first < n_red ? fetch8(a.G, prows * a.N, (row >> 2) * a.N + first) : Words8{~0u, ~0u, ~0u, 0u};
      }
    }
  };
  auto codes_of = [&](const Codes& c, uint64_t (&w)[2]) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if constexpr (QSIDE) w[r] = c.q[r][0] | (c.q[r][1] << 8);
      else w[r] = c.p[r].bytes() >> (2 * (uint32_t)((row0 + g + 8 * r) & 3));
    }
  };
  auto code_of = [&](uint64_t w, int idx) -> uint32_t {
    return (uint32_t)(w >> ((QSIDE ? 2 : 8) * idx)) & 3u;
  };

  double acc[NP][4], gacc[NTG][4];
#pragma unroll
  for (int n = 0; n < NP; ++n)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[n][v] = 0.0;
#pragma unroll
  for (int n = 0; n < NTG; ++n)
#pragma unroll
    for (int v = 0; v < 4; ++v) gacc[n][v] = 0.0;

  const int64_t n_chunks = (n_red + CJ - 1) / CJ;
  const int64_t ch0 = (int64_t)split * a.chunks_per_split;
  const int64_t ch1 = min(n_chunks, ch0 + a.chunks_per_split);
  // a chunk's genotypes and, where registers are left, its factor rows (contiguous; zeros past the
  // axis) are loaded a chunk ahead of their use. With 6 or 7 column tiles (K = 9, 10, 13, 14) at 3
  // CTAs per SM they spill: 7.6 ms on the P side at N=20,000 x M=50,000, K=10 where loading them at
  // use takes 7.2
  constexpr bool AHEAD = NP <= 5 || NP >= 8;
  constexpr int FPT = (CJ * K + 32 * MWARPS - 1) / (32 * MWARPS);
  Codes next;
  double fnext[FPT];
  auto load_factors = [&](int64_t red0) {
#pragma unroll
    for (int q = 0; q < FPT; ++q) {
      const int e = tid + q * 32 * MWARPS;
      fnext[q] = e < CJ * K && red0 * K + e < n_red * K ? redF[red0 * K + e] : 0.0;
    }
  };
  load_codes(ch0 * CJ, next);
  if (AHEAD) load_factors(ch0 * CJ);
  for (int64_t ch = ch0; ch < ch1; ++ch) {
    const int64_t red0 = ch * CJ;
    uint64_t w[2];
    codes_of(next, w);
    if (!AHEAD) load_factors(red0);
    __syncthreads();   // the previous chunk's readers are done
#pragma unroll
    for (int q = 0; q < FPT; ++q) {
      const int e = tid + q * 32 * MWARPS;
      const int r = e / K, k = e - r * K;
      // reduced entry 8 t + 2 nt + e is column 2 t + e of tile nt: row 8 nt + 2 t + e
      if (e < CJ * K) fac[(((r >> 1) & 3) * 8 + (r >> 3) * 2 + (r & 1)) * FS + k] = fnext[q];
    }
    if (ch + 1 < ch1) {
      load_codes(red0 + CJ, next);
      if (AHEAD) load_factors(red0 + CJ);
    }
    __syncthreads();
    for (int e = tid; e < (CJ / 2) * COLS; e += 32 * MWARPS) {
      const int u = e / COLS, c = e - u * COLS;
      const double* f0 = fac + (2 * u) * FS;
      const double* f1 = f0 + FS;
      double2 v0 = make_double2(0.0, 0.0), v1 = v0;
      if (c < TPC) {
        const int k = pk[c], l = pl[c];
        if (k != 0xFF) {
          const double x0 = f0[k], y0 = f0[l], x1 = f1[k], y1 = f1[l];
          v0 = make_double2(x0 * y0, x1 * y1);
          if (QSIDE) v1 = make_double2((1.0 - x0) * (1.0 - y0), (1.0 - x1) * (1.0 - y1));
        }
      } else if (c - TPC < K) {
        v0 = make_double2(f0[c - TPC], f1[c - TPC]);
        if (QSIDE) v1 = make_double2(1.0 - v0.x, 1.0 - v0.y);
      }
      reinterpret_cast<double2*>(pp)[u * CS + c] = v0;
      if (QSIDE) reinterpret_cast<double2*>(pp)[(CJ / 2) * CS + u * CS + c] = v1;
    }
    __syncthreads();
    if (red0 + CJ > n_red) {   // the last chunk: entries past the axis are missing
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (red0 + 8 * t + i >= n_red) w[r] |= 3ull << ((QSIDE ? 2 : 8) * i);
    }
#pragma unroll
    for (int nt = 0; nt < CJ / 8; ++nt) {
      double h[4] = {0.0, 0.0, 0.0, 0.0};
      const double* fb = fac + (nt * 8 + g) * FS + t;
#pragma unroll
      for (int ks = 0; ks + 1 < KS; ks += 2)
        mma_f64_k8(h, own[ks][0], own[ks][1], own[ks + 1][0], own[ks + 1][1], fb[4 * ks], fb[4 * ks + 4]);
      if constexpr (KS & 1) mma_f64(h, own[KS - 1][0], own[KS - 1][1], fb[4 * (KS - 1)]);
      double c1[4], c2[4], z1[4], z2[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t code = code_of(w[e >> 1], 2 * nt + (e & 1));
        // clamp to [1e-10, 1 - 1e-10] by the bit patterns (they order as the values do; a NaN
        // goes to the upper bound, as with fmin)
        const long long lo = __double_as_longlong(1e-10), hi = __double_as_longlong(1.0 - 1e-10);
        long long hb = __double_as_longlong(h[e]);
        hb = hb > hi ? hi : hb;
        hb = hb < lo ? lo : hb;
        const double hh = __longlong_as_double(hb), om = 1.0 - hh;
        // 1/h and 1/(1-h) from one reciprocal of x = h(1-h) in [1e-10, 0.25]: the hardware
        // approximation refined by two Newton-Raphson steps r <- r (2 - x r), each of which
        // squares the relative error (within a unit or two of the last place after both)
        const double x = hh * om;
        double r;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
        r = fma(r, fma(-x, r, 1.0), r);
        r = fma(r, fma(-x, r, 1.0), r);
        const double ih = om * r, iom = hh * r;
        z1[e] = times_weight(ih, code == 0u || code == 3u, code == 2u);
        z2[e] = times_weight(iom, code >= 2u, code == 0u);
        c1[e] = z1[e] * ih;
        c2[e] = z2[e] * iom;
        if (!QSIDE) {
          c1[e] += c2[e];
          z1[e] -= z2[e];
        }
      }
      const double2* pb = reinterpret_cast<const double2*>(pp) + (nt * 4 + t) * CS + g;
#pragma unroll
      for (int n = 0; n < NP; ++n) {
        const double2 f = pb[8 * n];
        mma_f64_k8(acc[n], c1[0], c1[2], c1[1], c1[3], f.x, f.y);
        if constexpr (QSIDE) {
          const double2 f2 = pb[(CJ / 2) * CS + 8 * n];
          mma_f64_k8(acc[n], c2[0], c2[2], c2[1], c2[3], f2.x, f2.y);
        }
      }
      if (pblk == 0) {
#pragma unroll
        for (int n = 0; n < NTG; ++n) {
          const double2 f = pb[TPC + 8 * n];
          mma_f64_k8(gacc[n], z1[0], z1[2], z1[1], z1[3], f.x, f.y);
          if constexpr (QSIDE) {
            const double2 f2 = pb[(CJ / 2) * CS + TPC + 8 * n];
            mma_f64_k8(gacc[n], z2[0], z2[2], z2[1], z2[3], f2.x, f2.y);
          }
        }
      }
    }
  }

  // both halves of the symmetric Hessian; accumulator v of a tile is row g (+8 for v >= 2),
  // column 2 t + (v & 1)
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const int64_t row = row0 + g + (v >> 1) * 8;
    if (row >= n_rows) continue;
    double* H = a.XtX + row * K * K;
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      const int c = 8 * n + 2 * t + (v & 1);
      const int k = pk[c], l = pl[c];
      if (k == 0xFF) continue;
      atomicAdd(H + k * K + l, acc[n][v]);
      if (l != k) atomicAdd(H + l * K + k, acc[n][v]);
    }
    if (pblk == 0) {
#pragma unroll
      for (int n = 0; n < NTG; ++n) {
        const int k = 8 * n + 2 * t + (v & 1);
        if (k < K) atomicAdd(a.Xtz + row * K + k, gacc[n][v]);
      }
    }
  }
}

}  // namespace gh
}  // namespace adx

using namespace adx;


template <bool QSIDE, int K>
static int grad_hess_mma_launch(const gh::Args& a, int64_t blocks, cudaStream_t st) {
  using S = gh::Shape<QSIDE, K>;
  ADX_CUDA_TRY(cudaFuncSetAttribute(gh::grad_hess_mma_kernel<QSIDE, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));
  ADX_CUDA_TRY(cudaFuncSetAttribute(gh::grad_hess_mma_kernel<QSIDE, K>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                    cudaSharedmemCarveoutMaxShared));
  gh::grad_hess_mma_kernel<QSIDE, K><<<(unsigned)blocks, 32 * gh::MWARPS, S::SMEM, st>>>(a);
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

template <bool QSIDE>
static int grad_hess(const uint8_t* G, int64_t M, int64_t N, int K, const double* P, const double* Q,
                     double* XtX, double* Xtz, void* stream, const char* name) {
  if (!G || !P || !Q || !XtX || !Xtz || M <= 0 || N <= 0 || K < 1 || K > ADX_MAX_K) {
    adx_set_message(name);
    return ADX_ERR_ARG;
  }
  cudaStream_t st = as_stream(stream);
  const int64_t n_rows = QSIDE ? N : M, n_red = QSIDE ? M : N;
  ADX_CUDA_TRY(cudaMemsetAsync(XtX, 0, (size_t)n_rows * K * K * sizeof(double), st));
  ADX_CUDA_TRY(cudaMemsetAsync(Xtz, 0, (size_t)n_rows * K * sizeof(double), st));
  gh::Args a{G, P, Q, M, N, K, XtX, Xtz, 0, 0, 0};
  const int n_pairs = K * (K + 1) / 2;
  const bool mma = K <= 16;
  a.n_pblk = mma ? gh::pair_blocks(K) : (n_pairs + gh::TP - 1) / gh::TP;
  const int64_t tiles = ceil_div(n_rows, gh::TR);
  const int64_t n_chunks = ceil_div(n_red, gh::CJ);
  int64_t split;
  if (mma) {
    // splits of the reduced axis: of the counts that just fill 1 to 12 rounds of resident CTAs,
    // the one whose rounds finish first, counting chunks and about 3 chunks of prologue and
    // atomics per CTA (at M=50,000 SNPs, K=10 on the P side: 5 splits, 8.8 rounds, 7.2 ms; 3
    // splits, 5.3 rounds, 7.7 ms)
    const int64_t slots = (int64_t)sm_count() * gh::ctas_per_sm(K);
    int64_t best = -1;
    split = 1;
    for (int64_t round = 1; round <= 12; ++round) {
      int64_t s = round * slots / (tiles * a.n_pblk);
      s = s < 1 ? 1 : (s > n_chunks ? n_chunks : s);
      const int64_t per = ceil_div(n_chunks, s);
      const int64_t time = ceil_div(tiles * a.n_pblk * ceil_div(n_chunks, per), slots) * (per + 3);
      if (best < 0 || time < best) { best = time; split = s; }
    }
  } else {
    // about 8 CTAs per SM in all
    split = ceil_div((int64_t)sm_count() * 8, tiles * a.n_pblk);
    split = split < 1 ? 1 : (split > n_chunks ? n_chunks : split);
  }
  a.chunks_per_split = ceil_div(n_chunks, split);
  a.n_split = (int)ceil_div(n_chunks, a.chunks_per_split);
  const int64_t blocks = tiles * a.n_pblk * a.n_split;
#define ADX_GH(KK) case KK: return grad_hess_mma_launch<QSIDE, KK>(a, blocks, st);
  switch (K) {
    ADX_GH(1) ADX_GH(2) ADX_GH(3) ADX_GH(4) ADX_GH(5) ADX_GH(6) ADX_GH(7) ADX_GH(8)
    ADX_GH(9) ADX_GH(10) ADX_GH(11) ADX_GH(12) ADX_GH(13) ADX_GH(14) ADX_GH(15) ADX_GH(16)
    default: break;
  }
#undef ADX_GH
  const size_t smem = gh::Smem::bytes(K, QSIDE ? 2 : 1);
  ADX_CUDA_TRY(cudaFuncSetAttribute(gh::grad_hess_kernel<QSIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  gh::grad_hess_kernel<QSIDE><<<(unsigned)blocks, gh::TPB, smem, st>>>(a);
  ADX_LAUNCH_CHECK();
  return ADX_OK;
}

extern "C" int adx_grad_hess_q(const uint8_t* G, int64_t M, int64_t N, int K, const double* P, const double* Q,
                               double* XtX_q, double* Xtz_q, void* stream) {
  return grad_hess<true>(G, M, N, K, P, Q, XtX_q, Xtz_q, stream, "adx_grad_hess_q: bad argument");
}

extern "C" int adx_grad_hess_p(const uint8_t* G, int64_t M, int64_t N, int K, const double* P, const double* Q,
                               double* XtX_p, double* Xtz_p, void* stream) {
  return grad_hess<false>(G, M, N, K, P, Q, XtX_p, Xtz_p, stream, "adx_grad_hess_p: bad argument");
}
