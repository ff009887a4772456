// Products of the centred genotype matrix with skinny float32 factors on the integer tensor
// cores (tcgen05.mma kind::i8, 32-bit accumulators in tensor memory), for the shifted
// randomized SVD (adamixture/model/svd_gpu.py:40-154):
//
//   rows:  Y[j] = sum_i x_ji B_i                    (x = g - 2 f_j, 0 where missing)
//   cols:  Z[i] = sum_j x_ji Y_j
//
// A genotype code c is 0..3 (3: missing). With m = 1 where missing, g = c - 3m and the
// centred entry is (c - 3m) - 2f (1 - m), so
//   rows:  Y_j = (S1 - 3 S2) - 2 f_j (sum_i B_i - S2),   S1 = sum_i c B_i, S2 = sum_i m B_i
//   cols:  Z_i = sum_j c y_j + sum_j m (2 f_j - 3) y_j - sum_j 2 f_j y_j
// and every sum over the matrix is one of small integers (c, m) times a factor column. The
// factor is taken to 31-bit fixed point relative to its column's largest magnitude and split
// into four signed 8-bit digits (columns 4 x L of the B operand); products and sums are
// exact in int32 (at most 3 x 128 x 0.5 Mi per digit and CTA), the CTAs' parts add exactly in
// int64, and one rounding to float32 ends it. What is left is the quantization: per entry at
// most 2^-30 of the column's largest magnitude, 64 times finer than float32's own rounding
// there (cols: the same of the codes' and of the flags' factor, the latter up to 3 times as
// large). Against float64 the relative error is 2.5e-8 (the final rounding) where float32 FMAs
// gave 5.6e-6 (N=100,000 x M=300,000).
//
// That error is the same for every entry of a column, so an output that meets small entries
// only can be less exact than float32 FMAs make it. Per output both errors are sums: of n_S met
// entries with the root mean square s they are about 2^-31 top sqrt(n_S) here and 2^-26 s n_S for
// FMAs, so this form is the finer one from s = 2^-5 top / sqrt(n_S) on. A column is called wide
// when more than 1/16 of its entries are inexact and below 2^-k of its largest magnitude, k = 4 +
// log2(n) / 2 at most 8 (a Gaussian column has 2 % there, one carried by a few samples nearly
// all). Wide columns take a second level, the same product with the remainders in 31 further
// bits, which keeps all bits of entries down to 2^-37 of the largest: a CTA walks its range
// twice when a column of its pass is wide. Columns that are wide once more (beyond 2^-31) and
// SNPs whose frequency is not finite (rows) are summed entry by entry in float32, in turn
// (finalize kernels). Infinite and NaN entries of the factor, and of f (cols), have no digits:
// their terms are added in float32 at the end.
//
// CTA: 256 rows of the product (two 128-row MMA tiles) over a range of 256-entry blocks of
// the contracted axis. Rows are SNPs and the contraction runs over samples, or the reverse:
// either way a block is 64 packed rows x 256 samples of G. Two groups of 8 warps unpack, taking turns:
// thread = row of the product; 64 entries at a time it forms the codes and the missing flags, 4 per 32-bit
// register, and stores them to tensor memory, which feeds the MMAs' A operand: no unpacked
// entry goes through shared memory. rows: a register is 4 samples of the SNP (one shift and
// mask of the packed word); cols: the 4 SNPs of the sample's packed byte, spread to bytes.
// One warp copies G (16-byte cp.async at any alignment, see row offsets) and the digit tiles
// (bulk copies) into a 3-slot ring; another issues the MMAs. Tensor memory: accumulators
// (2 tiles x {c, m} x 4 Lb columns), then a ring of 2 to 4 A stages of 64 columns. Lb, the factor
// columns of a pass, is at most 24 so that two A stages fit; a wider factor takes
// ceil(L / 24) passes of equal width.
//
// One pass each way at N=100,000 x M=300,000, L=20: 120.3 ms on float32 CUDA cores, 11.6 ms
// here (the packed matrix read twice is 2.3 ms of HBM time). Wide columns: N = M = 100,000, a
// product 2.0 -> 3.9 ms (21 and 35 on the CUDA cores).
// What bounds it now is the hand-over of the A stages: with no MMAs issued the loop still takes
// 60 % of the time, and each MMA adds the 50 cycles that it takes; the time does not depend on
// L (16 to 24), nor on the loads, nor on the unpacking itself.
#include "tcgen05.cuh"

#include <math.h>

#include <algorithm>

namespace adx {
namespace rt {

using tc::cp_async16;
using tc::cp_async_arrive;
using tc::fence_after;
using tc::fence_before;
using tc::mbar_arrive;
using tc::mma_commit;
using tc::smem_u32;

constexpr int TILE = 128;                 // rows of an MMA tile
constexpr int OWN = 2 * TILE;             // rows of the product per CTA
constexpr int BLK = 256;                  // contracted entries per block
constexpr int KST = 64;                   // contracted entries per A stage
constexpr int KSTEPS = BLK / KST;
constexpr int NDIG = 4;                   // 8-bit digits per factor entry
constexpr int LB_MAX = 24;                // factor columns per pass
constexpr int L_MAX = 80;
constexpr int NSLOT = 3;                  // G / digit slots
constexpr int NSTAGE_MIN = 2, NSTAGE_MAX = 4;   // A stages
constexpr int GROUPS = 2;                 // unpack groups, taking turns at the A stages
constexpr int GROUP_WARPS = 8;            // a thread per row of the product
constexpr int UNPACK_WARPS = GROUPS * GROUP_WARPS;
static_assert(GROUPS <= KSTEPS, "every group works on every block");
// A group waits for the MMAs of the stage's previous fill by that fill's parity, so it must
// not come to a fill while the one before the previous is still to be read: its own last wait
// (GROUPS stages ago, for MMAs nstage earlier still) proves that only if GROUPS <= nstage.
static_assert(GROUPS <= NSTAGE_MIN, "a stage's fills cannot be confused by their parity");
constexpr int LOAD_WARP = UNPACK_WARPS, MMA_WARP = UNPACK_WARPS + 1;
constexpr int TPB = 32 * (UNPACK_WARPS + 2);
constexpr int G_ROW = BLK + 16;           // bytes of a packed row in a slot, any alignment
constexpr int G_BYTES = (OWN / 4) * G_ROW;
constexpr int N_BARS = 2 * NSLOT + NSTAGE_MAX + 1;
constexpr uint32_t POLLS = 1u << 22;      // of a bounded wait: a fraction of a second to a few seconds
// A launch takes at most so many row tiles and contracted blocks, so that the workspace stays
// bounded (32 bytes an output, at most 16 L a contracted entry): 606,208 rows, 16 full rounds of
// CTAs, and 524,288 contracted entries. At L=20 that is 0.39 GB at most; one launch for all
// would take 6.4 GB for 10 million SNPs.
constexpr int64_t MAX_TILES = 148 * 16, MAX_BLOCKS = 2048;
static_assert(MAX_TILES * OWN * L_MAX < (1ll << 32), "32-bit output indices");
static_assert(OWN == BLK, "a block of G has the same shape in both products");
static_assert(3ll * 128 * MAX_BLOCKS * BLK < (1ll << 31), "int32 digit sums");
static_assert(2 * 2 * NDIG * LB_MAX + NSTAGE_MIN * 64 <= 512, "accumulators and the A stages in tensor memory");
static_assert(G_ROW % 16 == 0 && G_BYTES % 16 == 0, "16-byte copies");

struct Head;

struct Args {
  const uint8_t* G;
  int64_t M, N;
  const uint8_t* dc;       // digit tiles of the codes' factor: [pass][block][256 x 4 Lb bytes]
  const uint8_t* dm;       // of the flags' factor (rows: the same tiles)
  size_t level_bytes;      // from the first level's digits (dc, dm) to the second's
  int64_t level_sums;      // and of the sums (sc, sm)
  int L, Lb, n_pass;
  int64_t blk0, n_blk;     // contracted blocks
  int64_t tile0, tiles;    // row tiles of 256
  int n_split;             // ranges of the contracted axis
  int nstage;
  bool add;                // to the sums (several ranges or launches), else they are written
  long long* sc;           // [rows of the tiles][L] code sums (rows: S1 - 3 S2)
  long long* sm;           // [rows of the tiles][L] flag sums
  const Head* head;
  int* err;                // status of this product
  int* sticky;             // and of the workspace, until it is read
  uint32_t polls;          // limit of a wait
};

__host__ __device__ inline int digit_bytes(int Lb) { return BLK * NDIG * Lb; }

// Instruction descriptor, kind::i8: D int32, A and B signed 8-bit, both K-major, M = 128.
__device__ __forceinline__ uint32_t idesc_i8(int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
}

// D (tensor memory) += A (tensor memory) . B (shared memory), M=128, K=32.
__device__ __forceinline__ void mma_i8(uint32_t d, uint32_t a, uint64_t bd, uint32_t id, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}\n"
      :
      : "r"(d), "r"(a), "l"(bd), "r"(id), "r"(accumulate));
}

__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      :
      : "r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld4(uint32_t addr, uint32_t (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(addr));
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               :
               : "r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void arrive_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(bar),
               "r"(bytes)
               : "memory");
}

// Bounded wait of a whole warp. False once it has run out of polls, which raises the abort word,
// or another warp has given up.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, uint32_t polls) {
  for (uint32_t it = 0; it < polls; ++it) {
    if (tc::mbar_try(bar, parity)) return true;
    if ((it & 15u) == 0u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

// A stage's hand-over from the unpack group to the MMA warp: a named barrier, a generation per
// fill of the stage (1.95 ms a product at N = M = 100,000, L=20; an mbarrier here takes 2.25 to
// 2.35, whichever way its waiter polls). A named barrier has no limit of its own and counts
// arrivals without asking whose they are, so every generation must get exactly one arrival of each
// of its 9 warps and none before the previous generation of that stage is complete:
// - unpack and MMA warps never leave their loops early: after a wait that has run out they go on to
//   the end, where the results are discarded;
// - an unpack warp comes to a stage's next generation only when the MMA warp has passed the
//   one before: the AEMPTY wait proves it, and where that has been given up, `joined` (the
//   stages the MMA warp has passed) is waited for instead. That always ends: the warps whose
//   arrivals the MMA warp lacks are at its stage or before it, so what they wait for it has
//   already written.
constexpr int HANDOVER = 32 * (GROUP_WARPS + 1);
__device__ __forceinline__ void stage_arrive(int st) {
  asm volatile("bar.arrive %0, %1;" ::"r"(1 + st), "n"(HANDOVER) : "memory");
}
__device__ __forceinline__ void stage_sync(int st) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + st), "n"(HANDOVER) : "memory");
}
__device__ __forceinline__ void wait_joined(const volatile int* joined, int stages) {
  for (uint32_t it = 0; it < POLLS && *joined < stages; ++it) __nanosleep(200);
}

// 64 packed rows from row0 x 256 samples from i0 into a slot, by the load warp. AL: every
// packed row starts 16-byte aligned, 16 chunks a row; otherwise 17 chunks from the 16-byte
// boundary at or below the row's first byte (readers add row_offset). Chunks that would
// leave the matrix take byte loads (0 past the ends); rows past the matrix are not loaded.
// What is read for samples past N or SNPs past M does not matter: their digits are zero, or
// their product rows are not stored.
template <bool AL>
__device__ __forceinline__ void load_g(const Args& a, int64_t row0, int64_t i0, uint8_t* gs) {
  const int lane = threadIdx.x & 31;
  const int64_t rows = (a.M + 3) >> 2;
  const uint8_t* end = a.G + rows * a.N;
  auto chunk = [&](int r, int c) {
    const int64_t row = row0 + r;
    if (row >= rows) return;
    const uint8_t* src = a.G + row * a.N + i0;
    if constexpr (!AL) src -= reinterpret_cast<uintptr_t>(src) & 15;
    src += 16 * c;
    uint8_t* dst = gs + r * G_ROW + 16 * c;
    if (src >= a.G && src + 16 <= end) {
      cp_async16(smem_u32(dst), src);
    } else {
      for (int b = 0; b < 16; ++b) dst[b] = src + b >= a.G && src + b < end ? __ldg(src + b) : (uint8_t)0;
    }
  };
  const uint8_t* first = a.G + row0 * a.N + i0;
  // a block inside the matrix (and 16 bytes either way): one pointer walks the rows. The
  // general form's checks and 64-bit products, about 25 instructions a chunk in one warp, were
  // what the whole kernel waited for (3.4 ms a pass against 2.4 at N = M = 100,000)
  if (row0 + OWN / 4 <= rows && first - 16 >= a.G && first + (OWN / 4 - 1) * a.N + BLK + 16 <= end) {
    const uint8_t* src = first + (lane >> 4) * a.N + 16 * (lane & 15);
    uint32_t dst = smem_u32(gs) + (uint32_t)(lane >> 4) * G_ROW + 16u * (uint32_t)(lane & 15);
    const int64_t step = 2 * a.N;
#pragma unroll 8
    for (int r = 0; r < OWN / 4; r += 2, src += step, dst += 2 * G_ROW)
      cp_async16(dst, AL ? src : src - (reinterpret_cast<uintptr_t>(src) & 15));
    if constexpr (!AL) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint8_t* s16 = first + (lane + 32 * h) * a.N + BLK;
        cp_async16(smem_u32(gs) + (uint32_t)(lane + 32 * h) * G_ROW + BLK, s16 - (reinterpret_cast<uintptr_t>(s16) & 15));
      }
    }
    return;
  }
  for (int e = lane; e < (OWN / 4) * (BLK / 16); e += 32) chunk(e / (BLK / 16), e % (BLK / 16));
  if constexpr (!AL) {
    chunk(lane, BLK / 16);
    chunk(lane + 32, BLK / 16);
  }
}

// Offset (bytes) of a block's first sample in its packed row lr: blocks start at packed rows
// and samples that are multiples of 16, so it depends on lr mod 16 alone.
__device__ __forceinline__ uint32_t row_offset(const Args& a, int lr) {
  return ((uint32_t)(reinterpret_cast<uintptr_t>(a.G) & 15) + (uint32_t)lr * (uint32_t)(a.N & 15)) & 15u;
}

// The kernels of a product follow one another closely: each lets the next one's blocks come onto
// the chip as its own leave, and each begins by waiting until the one before is complete and its
// writes are visible (programmatic dependent launch). The first, top_kernel, is an ordinary launch.
// Rows and cols at N=300 x M=5,001, L=20 39 and 43 -> 31 and 33 us, N=1,003 x M=40,011, L=26 68
// and 64 -> 63 and 56, N=20,001 x M=50,003, L=24 290 and 310 -> 282 and 298.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... P, typename... A>
static cudaError_t launch_after(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// Head of the workspace: the quanta (0: a column of zeros), constant sums of the two levels,
// entries that the levels hold too coarsely, what follows from them, entries without digits,
// status. The first kernel of a product clears it.
constexpr int N_FACT = 3;       // factors: of the codes, of the flags, of the constant sum
constexpr int LEVELS = 2;
constexpr int WIDE = 1, DIRECT = 2, ODD = 4;   // takes the second level; summed directly; has entries without digits
constexpr int MAX_ODD = 64;     // entries added one by one; with more, their columns are summed directly
struct Head {
  double quantum[N_FACT][L_MAX];
  unsigned long long csum[LEVELS][L_MAX];
  unsigned long long coarse[LEVELS][L_MAX];
  int mode[L_MAX];                // of a column: bits
  int wide[L_MAX / LB_MAX + 1];   // a column of the pass is WIDE
  int n_odd;                      // entries without digits, the first MAX_ODD of them
  int64_t odd_row[MAX_ODD];
  int odd_col[MAX_ODD];
  int err;
};

template <bool ROWS, bool AL>
__global__ void __launch_bounds__(TPB, 1) product_kernel(Args a) {
  after_previous();
  extern __shared__ __align__(128) uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n4 = NDIG * a.Lb;
  const uint32_t dbytes = (uint32_t)digit_bytes(a.Lb);
  const uint32_t slot_bytes = G_BYTES + (ROWS ? 1u : 2u) * dbytes;
  uint8_t* ctl = sm + NSLOT * slot_bytes;
  const uint32_t bars = smem_u32(ctl);
  auto FULL = [&](int s) { return bars + 8u * (uint32_t)s; };
  auto EMPTY = [&](int s) { return bars + 8u * (uint32_t)(NSLOT + s); };
  auto AEMPTY = [&](int s) { return bars + 8u * (uint32_t)(2 * NSLOT + s); };
  const uint32_t DONE = bars + 8u * (uint32_t)(N_BARS - 1);
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(ctl + 8 * N_BARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(ctl + 8 * N_BARS + 4);
  volatile int* joined = reinterpret_cast<volatile int*>(ctl + 8 * N_BARS + 8);   // stages the MMA warp has passed

  int64_t b = blockIdx.x;
  const int64_t tile = a.tile0 + b % a.tiles; b /= a.tiles;
  const int split = (int)(b % a.n_split);
  const int pass = (int)(b / a.n_split);
  const int64_t per = (a.n_blk + a.n_split - 1) / a.n_split;
  const int64_t q0 = (int64_t)split * per;
  const int nq = (int)(min(a.n_blk, q0 + per) - q0);   // at least 1: the host's n_split is exact

  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_holder)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  const int levels = a.head->wide[pass] ? LEVELS : 1;
  for (int level = 0; level < levels; ++level) {
  if (tid == 0) {
    *abort_flag = 0;
    *joined = 0;
    if (level)   // the barriers of the first level, all complete
      for (int s = 0; s < N_BARS; ++s) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bars + 8u * (uint32_t)s) : "memory");
    for (int s = 0; s < NSLOT; ++s) {
      // 32 asynchronous and 32 plain arrivals of the load warp, and the bulk copies' expect
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 65;" ::"r"(FULL(s)));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(EMPTY(s)));
    }
    for (int s = 0; s < NSTAGE_MAX; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(AEMPTY(s)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(DONE));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_holder;
  const uint32_t col_a = tmem + 4u * (uint32_t)n4;      // A stages: per stage and tile 16 code, 16 flag columns

  int loaded = 0;   // blocks that the load warp has asked for
  if (warp == LOAD_WARP) {
    int slot = 0;
    uint32_t fill = 0;   // how often the ring has wrapped
    for (int q = 0; q < nq; ++q) {
      if (fill > 0 && !warp_wait(EMPTY(slot), (fill - 1) & 1u, abort_flag, a.polls)) break;
      uint8_t* gs = sm + slot * slot_bytes;
      const int64_t blk = a.blk0 + q0 + q;
      if (lane == 0) {
        arrive_expect(FULL(slot), (ROWS ? 1u : 2u) * dbytes);
        const int64_t at = ((int64_t)pass * a.n_blk + q0 + q) * dbytes + level * a.level_bytes;
        bulk_copy(smem_u32(gs + G_BYTES), a.dc + at, dbytes, FULL(slot));
        if constexpr (!ROWS) bulk_copy(smem_u32(gs + G_BYTES + dbytes), a.dm + at, dbytes, FULL(slot));
      }
      load_g<AL>(a, (ROWS ? tile * OWN : blk * BLK) >> 2, ROWS ? blk * BLK : tile * OWN, gs);
      cp_async_arrive(FULL(slot));
      mbar_arrive(FULL(slot));
      ++loaded;
      if (++slot == NSLOT) { slot = 0; ++fill; }
    }
  } else if (warp == MMA_WARP) {
    const uint32_t id = idesc_i8(n4);
    int slot = 0, st = 0;
    uint32_t fill = 0;
    for (int q = 0; q < nq; ++q) {
      warp_wait(FULL(slot), fill & 1u, abort_flag, a.polls);
      const uint32_t sb = smem_u32(sm + slot * slot_bytes + G_BYTES);
      const uint64_t dc = tc::sdesc(sb, 128, 256), dm = ROWS ? dc : tc::sdesc(sb + dbytes, 128, 256);
      const uint64_t step = (uint64_t)(32 * n4) >> 4;   // one 32-entry step of a digit tile
      for (int ks = 0; ks < KSTEPS; ++ks) {
        stage_sync(st);
        fence_after();
        if (lane == 0) {
          const uint32_t as = col_a + 64u * (uint32_t)st;
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {
            const uint64_t off = step * (uint64_t)(2 * ks + kk);
            const uint32_t acc = (q > 0 || ks > 0 || kk > 0) ? 1u : 0u;
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              mma_i8(tmem + (uint32_t)(2 * t * n4), as + 32u * t + 8u * kk, dc + off, id, acc);
              mma_i8(tmem + (uint32_t)((2 * t + 1) * n4), as + 32u * t + 16u + 8u * kk, dm + off, id, acc);
            }
          }
          mma_commit(AEMPTY(st));
          if (ks == KSTEPS - 1) mma_commit(EMPTY(slot));
          *joined = q * KSTEPS + ks + 1;
        }
        __syncwarp();
        if (++st == a.nstage) st = 0;
      }
      if (++slot == NSLOT) { slot = 0; ++fill; }
    }
    if (lane == 0) mma_commit(DONE);   // also after a wait that ran out: covers the MMAs issued
    __syncwarp();
  } else {
    const int wq = warp & 3, t = (warp >> 2) & 1, grp = warp / GROUP_WARPS;
    const int own = t * TILE + wq * 32 + lane;        // row of the product within the CTA
    const uint32_t lanes = (uint32_t)(wq * 32) << 16;
    uint32_t goff[ROWS ? 1 : 16];                     // byte offsets into a slot
    uint32_t sh = 0;
    if constexpr (ROWS) {
      const uint32_t o = AL ? 0u : row_offset(a, own >> 2);
      goff[0] = (uint32_t)(own >> 2) * G_ROW + (o & ~3u);
      sh = 2u * (uint32_t)(own & 3) + 8u * (o & 3u);
    } else {
#pragma unroll
      for (int p = 0; p < 16; ++p) goff[p] = (uint32_t)p * G_ROW + (AL ? 0u : row_offset(a, p)) + (uint32_t)own;
    }
    int slot = 0, st = 0, turn = 0;
    uint32_t fill = 0, sfill = 0;
    for (int q = 0; q < nq; ++q) {
      warp_wait(FULL(slot), fill & 1u, abort_flag, a.polls);
      const uint8_t* gs = sm + slot * slot_bytes;
      for (int ks = 0; ks < KSTEPS; ++ks) {
        const bool mine = turn == grp;
        if (++turn == GROUPS) turn = 0;
        const int my_st = st;
        const uint32_t my_fill = sfill;
        if (++st == a.nstage) { st = 0; ++sfill; }
        if (!mine) continue;
        uint32_t x[16], m[16];
        if constexpr (ROWS) {
          const uint8_t* src = gs + goff[0] + KST * ks;
          if constexpr (AL) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const uint4 v = *reinterpret_cast<const uint4*>(src + 16 * c);
              x[4 * c] = v.x >> sh; x[4 * c + 1] = v.y >> sh; x[4 * c + 2] = v.z >> sh; x[4 * c + 3] = v.w >> sh;
            }
          } else {
            uint32_t w = *reinterpret_cast<const uint32_t*>(src);
#pragma unroll
            for (int c = 0; c < 16; ++c) {
              const uint32_t nx = *reinterpret_cast<const uint32_t*>(src + 4 * c + 4);
              x[c] = __funnelshift_r(w, nx, sh);
              w = nx;
            }
          }
        } else {
#pragma unroll
          for (int p = 0; p < 16; ++p) {
            // the byte's fields to the low bits of four bytes
            const uint32_t v = (uint32_t)gs[goff[p] + (uint32_t)(16 * ks * G_ROW)] * 0x1001u;
            x[p] = v | (v << 6);
          }
        }
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          x[c] &= 0x03030303u;
          m[c] = x[c] & (x[c] >> 1) & 0x01010101u;
        }
        if (my_fill > 0) {
          if (!warp_wait(AEMPTY(my_st), (my_fill - 1) & 1u, abort_flag, a.polls))
            wait_joined(joined, q * KSTEPS + ks - a.nstage + 1);
        }
        fence_after();
        const uint32_t as = col_a + lanes + 64u * (uint32_t)my_st + 32u * (uint32_t)t;
        tmem_st16(as, x);
        tmem_st16(as + 16, m);
        tmem_wait_st();
        fence_before();
        stage_arrive(my_st);
      }
      if (++slot == NSLOT) { slot = 0; ++fill; }
    }
  }
  warp_wait(DONE, 0u, abort_flag, a.polls);
  const bool gave_up = __syncthreads_or(*abort_flag);
  if (gave_up) {
    // a wait ran out: before the block ends, the copies and MMAs in flight land (these waits are
    // bounded too)
    if (tid == 0) {
      atomicExch(a.err, ADX_ERR_TIMEOUT);
      atomicExch(a.sticky, ADX_ERR_TIMEOUT);
    }
    volatile int never = 0;
    if (warp == LOAD_WARP) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      for (int s = 0; s < NSLOT; ++s) {
        const int fills = (loaded - s + NSLOT - 1) / NSLOT;
        if (fills > 0) warp_wait(FULL(s), (uint32_t)(fills - 1) & 1u, &never, POLLS);
      }
    } else if (warp == MMA_WARP) {
      warp_wait(DONE, 0u, &never, POLLS);
    }
  } else {
    fence_after();
    if (warp < GROUP_WARPS) {
      const int wq = warp & 3, t = warp >> 2;
      const int64_t row = tile * OWN + t * TILE + wq * 32 + lane;
      const int64_t n_rows = ROWS ? a.M : a.N;
      const uint32_t at = tmem + ((uint32_t)(wq * 32) << 16) + (uint32_t)(2 * t * n4);
      for (int l = 0; l < a.Lb; l += 4) {
        uint32_t v[2][NDIG][4];
#pragma unroll
        for (int o = 0; o < 2; ++o)
#pragma unroll
          for (int d = 0; d < NDIG; ++d) tmem_ld4(at + (uint32_t)(o * n4 + d * a.Lb + l), v[o][d]);
        tc::tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int lg = pass * a.Lb + l + e;
          long long s[2];
#pragma unroll
          for (int o = 0; o < 2; ++o) {
            s[o] = (int)v[o][NDIG - 1][e];
#pragma unroll
            for (int d = NDIG - 2; d >= 0; --d) s[o] = s[o] * 256 + (int)v[o][d][e];
          }
          if (ROWS) s[0] -= 3 * s[1];
          if (row < n_rows && lg < a.L && (!level || (a.head->mode[lg] & WIDE))) {
            const int64_t w = level * a.level_sums + (row - a.tile0 * OWN) * a.L + lg;
            if (!a.add) {
              a.sc[w] = s[0];
              a.sm[w] = s[1];
            } else {   // integers: the order does not matter
              atomicAdd(reinterpret_cast<unsigned long long*>(a.sc + w), (unsigned long long)s[0]);
              atomicAdd(reinterpret_cast<unsigned long long*>(a.sm + w), (unsigned long long)s[1]);
            }
          }
        }
      }
    }
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (gave_up) break;
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(*tmem_holder));
  }
}

// ---------------------------------------------------------------- factors to digits

// The factors of a product, from F [n][L]: codes take F; flags take F (rows) or (2f - 3) F
// (cols, f per entry); the constant sum takes F (rows) or 2 f F (cols).
template <bool ROWS>
__device__ __forceinline__ double factor(int which, float y, float f) {
  if (ROWS || which == 0) return (double)y;
  const double u = 2.0 * (double)f * (double)y;
  return which == 1 ? u - 3.0 * (double)y : u;
}
// Their magnitudes as float bits, which order as the magnitudes do (float32 rounds them; the digits
// have room for that). An entry with one that is not finite has no digits.
template <bool ROWS>
__device__ __forceinline__ bool magnitudes(float y, float f, uint32_t (&t)[ROWS ? 1 : N_FACT]) {
  t[0] = __float_as_uint(y) & 0x7FFFFFFFu;
  if constexpr (!ROWS) {
    t[1] = __float_as_uint((2.0f * f - 3.0f) * y) & 0x7FFFFFFFu;
    t[2] = __float_as_uint(2.0f * f * y) & 0x7FFFFFFFu;
  }
  uint32_t top = t[0];
#pragma unroll
  for (int w = 1; w < (ROWS ? 1 : N_FACT); ++w) top = max(top, t[w]);
  return top < 0x7F800000u;
}
constexpr int BITS = 30;        // fixed point of the codes' and flags' factors
constexpr int SUM_BITS = 36;    // and of the cols product's constant sum
constexpr int LOW_BITS = 31;    // further bits of the second level

// Largest magnitudes of a block's entries per factor and column. The first block clears the head.
constexpr int TOP_BLOCKS = 296;
__host__ __device__ constexpr int top_stride(int w, int L) { return (w * L + 3) / 4 * 4; }   // 16-byte loads
template <bool ROWS>
__global__ void __launch_bounds__(256) top_kernel(const float* __restrict__ F, const float* __restrict__ f, int64_t n,
                                                  int L, Head* h, uint32_t* __restrict__ tops) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  constexpr int W = ROWS ? 1 : N_FACT;
  __shared__ uint32_t top[W][L_MAX];
  if (blockIdx.x == 0)
    for (int e = threadIdx.x; e < (int)(sizeof(Head) / 4); e += 256) reinterpret_cast<uint32_t*>(h)[e] = 0;
  for (int e = threadIdx.x; e < W * L_MAX; e += 256) top[e / L_MAX][e % L_MAX] = 0;
  __syncthreads();
  const int per = 256 / L, l = threadIdx.x % L, g = threadIdx.x / L;
  if (g < per) {
    uint32_t t[W] = {};
    constexpr int U = 8;   // entries in flight
    const int64_t step = (int64_t)gridDim.x * per;
    for (int64_t i0 = (int64_t)blockIdx.x * per + g; i0 < n; i0 += U * step) {
      float y[U], fi[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t i = i0 + u * step;
        y[u] = i < n ? F[i * L + l] : 0.0f;
        fi[u] = !ROWS && i < n ? f[i] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        uint32_t m[W];
        if (magnitudes<ROWS>(y[u], fi[u], m))
#pragma unroll
          for (int w = 0; w < W; ++w) t[w] = max(t[w], m[w]);
      }
    }
#pragma unroll
    for (int w = 0; w < W; ++w) atomicMax(&top[w][l], t[w]);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < top_stride(W, L); e += 256)
    tops[blockIdx.x * top_stride(W, L) + e] = e < W * L ? top[e / L][e % L] : 0u;
}

// Thread per (16 contracted entries, factor column): 16 bytes of each digit of a level, in the
// order of the shared-memory tile (32-entry steps of 4 Lb x 32 bytes: core matrices of 8
// columns x 16 entries), for n_blk blocks from blk0. Entries past n and columns past L are zero.
// LOW: the second level, whose launch does nothing when no column is wide. does: COUNT (constant
// sums, coarse and odd entries), WRITE (digits).
constexpr int COUNT = 1, WRITE = 2;
template <bool ROWS, bool LOW>
__global__ void __launch_bounds__(256, 3) digit_kernel(const float* __restrict__ F, const float* __restrict__ f,
                                                    int64_t n, int L, int Lb, int n_pass, int64_t blk0,
                                                    int64_t n_blk, int does, Head* h,
                                                    const uint32_t* __restrict__ tops, int n_tops,
                                                    uint8_t* __restrict__ dc, uint8_t* __restrict__ dm) {
  after_previous();
  constexpr int W = ROWS ? 1 : N_FACT;
  __shared__ unsigned long long csum[L_MAX];
  __shared__ uint32_t coarse[L_MAX];
  __shared__ __align__(16) uint32_t top[top_stride(W, L_MAX)];
  __shared__ double per_quantum[W][L_MAX];   // 0: the column has no digits
  if (LOW && !__syncthreads_or(threadIdx.x < n_pass && h->wide[threadIdx.x])) return;
  for (int e = threadIdx.x; e < L_MAX; e += 256) { csum[e] = 0; coarse[e] = 0; }
  if constexpr (!LOW) {
    const int quads = top_stride(W, L) / 4, groups = 256 / quads, part = threadIdx.x / quads;
    const int e = 4 * (threadIdx.x - part * quads);
    if (part == 0) *reinterpret_cast<uint4*>(top + e) = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    if (part < groups) {
      uint4 t = make_uint4(0u, 0u, 0u, 0u);
      constexpr int U = 8;   // loads in flight
      for (int b = part; b < n_tops; b += U * groups) {
        uint4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          v[u] = b + u * groups < n_tops ? *reinterpret_cast<const uint4*>(tops + (b + u * groups) * 4 * quads + e)
                                         : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int u = 0; u < U; ++u)
          t = make_uint4(max(t.x, v[u].x), max(t.y, v[u].y), max(t.z, v[u].z), max(t.w, v[u].w));
      }
      atomicMax(top + e, t.x);
      atomicMax(top + e + 1, t.y);
      atomicMax(top + e + 2, t.z);
      atomicMax(top + e + 3, t.w);
    }
  }
  __syncthreads();
  if (threadIdx.x < L) {
    const int l = threadIdx.x;
    const bool on = !LOW || (h->mode[l] & WIDE);
#pragma unroll
    for (int w = 0; w < W; ++w) {
      // a quantum is 2^-bits of a power of two above the largest magnitude
      double inv = 0.0;
      if constexpr (LOW) {
        if (on && h->quantum[w][l] > 0.0) inv = 1.0 / h->quantum[w][l];
      } else {
        const uint32_t t = top[w * L + l];
        if (t) inv = ldexp(1.0, (w == 2 ? SUM_BITS : BITS) - 1 - ilogbf(__uint_as_float(t)));
        if (blockIdx.x == 0) h->quantum[w][l] = inv > 0.0 ? 1.0 / inv : 0.0;
      }
      per_quantum[w][l] = inv;
    }
  }
  __syncthreads();
  // entries below `small` (the largest is at least 2^29) are below 2^-k of the largest
  const int k = 4 + min(4, (63 - __clzll(n)) / 2);
  const double low = (double)(1u << LOW_BITS), small = (double)(1 << (BITS - k)) / (LOW ? low : 1.0);
  const int cols = n_pass * Lb;
  const int64_t work = n_blk * (BLK / 16) * cols;
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < work; e += (int64_t)gridDim.x * 256) {
    const int64_t kg = work <= UINT32_MAX ? (uint32_t)e / (uint32_t)cols : e / cols;
    const int lg = (int)(e - kg * cols), pass = lg / Lb, lc = lg - pass * Lb;
    double inv[W] = {};
#pragma unroll
    for (int w = 0; w < W; ++w) inv[w] = lg < L ? per_quantum[w][lg] : 0.0;
    const bool on = lg < L && (!LOW || inv[0] > 0.0);
    long long c = 0;
    uint32_t n_coarse = 0, dig[2][NDIG][4] = {};
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int64_t i = blk0 * BLK + kg * 16 + u;
      const bool in = on && i < n;
      float y = in ? F[i * L + lg] : 0.0f, fi = !ROWS && in ? f[i] : 0.0f;
      uint32_t m[W];
      if (!magnitudes<ROWS>(y, fi, m)) {
        if (!LOW && (does & COUNT)) {
          atomicOr(&h->mode[lg], ODD);
          // counted until they are too many
          const int at = *(volatile int*)&h->n_odd <= MAX_ODD ? atomicAdd(&h->n_odd, 1) : MAX_ODD;
          if (at < MAX_ODD) { h->odd_row[at] = i; h->odd_col[at] = lg; }
        }
        y = fi = 0.0f;
      }
      bool lost = false;
#pragma unroll
      for (int w = 0; w < W; ++w) {
        const double x = factor<ROWS>(w, y, fi) * inv[w];
        const double r = LOW ? (x - rint(x)) * low : x;   // the difference is exact
        const double qr = rint(r);
        lost = lost || (qr != r && fabs(x) < small);
        if (ROWS || w == 2) c += (long long)qr;
        if (w < 2) {
          int q = (int)qr;
#pragma unroll
          for (int d = 0; d < NDIG; ++d) {
            const int lo = (int)(int8_t)(q & 0xFF);   // signed digit; the rest divides exactly
            dig[w][d][u >> 2] |= (uint32_t)(lo & 0xFF) << (8 * (u & 3));
            q = (q - lo) >> 8;
          }
        }
      }
      n_coarse += lost;
    }
    if (on) atomicAdd(&csum[lg], (unsigned long long)c);
    if (n_coarse) atomicAdd(&coarse[lg], n_coarse);
    if (!(does & WRITE)) continue;
    const int64_t base = ((int64_t)pass * n_blk * (BLK / 32) + (kg >> 1)) * (32 * NDIG * Lb);
#pragma unroll
    for (int d = 0; d < NDIG; ++d) {
      const int col = d * Lb + lc;
      const int64_t at = base + (col >> 3) * 256 + (kg & 1) * 128 + (col & 7) * 16;
      *reinterpret_cast<uint4*>(dc + at) = make_uint4(dig[0][d][0], dig[0][d][1], dig[0][d][2], dig[0][d][3]);
      if (!ROWS) *reinterpret_cast<uint4*>(dm + at) = make_uint4(dig[1][d][0], dig[1][d][1], dig[1][d][2], dig[1][d][3]);
    }
  }
  __syncthreads();
  if (!(does & COUNT)) return;
  for (int e = threadIdx.x; e < L; e += 256) {
    if (csum[e]) atomicAdd(&h->csum[LOW][e], csum[e]);
    // the block whose entries bring the count past n / 16 says so
    if (coarse[e] && 16 * (int64_t)(atomicAdd(&h->coarse[LOW][e], (unsigned long long)coarse[e]) + coarse[e]) > n) {
      atomicOr(&h->mode[e], LOW ? DIRECT : WIDE);
      if (!LOW) h->wide[e / Lb] = 1;
    }
  }
}

// v + the term of contracted entry r in output (row, l), in float32.
template <bool ROWS>
__device__ __forceinline__ float term(const uint8_t* __restrict__ G, int64_t N, const float* __restrict__ F,
                                      const float* __restrict__ f, int L, int64_t r, int64_t row, int l, float v) {
  const int64_t j = ROWS ? row : r, i = ROWS ? r : row;
  const unsigned g = genotype(__ldg(G + (j >> 2) * N + i), (int)(j & 3));
  const float x = g == 3u ? 0.0f : (float)g - 2.0f * __ldg(f + j);
  return fmaf(x, __ldg(F + r * L + l), v);
}

// Output (row, l) entry by entry; a NaN stays one.
template <bool ROWS>
__device__ __noinline__ float direct(const uint8_t* __restrict__ G, int64_t N, const float* __restrict__ F,
                                     const float* __restrict__ f, int L, int64_t n_red, int64_t row, int l) {
  float v = 0.0f;
  int64_t r = 0;
  for (; r + 8 <= n_red && v == v; r += 8)
#pragma unroll
    for (int u = 0; u < 8; ++u) v = term<ROWS>(G, N, F, f, L, r + u, row, l, v);
  for (; r < n_red && v == v; ++r) v = term<ROWS>(G, N, F, f, L, r, row, l, v);
  return v;
}

// v + the terms of the entries without digits.
template <bool ROWS>
__device__ __noinline__ float add_odd(const uint8_t* __restrict__ G, int64_t N, const float* __restrict__ F,
                                      const float* __restrict__ f, int L, const Head* __restrict__ h, int64_t row, int l,
                                      float v) {
  for (int k = 0; k < h->n_odd; ++k)
    if (h->odd_col[k] == l) v = term<ROWS>(G, N, F, f, L, h->odd_row[k], row, l, v);
  return v;
}

// One thread per output element of `rows` rows from row0: the integer sums to float32.
template <bool ROWS>
__global__ void __launch_bounds__(256) finalize_kernel(const uint8_t* __restrict__ G, int64_t M, int64_t N,
                                                       int64_t row0, int64_t rows,
                                                       const float* __restrict__ F, const float* __restrict__ f, int L,
                                                       const long long* __restrict__ sc,
                                                       const long long* __restrict__ sm, int64_t level_sums,
                                                       const Head* __restrict__ h, int accumulate,
                                                       float* __restrict__ out) {
  after_previous();
  const int64_t n_red = ROWS ? N : M;
  const uint32_t e = blockIdx.x * 256 + threadIdx.x;   // of at most MAX_TILES * OWN * L_MAX
  if (e >= rows * L) return;
  const int64_t row = row0 + e / (uint32_t)L;
  const int l = (int)(e % (uint32_t)L);
  const float fr = ROWS ? f[row] : 0.0f;
  const int mode = h->mode[l];
  float v;
  if (h->err) {
    v = __uint_as_float(0x7FFFFFFFu);   // a bounded wait ran out: not a result
  } else if ((mode & DIRECT) || ((mode & ODD) && h->n_odd > MAX_ODD) || (ROWS && !isfinite(fr))) {
    v = direct<ROWS>(G, N, F, f, L, n_red, row, l);
  } else {
    auto sum = [&](int u) {
      const int64_t at = u * level_sums + e;
      const long long cs = (long long)h->csum[u][l];
      return ROWS ? h->quantum[0][l] * ((double)sc[at] - 2.0 * (double)fr * (double)(cs - sm[at]))
                  : h->quantum[0][l] * (double)sc[at] + h->quantum[1][l] * (double)sm[at] - h->quantum[2][l] * (double)cs;
    };
    double t = sum(0);
    if (mode & WIDE) t += sum(1) * (1.0 / (double)(1u << LOW_BITS));
    v = (float)t;
    if (mode & ODD) v = add_odd<ROWS>(G, N, F, f, L, h, row, l, v);
  }
  float* o = out + row0 * L + e;
  *o = accumulate ? *o + v : v;
}

// ---------------------------------------------------------------- plan

constexpr size_t ALIGN = 256;   // of the workspace's parts (bulk copies read from it); any caller's pointer will do

struct Plan {
  int Lb, n_pass, nstage;
  int64_t n_blk, tiles;     // in all
  size_t head, tops, digits, sums, bytes;   // bytes of each part and in all
};

static Plan plan(int64_t n_rows, int64_t n_red, int L, bool rows) {
  Plan p{};
  p.n_pass = (L + LB_MAX - 1) / LB_MAX;
  p.Lb = ((L + p.n_pass - 1) / p.n_pass + 3) / 4 * 4;
  p.n_blk = ceil_div(n_red, BLK);
  p.tiles = ceil_div(n_rows, OWN);
  const int fit = (512 - 4 * NDIG * p.Lb) / 64;
  p.nstage = fit < NSTAGE_MAX ? fit : NSTAGE_MAX;
  auto pad = [](size_t b) { return (b + ALIGN - 1) & ~(ALIGN - 1); };
  p.head = pad(sizeof(Head));
  p.tops = pad((size_t)TOP_BLOCKS * top_stride(rows ? 1 : N_FACT, L) * sizeof(uint32_t));
  p.digits = pad((size_t)p.n_pass * std::min(p.n_blk, MAX_BLOCKS) * digit_bytes(p.Lb));
  p.sums = pad((size_t)std::min(n_rows, MAX_TILES * OWN) * L * sizeof(long long));
  p.bytes = ALIGN + p.head + p.tops + LEVELS * ((rows ? 1 : 2) * p.digits + 2 * p.sums) + ALIGN;
  return p;
}

// Splits of a launch's contracted axis: the count whose CTAs (one per SM) finish first, counting
// blocks and about 3 blocks of prologue and epilogue per CTA; the smallest of equals.
static int splits(int64_t tiles, int64_t n_blk, int n_pass) {
  const int64_t sms = 148;
  int64_t best = -1;
  int n_split = 1;
  for (int64_t s = 1; s <= std::min<int64_t>(n_blk, 256); ++s) {
    const int64_t per = ceil_div(n_blk, s);
    if (ceil_div(n_blk, per) != s) continue;   // the same ranges as a smaller count
    const int64_t t = ceil_div(tiles * n_pass * s, sms) * (per + 3);
    if (best < 0 || t < best) { best = t; n_split = (int)s; }
  }
  return n_split;
}

template <bool ROWS, bool AL>
static int launch(const Args& a, cudaStream_t st) {
  // one CTA per SM: it takes the SM's tensor memory
  const size_t need = (size_t)NSLOT * (G_BYTES + (ROWS ? 1 : 2) * digit_bytes(a.Lb)) + 8 * N_BARS + 16 + 128;
  const size_t smem = need > 120 * 1024 ? need : 120 * 1024;
  ADX_CUDA_TRY(cudaFuncSetAttribute(product_kernel<ROWS, AL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  ADX_CUDA_TRY(launch_after(product_kernel<ROWS, AL>, (unsigned)(a.tiles * a.n_split * a.n_pass), TPB, smem, st, a));
  return ADX_OK;
}
static_assert(NSLOT * (G_BYTES + 2 * BLK * NDIG * LB_MAX) + 8 * N_BARS + 16 + 128 <= 227 * 1024, "shared memory");

// The workspace's first aligned word is its status, which only adx_rsvd_status clears; the
// parts of a product follow.
static uint8_t* aligned(void* workspace) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(workspace) + ALIGN - 1) & ~uintptr_t(ALIGN - 1));
}

template <bool ROWS>
static int product(const uint8_t* G, int64_t M, int64_t N, const float* f, const float* F, int L, int accumulate,
                   float* out, void* workspace, size_t workspace_bytes, cudaStream_t st, uint32_t polls = POLLS) {
  const int64_t n_rows = ROWS ? M : N, n_red = ROWS ? N : M;
  const Plan p = plan(n_rows, n_red, L, ROWS);
  if (!workspace || workspace_bytes < p.bytes) return ADX_ERR_WORKSPACE;
  int* sticky = reinterpret_cast<int*>(aligned(workspace));
  uint8_t* w = aligned(workspace) + ALIGN;
  Head* h = reinterpret_cast<Head*>(w);
  uint32_t* tops = reinterpret_cast<uint32_t*>(w + p.head);
  uint8_t* dc = w + p.head + p.tops;
  uint8_t* dm = ROWS ? dc : dc + p.digits;
  const size_t level_bytes = (ROWS ? 1 : 2) * p.digits;
  long long* sc = reinterpret_cast<long long*>(dc + LEVELS * level_bytes);
  long long* sm = reinterpret_cast<long long*>(reinterpret_cast<uint8_t*>(sc) + p.sums);
  const int64_t level_sums = 2 * (int64_t)(p.sums / sizeof(long long));
  const int64_t cap = (int64_t)sm_count() * 8, tb = ceil_div(n_red, 8 * (256 / L));
  const int n_tops = (int)(tb < TOP_BLOCKS ? tb : TOP_BLOCKS);
  top_kernel<ROWS><<<n_tops, 256, 0, st>>>(F, f, n_red, L, h, tops);
  ADX_LAUNCH_CHECK();
  auto digits = [&](int64_t blk0, int does) -> int {
    const int64_t n_blk = std::min(p.n_blk - blk0, MAX_BLOCKS);
    const int64_t db = ceil_div(n_blk * (BLK / 16) * p.n_pass * p.Lb, 256);
    ADX_CUDA_TRY(launch_after(digit_kernel<ROWS, false>, (unsigned)std::min(db, cap), 256, 0, st, F, f, n_red, L, p.Lb, p.n_pass,
                              blk0, n_blk, does, h, tops, n_tops, dc, dm));
    return ADX_OK;
  };
  auto low_digits = [&](int64_t blk0, int does) -> int {
    const int64_t n_blk = std::min(p.n_blk - blk0, MAX_BLOCKS);
    const int64_t db = ceil_div(n_blk * (BLK / 16) * p.n_pass * p.Lb, 256);
    ADX_CUDA_TRY(launch_after(digit_kernel<ROWS, true>, (unsigned)std::min(db, cap / 4), 256, 0, st, F, f, n_red, L, p.Lb, p.n_pass,
                              blk0, n_blk, does, h, tops, n_tops, dc + level_bytes, dm + level_bytes));
    return ADX_OK;
  };
  const bool several = p.n_blk > MAX_BLOCKS;   // the counts of all blocks come before the first product
  int rc;
  if (several) {
    for (int64_t b = 0; b < p.n_blk; b += MAX_BLOCKS)
      if ((rc = digits(b, COUNT))) return rc;
    for (int64_t b = 0; b < p.n_blk; b += MAX_BLOCKS)
      if ((rc = low_digits(b, COUNT))) return rc;
  }
  const bool al = (N & 15) == 0 && (reinterpret_cast<uintptr_t>(G) & 15) == 0;
  for (int64_t tile0 = 0; tile0 < p.tiles; tile0 += MAX_TILES) {
    const int64_t tiles = std::min(p.tiles - tile0, MAX_TILES), row0 = tile0 * OWN, rows = std::min(n_rows - row0, tiles * OWN);
    for (int64_t blk0 = 0; blk0 < p.n_blk; blk0 += MAX_BLOCKS) {
      if (several || tile0 == 0) {   // else the digits stand
        const int does = several ? WRITE : COUNT | WRITE;
        if ((rc = digits(blk0, does)) || (rc = low_digits(blk0, does))) return rc;
      }
      const int64_t n_blk = std::min(p.n_blk - blk0, MAX_BLOCKS);
      const int n_split = splits(tiles, n_blk, p.n_pass);
      const bool add = several || n_split > 1;
      if (add && blk0 == 0) ADX_CUDA_TRY(cudaMemsetAsync(sc, 0, LEVELS * 2 * p.sums, st));
      const Args a{G, M, N, dc, dm, level_bytes, level_sums, L, p.Lb, p.n_pass, blk0, n_blk, tile0, tiles, n_split,
                   p.nstage, add, sc, sm, h, &h->err, sticky, polls};
      if ((rc = al ? launch<ROWS, true>(a, st) : launch<ROWS, false>(a, st))) return rc;
    }
    ADX_CUDA_TRY(launch_after(finalize_kernel<ROWS>, (unsigned)ceil_div(rows * L, 256), 256, 0, st, G, M, N, row0, rows, F, f, L,
                              sc, sm, level_sums, h, accumulate, out));
  }
  return ADX_OK;
}

}  // namespace rt
}  // namespace adx

using namespace adx;

extern "C" int adx_rsvd_workspace_bytes(int64_t M, int64_t N, int L, size_t* bytes) {
  if (!bytes || M <= 0 || N <= 0 || L < 1 || L > rt::L_MAX) {
    adx_set_message("adx_rsvd_workspace_bytes: bad argument");
    return ADX_ERR_ARG;
  }
  const size_t r = rt::plan(M, N, L, true).bytes, c = rt::plan(N, M, L, false).bytes;
  *bytes = r > c ? r : c;
  return ADX_OK;
}

extern "C" int adx_rsvd_rows_ws(const uint8_t* G, int64_t M, int64_t N, const float* f, const float* B, int L,
                                float* Y, void* workspace, size_t workspace_bytes, void* stream) {
  if (!G || !f || !B || !Y || M <= 0 || N <= 0 || L < 1 || L > rt::L_MAX) {
    adx_set_message("adx_rsvd_rows_ws: bad argument");
    return ADX_ERR_ARG;
  }
  const int rc = rt::product<true>(G, M, N, f, B, L, 0, Y, workspace, workspace_bytes, as_stream(stream));
  if (rc == ADX_ERR_WORKSPACE) adx_set_message("adx_rsvd_rows_ws: workspace too small");
  return rc;
}

extern "C" int adx_rsvd_cols(const uint8_t* G, int64_t M, int64_t N, const float* f, const float* Y, int L,
                             int accumulate, float* Z, void* workspace, size_t workspace_bytes, void* stream) {
  if (!G || !f || !Y || !Z || M <= 0 || N <= 0 || L < 1 || L > rt::L_MAX) {
    adx_set_message("adx_rsvd_cols: bad argument");
    return ADX_ERR_ARG;
  }
  const int rc = rt::product<false>(G, M, N, f, Y, L, accumulate, Z, workspace, workspace_bytes, as_stream(stream));
  if (rc == ADX_ERR_WORKSPACE) adx_set_message("adx_rsvd_cols: workspace too small");
  return rc;
}

extern "C" int adx_rsvd_status(void* workspace, size_t workspace_bytes, int* status, void* stream) {
  if (!workspace || !status) { adx_set_message("adx_rsvd_status: null pointer"); return ADX_ERR_ARG; }
  if (workspace_bytes < 2 * rt::ALIGN) { adx_set_message("adx_rsvd_status: workspace too small"); return ADX_ERR_WORKSPACE; }
  cudaStream_t st = as_stream(stream);
  int* word = reinterpret_cast<int*>(rt::aligned(workspace));
  ADX_CUDA_TRY(cudaMemcpyAsync(status, word, sizeof(int), cudaMemcpyDeviceToHost, st));
  ADX_CUDA_TRY(cudaStreamSynchronize(st));
  ADX_CUDA_TRY(cudaMemsetAsync(word, 0, sizeof(int), st));
  return ADX_OK;
}

extern "C" int adx_rsvd_wait_selftest(const uint8_t* G, int64_t M, int64_t N, const float* f, const float* F, int L,
                                      int cols, uint32_t limit, float* out, void* workspace, size_t workspace_bytes,
                                      void* stream) {
  if (!G || !f || !F || !out || M <= 0 || N <= 0 || L < 1 || L > rt::L_MAX || limit > rt::POLLS) {
    adx_set_message("adx_rsvd_wait_selftest: bad argument");
    return ADX_ERR_ARG;
  }
  cudaStream_t st = as_stream(stream);
  const int rc = cols ? rt::product<false>(G, M, N, f, F, L, 0, out, workspace, workspace_bytes, st, limit)
                      : rt::product<true>(G, M, N, f, F, L, 0, out, workspace, workspace_bytes, st, limit);
  if (rc == ADX_ERR_WORKSPACE) adx_set_message("adx_rsvd_wait_selftest: workspace too small");
  return rc;
}
