// f64-accurate GEMM from BF16 slices on tcgen05 tensor cores (Ozaki scheme).
//
// C = A*B with A (m x k) and B (k x n) row-major f64. No reference
// counterpart: it stands in for the f64 tier of kernels::gemm::gemm_2d
// (src/kernels/gemm.rs:290) where GB300's FP64 rate (~1.2 TFLOP/s) makes a
// native FP64 GEMM slow.
//
// 1. Scaling: e_a[i] = frexp exponent of max_k |a_ik| (|a_ik| < 2^e_a[i]),
//    e_b[j] likewise over column j of B. Powers of two: exact.
// 2. Slicing: x = a_ik * 2^-e_a[i] in (-1, 1) becomes the 126-bit fixed-point
//    integer X = round(x * 2^126), split into S signed b-bit digits
//    (b = 8, 7 or 6: the widest whose exactness bounds below hold for the
//    call's K and S) whose weighted sum is X rounded to the nearest
//    multiple of 2^(127 - b - b(S-1)): each digit lies in [-2^(b-1), 2^(b-1)],
//    exactly representable in BF16, and x = sum_t digit_t * 2^-(b - 1 + bt)
//    up to 2^-(bS). Slices are stored K-major ([S][rows][kpad] bf16) for A
//    and for B^T (the B slicer transposes through shared memory).
// 3. Products: for every slice pair (s, t) with s + t <= S-1 (what the others
//    can add up to counts in the choice of S: ozaki_count_holds in
//    f64_round.cuh), P = A_s * B_t^T on the
//    tensor cores with FP32 accumulation. |digit products| <= 2^(2b-2), so
//    every partial sum of a K <= 2^(26-2b) chunk (4096 for b = 7) is an
//    integer of at most 2^24: the FP32 accumulation is EXACT.
// 4. Cross-slice accumulation: the exact products of one diagonal
//    (s + t = d) are summed as int32 and carried, from d = S-1 up to d = 0,
//    in one int32 per element: R <- floor(R / 2^b) + D_d, the low b bits of
//    the old R being final (digit S-2-d). After d = 0 the exact total is
//    T = R 2^(b(S-1)) + sum_t digit_t 2^(bt), rounded once to f64 with
//    integer operations (no FP64 op) and scaled by
//    2^(e_a[i] + e_b[j] + 2 - 2b - b(S-1)).
//
// The tensor-core kernel is persistent (one CTA per SM) and warp-specialised:
//   warp 0      : TMA producer, ring of A and B bf16 tiles 64 wide in K,
//                 128-byte swizzle;
//   warp 1      : TMEM allocator and single-thread tcgen05.mma issuer;
//   warps 2..9  : epilogue (one TMEM lane = one tile row per thread, two warps
//                 per lane quarter splitting the columns): fold the finished
//                 accumulator into the carried int32 sums R, hand it back to
//                 the MMA warp, retire the digits, and round every element's
//                 exact total once after d = 0.
// One large problem runs on CTA pairs (cta_group::2, M=256 N=256 K=16): each
// CTA loads 128 rows of A and of B^T, 32 KB per 64-wide K block for the MMA
// time of 128 x 256 of C, and holds its two 128 x 256 accumulators in all of
// TMEM. One CTA with a 128 x 256 tile takes 48 KB for the same, and its one
// accumulator (R filled the other half of TMEM) kept the tensor pipe 63%
// active: its MMA warp waited for TMA data 29% of its time, for the epilogue
// 8%. 8192^3 with 28 slice products (30.8 TFLOP): 20.4 -> 18.2 ms, 1.69
// PFLOP/s, at the power limit.
// Small problems and grouped launches (many small problems, one tile list)
// use 128 x 128 tiles, a 6-stage ring and two accumulators in turn, and keep
// the digits in TMEM and registers (the grouped epilogue below describes it).
// Every mbarrier wait is bounded; on give-up the kernel records an error
// word, drains its own copies and MMAs (bounded), frees TMEM and returns.
#include <mutex>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "f64_round.cuh"
#include "nrs_internal.cuh"

namespace {

constexpr int OZ_BM = 128;
constexpr int OZ_BN = 256;
// K per ring stage: 64 bf16 = one 128-byte swizzle row. (32 per stage with
// the 64-byte swizzle and 9 stages computed the same results but ran 28%
// slower at 8192^3: the per-stage barrier and issue work doubles.)
constexpr int OZ_BK = 64;
constexpr int OZ_STAGES = 4;
constexpr int OZ_A_BYTES = OZ_BM * OZ_BK * 2;  // 16 KB
constexpr int OZ_THREADS = 320;                 // 10 warps: TMA, MMA, 8 epilogue
constexpr int OZ_TMEM_COLS = 512;               // accumulator(s) + diagonal sums
// Signed digits of b bits: |digit| <= 2^(b-1), exact in BF16 (8-bit
// significand) for b <= 8; products <= 2^(2b-2), so a K chunk of 2^(26-2b)
// sums exactly in FP32 (at most 2^24). Wider digits need fewer slices for
// the same precision (S = ceil(54 / b): 7 slices and 28 pairs for b = 8,
// 8 and 36 for b = 7, 9 and 45 for b = 6) but shorter exact K chunks.
constexpr int kChunkOf(int b) { return 1 << (26 - 2 * b); }
constexpr int kTopOf(int b) { return 127 - b; }  // position of the top digit in X
constexpr int OZ_MAX_SLICES = 16;

// Tile geometry per kernel. The estimate: 128 x 256 tiles, 4 stages (the
// constants above). Grouped launches, mostly small problems: 128 x 128 tiles
// (less padding for narrow problems), two accumulators in TMEM columns 0..255
// so the MMAs of the next group run while the epilogue reads the last one,
// the diagonal sums in 256..383, and 6 stages of 32 KB. One large problem:
// CTA pairs on 256 x 256 tiles; each CTA loads 128 rows of A and 128 of B^T
// (32 KB a stage) and holds 128 x 256 of C in two accumulators.
template <bool EST, bool G>
struct OzGeom {
  static constexpr bool PAIR = !EST && !G;
  static constexpr int BM = PAIR ? 2 * OZ_BM : OZ_BM;  // tile rows
  static constexpr int BN = G ? 128 : OZ_BN;           // tile columns, accumulator columns
  static constexpr int LOAD_N = EST ? OZ_BN : 128;     // B^T rows that a CTA loads
  static constexpr int STAGES = EST ? OZ_STAGES : PAIR ? 7 : 6;
  static constexpr int STAGE_BYTES = OZ_A_BYTES + LOAD_N * OZ_BK * 2;
  // The column exponents of each grouped epilogue warp's 64 tile columns,
  // staged once per tile.
  static constexpr int EB_BYTES = G ? 8 * 64 * 4 : 0;
  static constexpr int SMEM = STAGES * STAGE_BYTES + EB_BYTES + 1024 /*align*/ + 256 /*barriers*/;
  static_assert(SMEM <= 232448, "shared memory of one CTA");
  // Instruction descriptor, kind::f16: D f32 (bits 4-5 = 1), A and B bf16
  // (bits 7-9, 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 at bits
  // 17-22, M >> 4 at bits 24-28.
  static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                                    ((uint32_t)(BM >> 4) << 24);
};
// Grouped launches with S > 9 keep digits 8..14 in a per-CTA 128 x 128 slot
// of 8-byte records (column-major: for one column a warp's 32 rows are 256
// contiguous bytes).
constexpr int OZ_DIGIT_BYTES = 8;


// ---------------------------------------------------------------------------
// tcgen05 / TMEM wrappers
// ---------------------------------------------------------------------------
// (PAIR: the cta_group::2 forms, which a kernel uses throughout or not at all)
template <bool PAIR>
NRS_DEV void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
  if constexpr (PAIR) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  } else {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
}
template <bool PAIR>
NRS_DEV void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  if constexpr (PAIR)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
  else
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
NRS_DEV void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
NRS_DEV void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

template <bool PAIR>
NRS_DEV void tc_mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                         uint32_t accumulate) {
  if constexpr (PAIR)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives on `bar` (PAIR: in both CTAs, or in this one only) once the MMAs
// issued so far are done.
template <bool PAIR>
NRS_DEV void tc_commit(uint64_t* bar, bool own = false) {
  if (PAIR && own)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
  else if constexpr (PAIR)
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
            smem_u32(bar)),
        "h"((uint16_t)3)
        : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// One lane of a converged warp (the same one every time).
NRS_DEV bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "elect.sync _|P, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(p));
  return p != 0;
}

// 32 lanes x 16 columns into v[0..15] without waiting: several loads can be
// in flight before one tcgen05.wait::ld.
NRS_DEV void tmem_ld16_nowait(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
// 32 lanes x 8 columns into v[0..7] without waiting.
NRS_DEV void tmem_ld8_nowait(uint32_t taddr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                 "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
// Waits for every load; `v` (16 registers of one of them) is usable after it.
NRS_DEV void tmem_wait_ld16(uint32_t* v) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                 "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]),
                 "+r"(v[15])::"memory");
}
NRS_DEV void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

NRS_DEV void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
NRS_DEV void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor, K-major operand with 128-byte swizzle:
// rows of 128 B, 8-row core-matrix groups 1024 B apart (SBO), descriptor
// version 1 (bits 46-47), swizzle mode 2 = 128B (bits 61-63).
NRS_DEV uint64_t smem_desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)(16 >> 4) << 16;    // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;  // stride byte offset
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// What a slice count has to satisfy (oz_decide).
struct OzRule {
  int target_bits;  // operand bits wanted at spread 1 (53 for f64, 26 for f32)
  int digit_bits;
  int max_slices;   // beyond: 0 (the caller's FP64 / FP32 kernel runs instead)
  float drop_scale; // K / tau of ozaki_count_holds
  int exp_limit;    // max row + column exponent whose dot products cannot overflow T
};

// Words of the decision block, zeroed by oz_max, filled by oz_est and the
// estimate product.
// OZ_W_COUNT: the slice count that oz_slice decided on, read by the launches
// behind it.
// OZ_W_DROP: 1 / min_ij (|A'||B'|)_ij over its nonzero entries, as float bits.
// OZ_W_HOLE: pass 1 met a (|A'||B'|)_ij of 0 whose row or column is not zero.
// OZ_W_TINY: an operand holds a nonzero entry so small (est_bits) that its
// products with another can be lost in |A'||B'|.
enum {
  OZ_W_SPREAD = 0, OZ_W_NONFINITE = 1, OZ_W_DROP = 2, OZ_W_HOLE = 3, OZ_W_EXP_A = 4, OZ_W_EXP_B = 5, OZ_W_TINY = 6,
  OZ_W_COUNT = 8, OZ_WORDS = 9
};
// Raises a word to at least v; most callers find it there already.
__device__ __forceinline__ void raise_word(uint32_t* w, uint32_t v) {
  if (__ldcg(w) < v) atomicMax(w, v);
}
constexpr int kExpBias = 4096;  // exponents are collected biased, as unsigned maxima

// The slice count for the measured spread and smallest (|A'||B'|)_ij: the
// smallest S for which ozaki_count_holds; 0 when no count up to the limit
// does, an operand holds Inf or NaN, or a partial sum could overflow the
// element type (the plain kernel then gives its own Inf / NaN). Where
// (|A'||B'|)_ij is 0 (zero rows and columns, identity, block-diagonal and
// one-hot operands) every product of the sum has a zero factor, whose digits are
// zeros: C_ij is exact at any count. Only tiny entries make that uncertain.
__device__ __forceinline__ int oz_decide(const uint32_t* w, const OzRule& r) {
  // (two loads in flight together: every block of oz_slice starts with them, and
  // one load after another cost 13 us at 4096^3)
  const uint4 lo = __ldcg(reinterpret_cast<const uint4*>(w)), hi = __ldcg(reinterpret_cast<const uint4*>(w) + 1);
  static_assert(OZ_W_HOLE == 3 && OZ_W_EXP_A == 4 && OZ_W_EXP_B == 5 && OZ_W_TINY == 6, "the words' places");
  const float spread = __uint_as_float(lo.x), drop = __uint_as_float(lo.z) * r.drop_scale;
  if (lo.y | (lo.w & hi.z)) return 0;  // (both 0 or 1)
  const int e = (int)hi.x + (int)hi.y - 2 * kExpBias;
  if (e > r.exp_limit) return 0;
  int S = (r.target_bits + r.digit_bits - 1) / r.digit_bits;
  for (; S <= r.max_slices; ++S)
    if (ozaki_count_holds(S, r.digit_bits, r.target_bits, spread, drop)) return S;
  return 0;
}

// Fixed-point scale of the estimate's row / column sums of |x'| (smaller for
// K beyond 2^15): integers add in any order to the same sum.
constexpr float kSumScale = 65536.0f;

struct OzParams {
  int64_t m, n, k, kpad;
  int slices;
  int kchunks;     // estimate only, as n_pairs
  int n_pairs;     // pairs x kchunks work units per tile
  int tiles_m, tiles_n;
  int group_m;     // tile rasterisation group height
  const int* ea;   // row exponents of A
  const int* eb;   // column exponents of B
  uint8_t* acc;    // per-CTA digit slots (16-byte aligned)
  double* C;       // float when f32 (and not split)
  int64_t ldc;
  int digit_bits;  // b
  int kchunk;      // exact FP32 K chunk, 2^(26-2b)
  int accumulate;  // C += result instead of C = result
  uint32_t* err;
  // Spread estimate only (EST kernel): row sums of |A'| and column sums of
  // |B'| (operands scaled by their row / column exponents; fixed point, in
  // units of sum_unit), and the decision words, of which it raises the spread
  // (max_ij of the ratio) and the inverse of the smallest nonzero D, as float
  // bits.
  const uint32_t* ra;
  const uint32_t* cb;
  float sum_unit;
  uint32_t* est;
  // Slice count decided on the device (null: the count is `slices`). A count
  // of 0 makes the launch return at once.
  const uint32_t* count;
  // One problem (no tile list): K in `splits` ranges of split_blocks 64-wide blocks. With several, range z
  // writes its product to the f64 slab C + z m n (row pitch n).
  int splits, split_blocks;
  int f32;
  int n_tiles;  // tiles x splits
  // Grouped launch only: the tile list and the problems it points into.
  const struct OzTile* tiles;
  const struct OzProb* probs;
};

// One problem of a grouped launch: its slices are rows [rowoff, rowoff + m)
// of the stacked A slices and [coloff, coloff + n) of the stacked B^T slices
// (row pitch = the group's largest kpad; this problem's rows are zero from
// its own k to its kpad), and its exponents sit at the same offsets.
struct OzProb {
  int64_t m, n, kpad;
  int64_t rowoff, coloff;
  void* C;  // double, or float when f32
  int64_t ldc;
  int32_t kchunks, n_pairs;
  int32_t accumulate, f32;
};
struct OzTile {
  int32_t prob, tm, tn, pad;
};

// Everything a CTA needs about the tile it works on.
struct TileCtx {
  int64_t m, n;        // the problem's C dimensions
  int64_t arow, brow;  // TMA row coordinates of the tile's A / B^T boxes
  int kbase;           // first 64-wide K block
  int64_t row0, col0;  // tile origin inside the problem
  int kblocks, n_pairs, kchunks;
  const int* ea;
  const int* eb;
  void* C;  // double, or float when f32
  int64_t ldc;
  int accumulate, f32;
};

// Work units of a tile, in order: diagonals from the least significant
// (d = S-1) to the most significant (d = 0), within a diagonal the pairs
// (s, t = d - s) for s = 0..d, within a pair its K chunks; the last unit of a
// tile is pair (0,0). Walked incrementally (no search per unit).
struct PairIter {
  int d, s, chunk;
  __device__ __forceinline__ void start(int S) {
    d = S - 1;
    s = 0;
    chunk = 0;
  }
  __device__ __forceinline__ int t() const { return d - s; }
  __device__ __forceinline__ bool diag_first() const { return s == 0 && chunk == 0; }
  // units of the current diagonal from this one on, this one included
  __device__ __forceinline__ int left(int kchunks) const { return (d - s) * kchunks + (kchunks - chunk); }
  __device__ __forceinline__ void next(int kchunks) {
    if (++chunk == kchunks) {
      chunk = 0;
      if (s < d) {
        ++s;
      } else {
        --d;
        s = 0;
      }
    }
  }
};

__device__ __forceinline__ void tile_coords(int tile, const OzParams& P, int& tm, int& tn) {
  // Grouped rasterisation: consecutive tiles walk group_m tile rows before
  // moving along N, so concurrently active tiles share A and B panels in L2.
  const int per_group = P.group_m * P.tiles_n;
  const int g = tile / per_group;
  const int first_m = g * P.group_m;
  const int gm = (P.tiles_m - first_m) < P.group_m ? (P.tiles_m - first_m) : P.group_m;
  const int r = tile % per_group;
  tm = first_m + r % gm;
  tn = r / gm;
}

// Units of a tile that the tensor cores accumulate together. With one K
// chunk (kchunks == 1) consecutive units are consecutive pairs; the pairs of
// one diagonal can share the fp32 accumulator as long as the sum stays an
// exact integer: each pair's sum is at most kblocks * 64 * 2^(2b-2), so up
// to 2^24 / that many pairs. Several K chunks (and the spread estimate)
// keep one unit per accumulation.
__device__ __forceinline__ int merge_count(const TileCtx& c, const OzParams& P, bool est) {
  if (est || c.kchunks != 1) return 1;
  const int64_t per_pair = (int64_t)c.kblocks * OZ_BK << (2 * P.digit_bits - 2);
  const int64_t g = ((int64_t)1 << 24) / per_pair;
  return g < 1 ? 1 : (int)g;
}
// Units in the accumulation group that starts at `pi`: the same diagonal, at
// most `gm` units.
__device__ __forceinline__ int group_size(const PairIter& pi, int gm, int kchunks) {
  const int l = pi.left(kchunks);
  return l < gm ? l : gm;
}


// The first up to 8 of `nd` digit planes (a byte per column, 8 columns at
// `p`) as one word per column, digit t in byte t.
__device__ __forceinline__ void digits8(const uint8_t* p, size_t plane, int nd, uint64_t (&out)[8]) {
  uint2 d[8];
#pragma unroll
  for (int t = 0; t < 8; ++t)
    d[t] = t < nd ? __ldcg(reinterpret_cast<const uint2*>(p + t * plane)) : make_uint2(0, 0);
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    uint32_t h[2][4];  // [digits 0..3 / 4..7][column]
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const uint32_t a = g ? d[4 * t].y : d[4 * t].x, b = g ? d[4 * t + 1].y : d[4 * t + 1].x;
      const uint32_t c = g ? d[4 * t + 2].y : d[4 * t + 2].x, e = g ? d[4 * t + 3].y : d[4 * t + 3].x;
      const uint32_t ab0 = __byte_perm(a, b, 0x5140), ab1 = __byte_perm(a, b, 0x7362);  // a0 b0 a1 b1, a2 b2 a3 b3
      const uint32_t ce0 = __byte_perm(c, e, 0x5140), ce1 = __byte_perm(c, e, 0x7362);
      h[t][0] = __byte_perm(ab0, ce0, 0x5410);
      h[t][1] = __byte_perm(ab0, ce0, 0x7632);
      h[t][2] = __byte_perm(ab1, ce1, 0x5410);
      h[t][3] = __byte_perm(ab1, ce1, 0x7632);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) out[g * 4 + q] = (uint64_t)h[1][q] << 32 | h[0][q];
  }
}

// Writes 8 consecutive columns of one tile row of C (f64, or f32 when F32):
// R values w, digits 0..7 of each column in `lo` (digit t = byte t; with B8,
// i.e. 8-bit digits, and S <= 9 left-aligned instead, digit S-2 on top),
// digits 8..14 in `hi` (S > 9) and the column exponents; `left` of the 8 columns lie inside the problem; the row
// starts at element `off` of C. The conversions run straight-line for all 8
// (the digit width is a template argument and the slice count is tested
// once, so no branch separates the elements' chains: with both tested per
// element this pass took 75,000 cycles per 128 x 128 tile, two thirds of a
// small tile's time); zero, tiny, subnormal and overflowing results are redone by
// the exact path.
template <bool F32, bool B8>
__device__ __forceinline__ void retire8(const uint32_t (&w)[8], const uint64_t (&lo)[8], const uint64_t (&hi)[8],
                                        const int* eb, int left, int b, int S, int ebase, void* C,
                                        int64_t off, bool accumulate) {
  using Fmt = typename std::conditional<F32, NrsF32Fmt, NrsF64Fmt>::type;
  const int nd = S - 1;
  uint64_t bits[8];
  int ex[8];
  unsigned special = 0;
#pragma unroll
  for (int e = 0; e < 8; ++e) ex[e] = e < left ? eb[e] : 0;
  const bool top = B8 && nd <= 8;
  if (top) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      bool sp;
      bits[e] = ozaki_round96<Fmt>((int32_t)w[e], (uint32_t)(lo[e] >> 32), (uint32_t)lo[e], ebase + ex[e] + 8 * nd, sp);
      special |= (unsigned)sp << e;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      bool neg, sp;
      uint64_t mhi, mlo;
      ozaki_exact_total((int32_t)w[e], lo[e], hi[e], B8 ? 8 : b, S, neg, mhi, mlo);
      bits[e] = int128_to_float_bits_fast<Fmt>(neg, mhi, mlo, ebase + ex[e], sp);
      special |= (unsigned)sp << e;
    }
  }
  if (special) {
#pragma unroll 1
    for (int e = 0; e < 8; ++e) {
      if (!((special >> e) & 1)) continue;
      uint64_t l = 0, h = 0;
      uint32_t r = 0;
      int x = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q == e) {
          l = lo[q];
          h = hi[q];
          r = w[q];
          x = ex[q];
        }
      if (top) l = nd ? l >> (64 - 8 * nd) : 0;
      bool neg;
      uint64_t mhi, mlo;
      ozaki_exact_total((int32_t)r, l, h, b, S, neg, mhi, mlo);
      const uint64_t v = int128_to_float_bits<Fmt>(neg, mhi, mlo, ebase + x);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q == e) bits[q] = v;
    }
  }
  using T = typename std::conditional<F32, float, double>::type;
  constexpr int PER = 16 / (int)sizeof(T);
  T* cp = static_cast<T*>(C) + off;
  T v[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    if constexpr (F32) v[e] = __uint_as_float((uint32_t)bits[e]);
    else v[e] = __longlong_as_double((long long)bits[e]);
  }
  if (!accumulate && left >= 8 && (reinterpret_cast<uintptr_t>(cp) & 15) == 0) {
#pragma unroll
    for (int q = 0; q < 8 / PER; ++q) {
      uint4 u;
      memcpy(&u, &v[q * PER], 16);
      reinterpret_cast<uint4*>(cp)[q] = u;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (e < left) cp[e] = accumulate ? cp[e] + v[e] : v[e];
  }
}

// `S`: the launch's slice count (tile lists carry their own pair counts).
// `rank`: the CTA's in its pair, whose tile is 256 rows and loads 128 + 128
// rows of B^T.
template <bool EST, bool G>
__device__ __forceinline__ TileCtx tile_ctx(const OzParams& P, int S, int tile, uint32_t rank) {
  using Geo = OzGeom<EST, G>;
  TileCtx c;
  c.kbase = 0;
  if (!EST && !(G && P.tiles)) {
    const int per = P.tiles_m * P.tiles_n;
    const int z = tile / per;
    int tm, tn;
    tile_coords(tile - z * per, P, tm, tn);
    c.m = P.m;
    c.n = P.n;
    c.row0 = c.arow = (int64_t)tm * Geo::BM + rank * OZ_BM;
    c.col0 = (int64_t)tn * Geo::BN;
    c.brow = c.col0 + rank * OZ_BM;
    c.kbase = z * P.split_blocks;
    const int kb = (int)((P.kpad + OZ_BK - 1) / OZ_BK) - c.kbase;
    c.kblocks = kb < P.split_blocks ? kb : P.split_blocks;
    const int chunk_blocks = P.kchunk / OZ_BK;
    c.kchunks = (c.kblocks + chunk_blocks - 1) / chunk_blocks;
    c.n_pairs = S * (S + 1) / 2 * c.kchunks;
    c.ea = P.ea;
    c.eb = P.eb;
    if (P.splits > 1) {
      c.C = P.C + (int64_t)z * P.m * P.n;
      c.ldc = P.n;
      c.accumulate = c.f32 = 0;
    } else {
      c.C = P.C;
      c.ldc = P.ldc;
      c.accumulate = P.accumulate;
      c.f32 = P.f32;
    }
  } else if (G) {
    const OzTile t = P.tiles[tile];
    const OzProb& q = P.probs[t.prob];
    c.m = q.m;
    c.n = q.n;
    c.row0 = (int64_t)t.tm * OZ_BM;
    c.col0 = (int64_t)t.tn * Geo::BN;
    c.arow = q.rowoff + c.row0;
    c.brow = q.coloff + c.col0;
    c.kblocks = (int)((q.kpad + OZ_BK - 1) / OZ_BK);
    c.n_pairs = q.n_pairs;
    c.kchunks = q.kchunks;
    c.ea = P.ea + q.rowoff;
    c.eb = P.eb + q.coloff;
    c.C = q.C;
    c.ldc = q.ldc;
    c.accumulate = q.accumulate;
    c.f32 = q.f32;
  } else {
    int tm, tn;
    tile_coords(tile, P, tm, tn);
    c.m = P.m;
    c.n = P.n;
    c.row0 = c.arow = (int64_t)tm * OZ_BM;
    c.col0 = c.brow = (int64_t)tn * OZ_BN;
    c.kblocks = (int)((P.kpad + OZ_BK - 1) / OZ_BK);
    c.n_pairs = P.n_pairs;
    c.kchunks = P.kchunks;
  }
  return c;
}

// EST = false: the slice-pair GEMM described in the file header.
// EST = true : the same pipeline on the spread-estimate operands (one K chunk
//              covering all of K): pass 1 (slices = 1) runs the one product
//              D = |A'| |B'|^T; pass 2 (slices = 2) also runs the two cross
//              products N = |A'| 1_B^T + 1_A |B'|^T of slices 0 and 1 (|x'|
//              and the nonzero indicator). The epilogue folds
//              max_ij (numerator_ij / D_ij) and the smallest nonzero D_ij into
//              P.est instead of writing C.
// B8: 8-bit digits (else 7 or 6, P.digit_bits).
template <bool EST, bool G, bool B8>
__global__ void __launch_bounds__(OZ_THREADS, 1)
    ozaki_tc_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                    OzParams P) {
  using Geo = OzGeom<EST, G>;
  constexpr bool PAIR = Geo::PAIR;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Geo::STAGES * Geo::STAGE_BYTES + Geo::EB_BYTES);
  uint64_t* empty = full + Geo::STAGES;
  uint64_t* accf = empty + Geo::STAGES;
  uint64_t* acce = accf + 2;
  uint64_t* drain = acce + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  // (warp-uniform, and known to be)
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int n_tiles = P.n_tiles;
  // A pair works on one tile: its rank 0 issues the MMAs of both.
  const uint32_t rank = PAIR ? cluster_rank() : 0;
  const int tile0 = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int tile_step = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  launch_next();

  if (threadIdx.x == 0) {
    for (int s = 0; s < Geo::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&accf[b], 1);
      mbar_init(&acce[b], PAIR ? 16 : 8);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_mbar_init();
    prefetch_tensormap(&mapA);
    prefetch_tensormap(&mapB);
  }
  if (warp == 1) {
    tmem_alloc<PAIR>(tmem_slot, OZ_TMEM_COLS);
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();  // both CTAs' barriers are set up
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // (the barriers and TMEM are set up while the kernel before drains)
  launch_wait();
  const int S = P.count ? (int)__ldcg(P.count) : P.slices;
  if (S == 0) {  // (the same word for every thread)
    if (warp == 1) tmem_dealloc<PAIR>(tmem_base, OZ_TMEM_COLS);
    return;
  }
  const int final_shift = 2 - 2 * P.digit_bits - P.digit_bits * (S - 1);

  auto bounded = [&](uint64_t* bar, uint32_t phase, uint32_t site, auto cluster) -> bool {
    for (uint32_t i = 0; i < NRS_WAIT_LIMIT; ++i) {
      if (cluster ? mbar_try_wait_cluster(bar, phase) : mbar_try_wait(bar, phase)) return true;
      if (*abort_flag) return false;
    }
    *abort_flag = 1;
    atomicOr(P.err, NRS_DEVERR_GEMM_TC | (site << 8));
    return false;
  };

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (elect_one()) {
      uint32_t s = 0, ph = 1, it = 0;  // ring slot, its empty phase, loads issued
      bool ok = true;
      const int chunk_blocks = P.kchunk / OZ_BK;
      for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
        const TileCtx c = tile_ctx<EST, G>(P, S, tile, rank);
        const int32_t arow = (int32_t)c.arow, brow = (int32_t)c.brow;
        PairIter pr;
        pr.start(S);
        for (int u = 0; u < c.n_pairs && ok; ++u, pr.next(c.kchunks)) {
          const int kb0 = pr.chunk * chunk_blocks;
          const int kb1 = kb0 + chunk_blocks < c.kblocks ? kb0 + chunk_blocks : c.kblocks;
          const int32_t sa = pr.s, sb = pr.t();
          int32_t x = (c.kbase + kb0) * OZ_BK;
          for (int kb = kb0; kb < kb1; ++kb, ++it, x += OZ_BK) {
            if (!bounded(&empty[s], ph, 1, std::false_type{})) { ok = false; break; }
            uint8_t* st = smem + s * Geo::STAGE_BYTES;
            if constexpr (PAIR) {
              // both CTAs' bytes are counted by rank 0's barrier
              if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * Geo::STAGE_BYTES);
              const uint32_t bar = cluster_addr(&full[s], 0);
              tma_load_3d_pair(st, &mapA, bar, x, arow, sa);
              tma_load_3d_pair(st + OZ_A_BYTES, &mapB, bar, x, brow, sb);
            } else {
              mbar_arrive_expect_tx(&full[s], Geo::STAGE_BYTES);
              tma_load_3d(st, &mapA, &full[s], x, arow, sa);
              tma_load_3d(st + OZ_A_BYTES, &mapB, &full[s], x, brow, sb);
            }
            if (++s == Geo::STAGES) {
              s = 0;
              ph ^= 1;
            }
          }
        }
      }
      if (PAIR && ok) {
        // rank 0's MMAs release this CTA's stages too: let the last of those
        // arrivals land before the CTA can exit
        for (int j = 0; j < Geo::STAGES && ok; ++j) {
          ok = bounded(&empty[s], ph, 1, std::false_type{});
          if (++s == Geo::STAGES) {
            s = 0;
            ph ^= 1;
          }
        }
      }
      if (PAIR && !ok && rank != 0) {
        // Rank 0's barriers, which this CTA cannot wait on, count its copies
        // in flight: they take microseconds, this a millisecond.
        for (int j = 0; j < 100; ++j) __nanosleep(10000);
      } else if (!ok) {
        // Drain: wait (bounded) for the copies still in flight.
        for (uint32_t j = (it >= Geo::STAGES ? it - Geo::STAGES : 0); j < it; ++j)
          mbar_wait_bounded(&full[j % Geo::STAGES], (j / Geo::STAGES) & 1, 1u << 16);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (rank == 0 && elect_one()) {
      uint32_t s = 0, ph = 0, ai = 0;  // ring slot, its full phase, accumulation groups
      bool ok = true;
      const bool two = !EST || P.slices == 1;
      const int chunk_blocks = P.kchunk / OZ_BK;
      const uint64_t adesc0 = smem_desc_sw128(smem_u32(smem));
      const uint64_t bdesc0 = smem_desc_sw128(smem_u32(smem) + OZ_A_BYTES);
      for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
        const TileCtx c = tile_ctx<EST, G>(P, S, tile, rank);
        const int gm = merge_count(c, P, EST);
        PairIter pr;
        pr.start(S);
        for (int u = 0; u < c.n_pairs && ok; ++ai) {
          const int g = group_size(pr, gm, c.kchunks);
          // Two accumulators (TMEM columns 0..127, 128..255 in grouped
          // launches, else 0..255, 256..511; the estimate's second pass has
          // only the first), used in turn; the epilogue frees one as soon as
          // it has read it.
          const int buf = two ? (int)(ai & 1) : 0;
          const uint32_t aph = (two ? ai >> 1 : ai) & 1;
          if (!bounded(&acce[buf], aph ^ 1, 2, std::bool_constant<PAIR>{})) { ok = false; break; }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + (uint32_t)(buf * Geo::BN);
          uint32_t accum = 0;
          for (int j = 0; j < g && ok; ++j, pr.next(c.kchunks)) {
            const int kb0 = pr.chunk * chunk_blocks;
            const int kb1 = kb0 + chunk_blocks < c.kblocks ? kb0 + chunk_blocks : c.kblocks;
            for (int kb = kb0; kb < kb1; ++kb) {
              if (!bounded(&full[s], ph, 3, std::false_type{})) { ok = false; break; }
              tc_fence_after();
              // (a stage or K step moves the descriptors' 16-byte address field)
              const uint64_t off = (uint64_t)(s * (Geo::STAGE_BYTES / 16));
#pragma unroll
              for (int kk = 0; kk < OZ_BK / 16; ++kk) {
                tc_mma_bf16<PAIR>(d_tmem, adesc0 + off + kk * 2, bdesc0 + off + kk * 2, Geo::IDESC, accum);
                accum = 1;
              }
              tc_commit<PAIR>(&empty[s]);  // frees the stage once these MMAs have read it
              if (++s == Geo::STAGES) {
                s = 0;
                ph ^= 1;
              }
            }
          }
          if (!ok) break;
          tc_commit<PAIR>(&accf[buf]);  // accumulator ready once every MMA above completes
          u += g;
        }
      }
      // Make sure no MMA is still running before TMEM is released.
      tc_commit<PAIR>(drain, true);
      mbar_wait_bounded(drain, 0, 1u << 20);
    }
  } else if (EST) {
    // ---------------- spread-estimate epilogue (warps 2..9) ----------------
    // Same TMEM geometry as below. Units of a tile: pass 1: (0,0) = D;
    // pass 2: (0,1), (1,0) summed in fp32 into columns 256..511 = N, then
    // (0,0) = D. Per element r = numerator / D (pass 1: numerator =
    // (ra_i + cb_j) 2^96, the operands' 2^48 scale factors). D = 0 with a
    // nonzero numerator: pass 1 notes a hole; in pass 2 a product was lost,
    // which gives +inf. The running max is float bits.
    __shared__ float est_cb[EST ? 8 : 1][EST ? OZ_BN / 2 : 1];
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row_in_tile = q * 32 + lane;
    const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16) + half * (OZ_BN / 2);
    const uint32_t acc_t = lane_base;
    const uint32_t dsum_t = lane_base + OZ_BN;
    uint32_t ai = 0;
    const float inf = __uint_as_float(0x7f800000u);
    // (the numerators' scale, in the sums already: 2^31 2^96 2^-16 at most)
    const float unit = 0x1p96f * P.sum_unit;
    float rmax = 0.0f, dmin = inf;
    bool hole = false;
    bool ok = true;
    for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
      const TileCtx tc = tile_ctx<EST, G>(P, S, tile, rank);
      const int64_t row = tc.row0 + row_in_tile;
      const bool row_ok = row < tc.m;
      const int64_t col0 = tc.col0 + half * (OZ_BN / 2);
      // Rows and columns outside the problem have D = 0 (the loads fill with
      // zeros) and here a numerator of -inf: no ratio and no hole. Pass 2's is
      // 0 there.
      const float ra = row_ok ? (float)P.ra[row] * unit : -inf;
      const bool pass1 = P.slices == 1;
      // this warp's column sums, read while the product runs
      __syncwarp();
#pragma unroll
      for (int j = 0; j < OZ_BN / 2; j += 32) {
        const int64_t col = col0 + j + lane;
        est_cb[warp - 2][j + lane] = pass1 && col < tc.n ? (float)P.cb[col] * unit : -inf;
      }
      __syncwarp();
      PairIter pr;
      pr.start(S);
      for (int u = 0; u < tc.n_pairs; ++u, ++ai, pr.next(1)) {
        const int buf = pass1 ? (int)(ai & 1) : 0;
        if (!bounded(&accf[buf], (pass1 ? ai >> 1 : ai) & 1, 4, std::false_type{})) { ok = false; break; }
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < OZ_BN / 32; ++c) {
          uint32_t v[16], w[16];
          tmem_ld16_nowait(acc_t + buf * OZ_BN + c * 16, v);
          if (!pass1 && (pr.d == 0 || pr.s == 1)) tmem_ld16_nowait(dsum_t + c * 16, w);
          tmem_wait_ld();
          if (pr.d == 1) {
            if (pr.s == 1) {
#pragma unroll
              for (int e = 0; e < 16; ++e)
                w[e] = __float_as_uint(__uint_as_float(w[e]) + __uint_as_float(v[e]));
              tmem_st16(dsum_t + c * 16, w);
            } else {
              tmem_st16(dsum_t + c * 16, v);
            }
            continue;
          }
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            // (straight-line: with a mask and a branch per element 1024^3 took
            // 12 us more)
            const float D = __uint_as_float(v[e]);
            const float num = pass1 ? ra + est_cb[warp - 2][c * 16 + e] : __uint_as_float(w[e]);
            const bool some = D > 0.0f;
            // (the threshold test of the count tolerates the approximate
            // division's two ulp)
            rmax = fmaxf(rmax, some ? __fdividef(num, D) : 0.0f);
            dmin = fminf(dmin, some ? D : inf);
            hole |= !some & (num > 0.0f);
          }
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acce[buf]);
      }
    }
    for (int off = 16; off; off >>= 1) {
      rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, off));
      dmin = fminf(dmin, __shfl_xor_sync(0xffffffffu, dmin, off));
    }
    hole = __any_sync(0xffffffffu, hole);
    if (lane == 0 && ok) {
      if (hole && P.slices == 1) raise_word(P.est + OZ_W_HOLE, 1);
      if (hole && P.slices != 1) rmax = inf;
      atomicMax(P.est + OZ_W_SPREAD, __float_as_uint(rmax));
      if (dmin < inf) atomicMax(P.est + OZ_W_DROP, __float_as_uint(0x1p96f / dmin));
    }
  } else if (G) {
    // ---------------- grouped epilogue (warps 2..9) ----------------
    // Warp w reads TMEM lane quarter w % 4 (one tile row per thread); the
    // two warps of a quarter take alternate 16-column chunks (half h:
    // chunks h, h+2, h+4, h+6), so narrow problems keep both busy. Chunks
    // right of the problem's n and quarters below its m skip all TMEM work
    // (warp-uniform tests).
    //
    // Exact accumulation without a 128-bit read-modify-write: one int32 per
    // element, R (TMEM columns 256..383), runs over the diagonals from
    // d = S-1 (least significant) to d = 0. Moving from diagonal d+1 to d,
    // R <- floor(R / 2^b) + D_d and the low b bits of the old R are final:
    // digit S-2-d. After d = 0,
    //   T = R 2^(b(S-1)) + sum_t digit_t 2^(bt)
    // is the exact sum of D_d 2^(b(S-1-d)), converted once to f64.
    // |R| < 2^31: |D_d| <= 120 * 2^24 (host limit on K chunks x S) and the
    // carry adds at most |R| / 2^b + 1.
    // Digits are kept one byte each, four to a word per element: digits
    // 0..3 in a register word that moves to TMEM columns 384..511 once full,
    // digits 4..7 in the register word after it, digits 8..14 (S > 9 only)
    // in this CTA's slot of 8-byte records in global memory.
    constexpr int BN = Geo::BN;
    constexpr size_t kColPitch = (size_t)OZ_BM * OZ_DIGIT_BYTES;  // slot bytes per tile column
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row_in_tile = q * 32 + lane;
    const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16);
    const uint32_t dsum_t = lane_base + 2 * BN;  // R
    const uint32_t dig_t = lane_base + 3 * BN;   // digits 0..3
    const int b = B8 ? 8 : P.digit_bits, nd = S - 1;
    const uint32_t dmask = (1u << b) - 1;
    uint8_t* const slot = P.acc + (size_t)blockIdx.x * (kColPitch * BN) +
                          (size_t)row_in_tile * OZ_DIGIT_BYTES;
    uint32_t dreg[BN / 2];  // this thread's digit word per element (chunk i, column e: [i * 16 + e])
    // this warp's column exponents, [i * 16 + e] for chunk i, column e
    int* const sm_eb = reinterpret_cast<int*>(smem + Geo::STAGES * Geo::STAGE_BYTES) + (warp - 2) * 64;
    uint32_t ai = 0;
    bool ok = true;
    for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
      const TileCtx tc = tile_ctx<EST, G>(P, S, tile, rank);
      const int64_t row = tc.row0 + row_in_tile;
      const bool row_ok = row < tc.m;
      const int ncols = (int)(tc.n - tc.col0 < BN ? tc.n - tc.col0 : BN);
      int nch = (ncols - 16 * half + 31) / 32;  // chunks of this warp inside the problem
      if (nch < 0 || tc.row0 + q * 32 >= tc.m) nch = 0;
      const int ecol_base = row_ok ? tc.ea[row] + final_shift : 0;
      // Column exponents of this warp's columns j = lane, lane + 32 (chunk
      // j / 16, column j % 16): loaded now, used by the retire pass at the
      // end of the tile (their latency hides behind the tile's groups).
      int ebj[2];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int j = lane + 32 * t;
        const int64_t col = tc.col0 + (2 * (j >> 4) + half) * 16 + (j & 15);
        ebj[t] = col < tc.n ? tc.eb[col] : 0;
      }
      const int gm = merge_count(tc, P, false);
#pragma unroll
      for (int e = 0; e < BN / 2; ++e) dreg[e] = 0;  // (no value survives a tile)
      PairIter pr;
      pr.start(S);
      int last_buf = 0;
      for (int u = 0; u < tc.n_pairs && ok; ++ai) {
        const int g = group_size(pr, gm, tc.kchunks);
        const int d = pr.d;
        const bool diag_start = pr.diag_first();
        const bool tile_first = u == 0;
        u += g;
        for (int j = 0; j < g; ++j) pr.next(tc.kchunks);
        const bool final_group = u == tc.n_pairs;  // the last group of d = 0
        const int buf = (int)(ai & 1);
        if (!bounded(&accf[buf], (ai >> 1) & 1, 4, std::false_type{})) { ok = false; break; }
        tc_fence_after();
        // Chunk by chunk: the accumulator and R in flight together, R
        // updated and stored back; the accumulator goes back to the MMA warp
        // after the last chunk is read (the other one is in use meanwhile).
        // The conditions are uniform and tested per chunk, not per element
        // (a test per element cost 3,500 of a group's 5,200 cycles).
        const int dig_i = nd - 1 - d;  // digit index of diagonal d + 1
        const bool push = diag_start && !tile_first;
        const int rsh = push ? b : 0;
#pragma unroll
        for (int i = 0; i < BN / 32; ++i) {
          if (i >= nch) continue;
          const int col_t = (2 * i + half) * 16;
          uint32_t v[16], w[16];
          tmem_ld16_nowait(lane_base + buf * BN + col_t, v);
          if (!tile_first) {
            tmem_ld16_nowait(dsum_t + col_t, w);
          } else {
#pragma unroll
            for (int e = 0; e < 16; ++e) w[e] = 0;
          }
          tmem_wait_ld();
          if (push) {
            if (dig_i < 8) {
              // 8-bit digits enter at the top of the word, so that a word
              // that is not full is left-aligned
              if constexpr (B8) {
#pragma unroll
                for (int e = 0; e < 16; ++e) dreg[i * 16 + e] = __funnelshift_r(dreg[i * 16 + e], w[e], 8);
              } else {
                const int dsh = 8 * (dig_i & 3);
#pragma unroll
                for (int e = 0; e < 16; ++e) dreg[i * 16 + e] |= (w[e] & dmask) << dsh;
              }
            } else if (row_ok) {
#pragma unroll
              for (int e = 0; e < 16; ++e)
                if (col_t + e < ncols) slot[(size_t)(col_t + e) * kColPitch + (dig_i - 8)] = (uint8_t)(w[e] & dmask);
            }
          }
#pragma unroll
          for (int e = 0; e < 16; ++e) w[e] = (uint32_t)(((int32_t)w[e] >> rsh) + __float2int_rn(__uint_as_float(v[e])));
          tmem_st16(dsum_t + col_t, w);
          if (push && dig_i == 3) {
            tmem_st16(dig_t + col_t, *reinterpret_cast<const uint32_t(*)[16]>(dreg + i * 16));
#pragma unroll
            for (int e = 0; e < 16; ++e) dreg[i * 16 + e] = 0;
          }
          // The last group parks the register digit word in TMEM for the
          // retire pass below: digits 4..7 in this accumulator's columns
          // (held until then), or digits 0..S-2 in 384..511 when S < 5.
          if (final_group && nd != 4)
            tmem_st16(nd > 4 ? lane_base + buf * BN + col_t : dig_t + col_t,
                      *reinterpret_cast<const uint32_t(*)[16]>(dreg + i * 16));
        }
        if (!final_group) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acce[buf]);
        }
        tmem_wait_st();
        last_buf = buf;
      }
      if (!ok) break;
      // After the last group of d = 0 (whose accumulator is still held): read
      // R and the digit words back, add the digits 8.. of the records,
      // convert, write C, then free the accumulator.
      sm_eb[lane] = ebj[0];
      sm_eb[lane + 32] = ebj[1];
      __syncwarp();
#pragma unroll 1
      for (int i = 0; i < nch; ++i) {
#pragma unroll
        for (int h8 = 0; h8 < 16; h8 += 8) {
          const int col_t = (2 * i + half) * 16 + h8;
          uint32_t w[8], lw[8], hw[8];
          tmem_ld8_nowait(dsum_t + col_t, w);
          tmem_ld8_nowait(dig_t + col_t, lw);
          if (nd > 4) tmem_ld8_nowait(lane_base + last_buf * BN + col_t, hw);
          tmem_wait_ld();
          if (row_ok) {
          // digits 0..7 as retire8 takes them: with 8-bit digits the last
          // word is left-aligned, a full first word follows it
          uint64_t lo[8];
          const int fsh = nd >= 8 || !B8 ? 0 : nd > 4 ? 64 - 8 * nd : 32;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            lo[e] = nd > 4 ? (uint64_t)hw[e] << 32 | (uint64_t)lw[e] << fsh : (uint64_t)lw[e] << fsh;
          }
          const int64_t off = row * tc.ldc + tc.col0 + col_t;
          const uint8_t* rec = slot + (size_t)col_t * kColPitch;
          uint64_t hi[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) hi[e] = 0;
          if (S > 9) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (col_t + e < ncols)
                hi[e] = __ldcg(reinterpret_cast<const unsigned long long*>(rec + (size_t)e * kColPitch));
          }
          if (tc.f32)
            retire8<true, B8>(w, lo, hi, sm_eb + i * 16 + h8, ncols - col_t, b, S, ecol_base, tc.C, off,
                              tc.accumulate);
          else
            retire8<false, B8>(w, lo, hi, sm_eb + i * 16 + h8, ncols - col_t, b, S, ecol_base, tc.C, off,
                               tc.accumulate);
          }
          __syncwarp();  // (the loads above are warp-wide)
        }
      }
      tc_fence_before();
      __syncwarp();  // (also: sm_eb is rewritten by the next tile only after this)
      if (lane == 0) mbar_arrive(&acce[last_buf]);
    }
  } else {
    // ---------------- epilogue of a pair (warps 2..9) ----------------
    // Warp w reads TMEM lane quarter w % 4 (one tile row per thread) and
    // column half (w - 2) / 4 (128 columns). As in the grouped epilogue, one
    // int32 per element, R, carries the exact diagonal sums from d = S-1 to
    // d = 0 (R <- floor(R / 2^b) + D_d); the two accumulators take all of
    // TMEM, so R stays in this thread's registers. The low b bits retire as
    // digit S-2-d: a thread packs its 128 into eight 16-byte stores to the
    // digit's plane of this CTA's slot ([digit][column / 16][row][16]: a
    // warp's store is 512 contiguous bytes), each read once by the retire
    // pass, which transposes the bytes of 8 columns back. (Byte stores into
    // 16-byte records per element: 4096 x 64 x 4096 516 us, 249 us.)
    // After d = 0 each element's exact total R 2^(b(S-1)) + sum_t digit_t
    // 2^(bt) is rounded once to f64.
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row_in_tile = q * 32 + lane;
    const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16) + half * (OZ_BN / 2);
    const int b = B8 ? 8 : P.digit_bits, nd = S - 1;
    constexpr size_t kChunk = (size_t)OZ_BM * 16;        // bytes of 16 columns of a digit
    constexpr size_t kPlane = (size_t)OZ_BM * OZ_BN;      // bytes of a digit
    uint8_t* const slot = P.acc + (size_t)blockIdx.x * (kPlane * 16) +
                          (size_t)(half * (OZ_BN / 32)) * kChunk + (size_t)row_in_tile * 16;
    const uint32_t acce0 = cluster_addr(&acce[0], 0);  // rank 0's barriers
    auto release = [&](int buf) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acce0 + buf * (uint32_t)sizeof(uint64_t));
    };
    uint32_t R[OZ_BN / 2];
    uint32_t ai = 0;
    bool ok = true;
    for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
      const TileCtx tc = tile_ctx<EST, G>(P, S, tile, rank);
      const int64_t row = tc.row0 + row_in_tile;
      const bool row_ok = row < tc.m;
      const int64_t col0 = tc.col0 + half * (OZ_BN / 2);
      const int ncols = (int)(tc.n - col0 < OZ_BN / 2 ? (tc.n - col0 > 0 ? tc.n - col0 : 0) : OZ_BN / 2);
      const int ecol_base = row_ok ? tc.ea[row] + final_shift : 0;
      const int gm = merge_count(tc, P, false);
      PairIter pr;
      pr.start(S);
      int last_buf = 0;
#pragma unroll
      for (int e = 0; e < OZ_BN / 2; ++e) R[e] = 0;
      for (int u = 0; u < tc.n_pairs && ok; ++ai) {
        const int g = group_size(pr, gm, tc.kchunks);
        const int d = pr.d;
        const bool push = pr.diag_first() && u != 0;
        u += g;
        for (int j = 0; j < g; ++j) pr.next(tc.kchunks);
        const int buf = (int)(ai & 1);
        last_buf = buf;
        if (push) {  // digit of diagonal d + 1
          uint8_t* const sp = slot + (size_t)(nd - 1 - d) * kPlane;
          const uint32_t dmask = ((1u << b) - 1) * 0x01010101u;
#pragma unroll
          for (int c = 0; c < OZ_BN / 32; ++c) {
            uint32_t u4[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t* r = R + c * 16 + j * 4;
              u4[j] = __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410) & dmask;
            }
            *reinterpret_cast<uint4*>(sp + c * kChunk) = make_uint4(u4[0], u4[1], u4[2], u4[3]);
          }
#pragma unroll
          for (int e = 0; e < OZ_BN / 2; ++e) R[e] = (uint32_t)((int32_t)R[e] >> b);
        }
        if (!bounded(&accf[buf], (ai >> 1) & 1, 4, std::false_type{})) { ok = false; break; }
        tc_fence_after();
        // 16 columns are folded into R while the next 16 load
        uint32_t v[2][16];
        tmem_ld16_nowait(lane_base + buf * OZ_BN, v[0]);
#pragma unroll
        for (int c = 0; c < OZ_BN / 32; ++c) {
          tmem_wait_ld16(v[c & 1]);
          if (c + 1 < OZ_BN / 32) tmem_ld16_nowait(lane_base + buf * OZ_BN + (c + 1) * 16, v[(c + 1) & 1]);
#pragma unroll
          for (int e = 0; e < 16; ++e) R[c * 16 + e] += (uint32_t)__float2int_rn(__uint_as_float(v[c & 1][e]));
        }
        if (u < tc.n_pairs) release(buf);
      }
      if (!ok) break;
      // The last group's accumulator is still held: R goes through it to the
      // retire pass, which runs as a loop.
#pragma unroll
      for (int c = 0; c < OZ_BN / 32; ++c)
        tmem_st16(lane_base + last_buf * OZ_BN + c * 16, *reinterpret_cast<const uint32_t(*)[16]>(R + c * 16));
      tmem_wait_st();
      const uint32_t dsum_t = lane_base + last_buf * OZ_BN;
      // After the last group of d = 0: R and the digits of 8 columns at a
      // time (loads in flight together), rounded once, written to C.
#pragma unroll 1
      for (int c8 = 0; c8 < OZ_BN / 2; c8 += 8) {
        if (c8 >= ncols) break;  // warp-uniform
        uint32_t w[8];
        uint64_t lo[8], hi[8];
        tmem_ld8_nowait(dsum_t + c8, w);
        const uint8_t* dp = slot + (size_t)(c8 >> 4) * kChunk + (c8 & 8);
        digits8(dp, kPlane, nd, lo);
        if (S > 9) {
          digits8(dp + 8 * kPlane, kPlane, nd - 8, hi);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) hi[e] = 0;
        }
        tmem_wait_ld();
        if (row_ok) {
        if (B8 && nd <= 8) {  // left-aligned; bytes the digits do not reach drop out
#pragma unroll
          for (int e = 0; e < 8; ++e) lo[e] = nd ? lo[e] << (64 - 8 * nd) : 0;
        }
        const int64_t off = row * tc.ldc + col0 + c8;
        if (tc.f32)
          retire8<true, B8>(w, lo, hi, tc.eb + col0 + c8, ncols - c8, b, S, ecol_base, tc.C, off,
                            tc.accumulate);
        else
          retire8<false, B8>(w, lo, hi, tc.eb + col0 + c8, ncols - c8, b, S, ecol_base, tc.C, off,
                             tc.accumulate);
        }
        __syncwarp();  // (the loads above are warp-wide)
      }
      release(last_buf);
    }
  }
  tc_fence_before();
  __syncthreads();
  // (a pair's CTAs reach into each other until both are done)
  if constexpr (PAIR) cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<PAIR>(tmem_base, OZ_TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------
// Scaling exponents and slicing
// ---------------------------------------------------------------------------
constexpr int kColStrip = 256;  // K rows per block of the grouped column maxima

// frexp-style exponent from a max-magnitude bit pattern.
__global__ void exponents_from_bits(const unsigned long long* __restrict__ mx, int64_t n,
                                    int* __restrict__ e) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const unsigned long long b = mx[i];
  e[i] = ((b >> 52) == 0) ? -1021 : (int)(b >> 52) - 1022;
}

// X = round(x * 2^(126 - e)) as a signed 128-bit integer (|x| < 2^e).
template <typename T>
__device__ __forceinline__ __int128 fixed126(T x, int e) {
  bool neg;
  uint64_t mant;
  int E;
  ozaki_decode(x, neg, mant, E);  // |x| = mant 2^E
  const int sh = E + 126 - e;
  __int128 X;
  if (mant == 0) {
    X = 0;
  } else if (sh >= 0) {
    X = (__int128)mant << sh;  // sh <= 73 because |x| < 2^e (102 for a float)
  } else if (sh > -64) {
    X = (__int128)((mant + (1ULL << (-sh - 1))) >> (-sh));
  } else {
    X = 0;
  }
  return neg ? -X : X;
}

// Signed b-bit digits of X at positions p_t = 127 - b - b t, t < S, with
//   sum_t d_t 2^p_t = X rounded to the nearest multiple of 2^p_(S-1) (ties up).
// Z = X + h * sum_t 2^p_t + 2^(p_(S-1) - 1), h = 2^(b-1), makes every b-bit
// field of Z the digit plus h, so each digit is one shift and mask: d_t in
// [-h, h - 1] for t >= 1, the top digit (Z >> p_0) - h in [-h, h]. Every
// digit is exact in BF16 and |d_s d_t| <= 2^(2b-2), as the file header
// requires.
// Z is unsigned: X + C lies in (0, 2^127 + 2^122), beyond the signed range.
__device__ __forceinline__ unsigned __int128 digit_offset(int S, int b) {
  unsigned __int128 c = (unsigned __int128)1 << (kTopOf(b) - b * (S - 1) - 1);
  for (int t = 0; t < S; ++t) c += (unsigned __int128)(1u << (b - 1)) << (kTopOf(b) - b * t);
  return c;
}
// B is a template argument so that every digit position is a constant shift.
template <int B>
__device__ __forceinline__ int digit_at(unsigned __int128 Z, int t) {
  const int p = kTopOf(B) - B * t;
  const int f = (int)(uint32_t)(uint64_t)(Z >> p);
  return (t == 0 ? f : (f & ((1 << B) - 1))) - (1 << (B - 1));
}

__device__ __forceinline__ uint32_t bf16_of_int(int v) {
  // |v| <= 2^(b-1) <= 128: exact in bf16; its fp32 bit pattern's top half.
  return __float_as_uint((float)v) >> 16;
}

// ---------------------------------------------------------------------------
// One problem's operands: exponents, spread-estimate operands, slices
// ---------------------------------------------------------------------------
// One operand as the kernels see it: `rows` output rows (m for A, n for B)
// along K. rows_contig: element (r, kk) at p[r * ld + kk] (A as given, or B
// passed transposed); otherwise at p[kk * ld + r] (B as given, or A passed
// transposed), which is read coalesced along r and transposed through shared
// memory. Each kernel takes both operands in one launch: the first `blocks`
// blocks work on the first operand.
//
// All three kernels stream their operand once and are bound by HBM at large
// sizes; for small products what counts is that they are three launches
// instead of eight (512^3: 0.05 ms -> 0.015 ms of the chain before the
// products).
template <typename T>
struct OzPrep {
  const T* p;
  int64_t ld, rows;
  int rows_contig;
  int vec;            // rows_contig: every row starts 16-byte aligned
  int strips;         // column layout: K strips of the partial maxima
  int64_t strip_len;
  uint32_t* part;     // column layout: [strips][rows] maxima, as abs_bits
  int* e;             // exponents
  uint32_t* sums;     // sum_k |x'| in units of 1 / scale
  uint16_t* out;      // slices (or estimate slices) [S][rows][kpad]
  unsigned blocks;
};

// The bits of |x| that decide its exponent, ordered like |x| up to equal
// exponents: the high word of a double, all of a float.
__device__ __forceinline__ uint32_t abs_bits(double x) { return (uint32_t)__double2hiint(x) & 0x7FFFFFFFu; }
__device__ __forceinline__ uint32_t abs_bits(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }
// frexp-style exponent (|x| < 2^e) of a maximum's abs_bits; a double that is
// zero or subnormal gives -1021, Inf / NaN the value kNonFinite.
template <typename T>
__device__ __forceinline__ int exp_of_bits(uint32_t m) {
  if constexpr (sizeof(T) == 8) {
    const int be = (int)(m >> 20);
    return be == 0 ? -1021 : be - 1022;
  } else {
    const int be = (int)(m >> 23);
    if (be == 0) return m == 0 ? -1021 : -116 - __clz((int)m);  // 2^(31 - clz) 2^-149 <= |x|
    return be - 126;
  }
}
template <typename T>
constexpr int kNonFinite = sizeof(T) == 8 ? 1025 : 129;

// 16 bytes of T (8 doubles' worth of slots are filled by several calls).
template <typename T, int N>
__device__ __forceinline__ void load_run(const T* src, bool vec, int64_t left, T (&x)[N]) {
  constexpr int PER = 16 / (int)sizeof(T);
  if (vec && left >= N) {
#pragma unroll
    for (int q = 0; q < N / PER; ++q) {
      const uint4 u = reinterpret_cast<const uint4*>(src)[q];
      memcpy(&x[q * PER], &u, 16);
    }
  } else {
#pragma unroll
    for (int q = 0; q < N; ++q) x[q] = q < left ? src[q] : T(0);
  }
}

// Exponents of contiguous rows; per-strip maxima of columns. Also zeroes
// the decision words and the column sums that oz_est adds into.
template <typename T>
__global__ void __launch_bounds__(256) oz_max(OzPrep<T> a, OzPrep<T> bT, int64_t k, uint32_t* __restrict__ words) {
  launch_wait();
  launch_next();
  if (blockIdx.x == 0 && threadIdx.x < OZ_WORDS) words[threadIdx.x] = 0;
  const bool first = blockIdx.x < a.blocks;
  const OzPrep<T>& o = first ? a : bT;
  const int64_t blk = first ? blockIdx.x : blockIdx.x - a.blocks;
  if (o.rows_contig) {
    const int64_t row = blk * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= o.rows) return;
    const T* xr = o.p + row * o.ld;
    uint32_t mx = 0;
#pragma unroll 2
    for (int64_t j = lane * 8; j < k; j += 256) {
      T x[8];
      load_run(xr + j, o.vec, k - j, x);
#pragma unroll
      for (int q = 0; q < 8; ++q) mx = max(mx, abs_bits(x[q]));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) o.e[row] = exp_of_bits<T>(mx);
  } else {
    const int64_t nx = (o.rows + 255) / 256;
    const int64_t strip = blk / nx, col = (blk - strip * nx) * 256 + threadIdx.x;
    if (col >= o.rows) return;
    const int64_t r0 = strip * o.strip_len;
    const int64_t r1 = r0 + o.strip_len < k ? r0 + o.strip_len : k;
    uint32_t mx = 0;
#pragma unroll 8
    for (int64_t i = r0; i < r1; ++i) mx = max(mx, abs_bits(o.p[i * o.ld + col]));
    o.part[strip * o.rows + col] = mx;
    if (strip == 0 && o.sums) o.sums[col] = 0;
  }
}

constexpr int kSliceColK = 64, kSliceColN = 32, kSliceColPitch = kSliceColK / 2 + 1;

// The exponents of a block's 32 columns from the strip maxima (a whole block
// of 256 threads); thread `ty * 32 + tx` returns column n0 + tx's. The
// blocks of the first K tile also store them.
template <typename T>
__device__ __forceinline__ int block_col_exps(const OzPrep<T>& o, int64_t n0, bool store, uint32_t (&sh)[8][32]) {
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t nn = n0 + tx;
  uint32_t mx = 0;
  if (nn < o.rows)
    for (int s = ty; s < o.strips; s += 8) mx = max(mx, o.part[(int64_t)s * o.rows + nn]);
  sh[ty][tx] = mx;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 8; ++q) mx = max(mx, sh[q][tx]);
  const int e = exp_of_bits<T>(mx);
  if (store && ty == 0 && nn < o.rows) o.e[nn] = e;
  return e;
}

// ---------------------------------------------------------------------------
// Spread estimate operands
// ---------------------------------------------------------------------------
// For a slice count that follows the operands' spread they are also written
// as two BF16 "slices": slice 0 = |x'| 2^48 (x' = x 2^-e, so |x'| < 1;
// rounded to nearest) and, for the second pass only, slice 1 = 2^48 where
// x != 0, else 0. The 2^48 factors keep products of small |x'| above FP32's
// underflow threshold while every sum over K stays below 2^96 * 2^31 <
// 2^128. Row sums of |x'| (fixed point) give the pass-1 numerator.
constexpr uint32_t kBf16Two48 = 0x5780u;  // 2^48 in BF16

// |x| 2^-e from the bit pattern alone (no FP64 arithmetic: GB300's FP64 pipe
// is slow): *f = |x'| as fp32 (mantissa truncated), return value = |x'| 2^48
// as BF16 (round to nearest even). Subnormal x and values below the formats'
// normal ranges give 0 (the estimate then only grows). `tiny`: x is not 0 and
// 0 here or below 2^-110 (two entries from there on have a product of 2^-124,
// scaled, which fp32 holds).
constexpr int kTinyExp = -110;
// With e's limit, tiny is one comparison of |x|'s bits.
template <typename T>
struct TinyLimit;
template <>
struct TinyLimit<double> {
  uint64_t v;
  __device__ __forceinline__ explicit TinyLimit(int e) : v(((uint64_t)max(1, 1023 + e + kTinyExp) << 52) - 1) {}
};
template <>
struct TinyLimit<float> {
  uint32_t v;
  __device__ __forceinline__ explicit TinyLimit(int e) : v(((uint32_t)max(1, 127 + e + kTinyExp) << 23) - 1) {}
};
__device__ __forceinline__ uint32_t est_bits(double x, int e, TinyLimit<double> lim, float* f, bool& tiny) {
  const uint64_t u = (uint64_t)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFULL;
  const int be = (int)(u >> 52);
  const uint64_t mant = u & 0xFFFFFFFFFFFFFULL;
  const int fe = be - 1023 - e;  // unbiased exponent of |x'| (<= -1)
  tiny |= u - 1 < lim.v;
  if (be == 0) {
    *f = 0.0f;
    return 0u;
  }
  *f = (fe + 127 >= 1) ? __uint_as_float(((uint32_t)(fe + 127) << 23) | (uint32_t)(mant >> 29)) : 0.0f;
  if (fe + 48 + 127 < 1) return 0u;
  uint32_t h = ((uint32_t)(fe + 48 + 127) << 7) | (uint32_t)(mant >> 45);
  const uint64_t rem = mant & ((1ULL << 45) - 1), half = 1ULL << 44;
  if (rem > half || (rem == half && (h & 1u))) ++h;
  return h;
}
__device__ __forceinline__ uint32_t est_bits(float x, int e, TinyLimit<float> lim, float* f, bool& tiny) {
  const uint32_t u = __float_as_uint(x) & 0x7FFFFFFFu;
  const int be = (int)(u >> 23);
  const uint32_t mant = u & 0x7FFFFFu;
  const int fe = be - 127 - e;
  tiny |= u - 1 < lim.v;
  if (be == 0) {
    *f = 0.0f;
    return 0u;
  }
  *f = (fe + 127 >= 1) ? __uint_as_float(((uint32_t)(fe + 127) << 23) | mant) : 0.0f;
  if (fe + 48 + 127 < 1) return 0u;
  uint32_t h = ((uint32_t)(fe + 48 + 127) << 7) | (mant >> 16);
  const uint32_t rem = mant & 0xFFFFu;
  if (rem > 0x8000u || (rem == 0x8000u && (h & 1u))) ++h;
  return h;
}
// 2^48 in BF16 where x is not +-0 (an integer test)
__device__ __forceinline__ uint32_t two48_if(double x) {
  return ((uint64_t)__double_as_longlong(x) << 1) != 0 ? kBf16Two48 : 0u;
}
__device__ __forceinline__ uint32_t two48_if(float x) { return x != 0.0f ? kBf16Two48 : 0u; }

// Both operands' estimate slices, sums and exponent maxima. `kside`: the
// decision word of the operand's exponent maximum.
template <typename T, bool PASS2>
__global__ void __launch_bounds__(256)
    oz_est(OzPrep<T> a, OzPrep<T> bT, int64_t k, int64_t kpad, float scale, uint32_t* __restrict__ words) {
  launch_wait();
  launch_next();
  __shared__ uint32_t tile[PASS2 ? 2 : 1][kSliceColN][kSliceColPitch];
  __shared__ float csum[8][kSliceColN];
  __shared__ uint32_t cexp[8][32];
  const bool first = blockIdx.x < a.blocks;
  const OzPrep<T>& o = first ? a : bT;
  const int64_t blk = first ? blockIdx.x : blockIdx.x - a.blocks;
  const int word = first ? OZ_W_EXP_A : OZ_W_EXP_B;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  if (o.rows_contig) {
    const int64_t row = blk * 8 + ty;
    if (row >= o.rows) return;
    const int er = o.e[row];
    const T* xr = o.p + row * o.ld;
    float s = 0.0f;
    bool tiny = false;
    const TinyLimit<T> lim(er);
    for (int64_t j0 = (int64_t)tx * 8; j0 < kpad; j0 += 256) {
      T x[8];
      load_run(xr + j0, o.vec, k - j0, x);
      uint32_t pa[4], pi[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        float f0, f1;
        const uint32_t b0 = est_bits(x[2 * h], er, lim, &f0, tiny), b1 = est_bits(x[2 * h + 1], er, lim, &f1, tiny);
        s += f0;
        s += f1;
        pa[h] = b0 | (b1 << 16);
        pi[h] = two48_if(x[2 * h]) | (two48_if(x[2 * h + 1]) << 16);
      }
      uint16_t* q = o.out + row * kpad + j0;
      *reinterpret_cast<uint4*>(q) = make_uint4(pa[0], pa[1], pa[2], pa[3]);
      if (PASS2) *reinterpret_cast<uint4*>(q + o.rows * kpad) = make_uint4(pi[0], pi[1], pi[2], pi[3]);
    }
    for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    tiny = __any_sync(0xffffffffu, tiny);
    if (tx == 0) {
      if (tiny) raise_word(&words[OZ_W_TINY], 1);
      o.sums[row] = __float2uint_ru(s * scale);
      raise_word(&words[word], (uint32_t)(er + kExpBias));
      if (er == kNonFinite<T>) words[OZ_W_NONFINITE] = 1;
    }
    return;
  }
  // 64 k x 32 columns, transposed through shared memory (the pad word of a
  // tile row keeps both phases free of bank conflicts)
  const int64_t nx = (o.rows + kSliceColN - 1) / kSliceColN;
  const int64_t ky = blk / nx, n0 = (blk - ky * nx) * kSliceColN, k0 = ky * kSliceColK;
  const int64_t nn = n0 + tx;
  T x0[kSliceColK / 16], x1[kSliceColK / 16];
#pragma unroll
  for (int r = 0; r < kSliceColK / 16; ++r) {  // word column w = ty + 8r: k rows 2w, 2w+1
    const int64_t kk = k0 + 2 * (ty + 8 * r);
    x0[r] = kk < k && nn < o.rows ? o.p[kk * o.ld + nn] : T(0);
    x1[r] = kk + 1 < k && nn < o.rows ? o.p[(kk + 1) * o.ld + nn] : T(0);
  }
  const int ec = block_col_exps(o, n0, ky == 0, cexp);
  float s = 0.0f;
  bool tiny = false;
  const TinyLimit<T> lim(ec);
#pragma unroll
  for (int r = 0; r < kSliceColK / 16; ++r) {
    const int w = ty + 8 * r;
    float f0, f1;
    const uint32_t b0 = est_bits(x0[r], ec, lim, &f0, tiny), b1 = est_bits(x1[r], ec, lim, &f1, tiny);
    s += f0;
    s += f1;
    tile[0][tx][w] = b0 | (b1 << 16);
    if (PASS2) tile[PASS2 ? 1 : 0][tx][w] = two48_if(x0[r]) | (two48_if(x1[r]) << 16);
  }
  csum[ty][tx] = s;
  tiny = __any_sync(0xffffffffu, tiny);
  if (tiny && tx == 0) raise_word(&words[OZ_W_TINY], 1);
  __syncthreads();
  if (ty == 0 && nn < o.rows) {
    float t = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; ++q) t += csum[q][tx];
    atomicAdd(&o.sums[nn], __float2uint_ru(t * scale));  // (integers: any order)
    if (ky == 0) {
      raise_word(&words[word], (uint32_t)(ec + kExpBias));
      if (ec == kNonFinite<T>) words[OZ_W_NONFINITE] = 1;
    }
  }
  const int r = threadIdx.x >> 3, c = threadIdx.x & 7;
  const int64_t n2 = n0 + r, k2 = k0 + c * 8;
  if (n2 < o.rows && k2 < kpad) {
#pragma unroll
    for (int t = 0; t < (PASS2 ? 2 : 1); ++t) {
      const uint32_t* src = &tile[t][r][c * 4];
      *reinterpret_cast<uint4*>(o.out + (int64_t)t * o.rows * kpad + n2 * kpad + k2) =
          make_uint4(src[0], src[1], src[2], src[3]);
    }
  }
}

// The digits of N values at slice t: 64-bit arithmetic when b S <= 64, else
// 128-bit (the same digits).
template <int b, int N>
struct OzDigits64 {
  OzakiZ64 z[N];
  template <typename T>
  __device__ __forceinline__ void set(int i, T x, int e, int S, uint64_t off) { z[i] = ozaki_z64(x, e, b, S, off); }
  __device__ __forceinline__ uint32_t pair(int i, int t) const {
    return bf16_of_int(ozaki_digit64<b>(z[i], t)) | (bf16_of_int(ozaki_digit64<b>(z[i + 1], t)) << 16);
  }
};
template <int b, int N>
struct OzDigits128 {
  unsigned __int128 z[N];
  template <typename T>
  __device__ __forceinline__ void set(int i, T x, int e, int S, unsigned __int128 off) {
    z[i] = (unsigned __int128)fixed126(x, e) + off;
  }
  __device__ __forceinline__ uint32_t pair(int i, int t) const {
    return bf16_of_int(digit_at<b>(z[i], t)) | (bf16_of_int(digit_at<b>(z[i + 1], t)) << 16);
  }
};

// 8 consecutive k of one row -> one 16-byte vector per slice, one slice at a
// time so that only the current slice's packed words are live.
template <typename D, typename T, typename O>
__device__ __forceinline__ void slice_run8(const T (&x)[8], int e, int S, O off, uint16_t* out, int64_t plane) {
  D d;
#pragma unroll
  for (int q = 0; q < 8; ++q) d.set(q, x[q], e, S, off);
#pragma unroll
  for (int t = 0; t < OZ_MAX_SLICES; ++t)
    if (t < S)
      *reinterpret_cast<uint4*>(out + (int64_t)t * plane) =
          make_uint4(d.pair(0, t), d.pair(2, t), d.pair(4, t), d.pair(6, t));
}

// 64 k x 32 columns: thread (tx, ty) holds the k pairs 2 (ty + 8 r), packs
// two digits of a column into one word of a shared tile per slice, and every
// thread writes one 16-byte vector (8 k of one column) per slice; kSliceSet
// slices at a time share the tile.
constexpr int kSliceSet = 8;
template <typename D, typename T, typename O>
__device__ __forceinline__ void slice_tile(const T (&x0)[4], const T (&x1)[4], int e, int S, O off, uint32_t* tile,
                                           uint16_t* out, int64_t rows, int64_t kpad, int64_t n0, int64_t k0) {
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  D d;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    d.set(2 * r, x0[r], e, S, off);
    d.set(2 * r + 1, x1[r], e, S, off);
  }
  const int rr = threadIdx.x >> 3, c = threadIdx.x & 7;  // column, 16-byte chunk (8 k)
  const int64_t nn = n0 + rr, kk = k0 + c * 8;
#pragma unroll
  for (int t0 = 0; t0 < OZ_MAX_SLICES; t0 += kSliceSet) {
    if (t0 >= S) break;
    if (t0) __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int t = t0; t < t0 + kSliceSet; ++t)
        if (t < S) tile[((t - t0) * kSliceColN + tx) * kSliceColPitch + ty + 8 * r] = d.pair(2 * r, t);
    __syncthreads();
    if (nn < rows && kk < kpad) {
#pragma unroll
      for (int t = 0; t < kSliceSet; ++t) {
        if (t0 + t >= S) break;
        const uint32_t* src = tile + (t * kSliceColN + rr) * kSliceColPitch + c * 4;
        *reinterpret_cast<uint4*>(out + (int64_t)(t0 + t) * rows * kpad + nn * kpad + kk) =
            make_uint4(src[0], src[1], src[2], src[3]);
      }
    }
  }
}

// Both operands -> slices [S][rows][kpad], K-major, zero beyond k. S as
// given, or decided on the device (0: nothing to do).
template <typename T, int b>
__global__ void __launch_bounds__(256)
    oz_slice(OzPrep<T> a, OzPrep<T> bT, int64_t k, int64_t kpad, int S_given, uint32_t* decide, OzRule rule) {
  __shared__ uint32_t tile[kSliceSet * kSliceColN * kSliceColPitch];
  __shared__ uint32_t cexp[8][32];
  launch_wait();
  launch_next();
  const int S = decide ? oz_decide(decide, rule) : S_given;
  if (decide && blockIdx.x == 0 && threadIdx.x == 0) decide[OZ_W_COUNT] = (uint32_t)S;
  if (S == 0) return;
  const bool first = blockIdx.x < a.blocks;
  const OzPrep<T>& o = first ? a : bT;
  const int64_t blk = first ? blockIdx.x : blockIdx.x - a.blocks;
  const bool small = b * S <= 64;
  const uint64_t c64 = small ? ozaki_offset64(S, b) : 0;
  const unsigned __int128 c128 = small ? 0 : digit_offset(S, b);
  if (o.rows_contig) {
    const int64_t gpr = kpad / 8, total = o.rows * gpr, plane = o.rows * kpad;
    for (int64_t g = blk * 256 + threadIdx.x; g < total; g += (int64_t)o.blocks * 256) {
      const int64_t i = g / gpr, j0 = (g - i * gpr) * 8;
      T x[8];
      load_run(o.p + i * o.ld + j0, o.vec, k - j0, x);
      uint16_t* out = o.out + i * kpad + j0;
      if (small)
        slice_run8<OzDigits64<b, 8>>(x, o.e[i], S, c64, out, plane);
      else
        slice_run8<OzDigits128<b, 8>>(x, o.e[i], S, c128, out, plane);
    }
    return;
  }
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t nx = (o.rows + kSliceColN - 1) / kSliceColN;
  const int64_t ky = blk / nx, n0 = (blk - ky * nx) * kSliceColN, k0 = ky * kSliceColK;
  const int64_t nn = n0 + tx;
  T x0[4], x1[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int64_t kk = k0 + 2 * (ty + 8 * r);
    x0[r] = kk < k && nn < o.rows ? o.p[kk * o.ld + nn] : T(0);
    x1[r] = kk + 1 < k && nn < o.rows ? o.p[(kk + 1) * o.ld + nn] : T(0);
  }
  const int e = block_col_exps(o, n0, ky == 0, cexp);
  if (small)
    slice_tile<OzDigits64<b, 8>>(x0, x1, e, S, c64, tile, o.out, o.rows, kpad, n0, k0);
  else
    slice_tile<OzDigits128<b, 8>>(x0, x1, e, S, c128, tile, o.out, o.rows, kpad, n0, k0);
}

bool make_slice_map(CUtensorMap* map, const void* base, int64_t kpad, int64_t rows, int S,
                    uint32_t box_rows) {
  auto enc = nrs_get_encode_tiled();
  if (!enc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)kpad, (cuuint64_t)rows, (cuuint64_t)S};
  const cuuint64_t strides[2] = {(cuuint64_t)kpad * 2, (cuuint64_t)(kpad * rows * 2)};
  const cuuint32_t box[3] = {OZ_BK, box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box,
             estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}


// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct OzOperand {
  const void* p;  // double or float
  int64_t ld;
  int64_t rows;
  bool rows_contig;
};

// Device buffers of one problem, carved from one block of scratch memory:
// exponents | sums | strip maxima | decision words, then an area that holds
// the estimate operands first and the slices after the estimate product.
struct OzScratch {
  int *ea, *eb;
  uint32_t *ra, *cb;
  uint32_t *part_a, *part_b;
  uint32_t* words;
  uint16_t* area_a;
  uint16_t* area_b;
  uint8_t* tail;  // `tail_bytes` behind the areas
};
constexpr int kMaxStrips = 32;
inline size_t oz_al(size_t v) { return (v + 1023) & ~size_t(1023); }
// `planes`: BF16 planes per operand that the areas hold.
size_t oz_scratch(int64_t m, int64_t n, int64_t kpad, int planes, size_t tail_bytes, uint8_t* base, OzScratch* o) {
  const size_t mb = oz_al((size_t)m * 4), nb = oz_al((size_t)n * 4);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    uint8_t* q = base + off;
    off += bytes;
    return q;
  };
  OzScratch r;
  r.ea = (int*)take(mb);
  r.eb = (int*)take(nb);
  r.ra = (uint32_t*)take(mb);
  r.cb = (uint32_t*)take(nb);
  r.part_a = (uint32_t*)take(oz_al((size_t)kMaxStrips * m * 4));
  r.part_b = (uint32_t*)take(oz_al((size_t)kMaxStrips * n * 4));
  r.words = (uint32_t*)take(1024);
  r.area_a = (uint16_t*)take(oz_al((size_t)planes * m * kpad * 2));
  r.area_b = (uint16_t*)take(oz_al((size_t)planes * n * kpad * 2));
  r.tail = take(oz_al(tail_bytes));
  if (o) *o = r;
  return off;
}

template <typename T>
OzPrep<T> oz_prep(const OzOperand& o, int64_t k, int* e, uint32_t* part, uint32_t* sums, uint16_t* out) {
  OzPrep<T> q{};
  q.p = static_cast<const T*>(o.p);
  q.ld = o.ld;
  q.rows = o.rows;
  q.rows_contig = o.rows_contig ? 1 : 0;
  q.vec = (reinterpret_cast<uintptr_t>(o.p) & 15) == 0 && (o.ld * sizeof(T)) % 16 == 0;
  // at least 32 K rows per strip, so that small operands still fill the GPU
  q.strips = (int)std::min<int64_t>(kMaxStrips, (k + 31) / 32);
  q.strip_len = (k + q.strips - 1) / q.strips;
  q.part = part;
  q.e = e;
  q.sums = sums;
  q.out = out;
  return q;
}

// Exponents (columns: strip maxima) of both operands; zeroes the words.
template <typename T>
int launch_oz_max(nrs_handle* h, const OzOperand& a, const OzOperand& bT, int64_t k, const OzScratch& w) {
  auto blocks = [](const OzPrep<T>& q) {
    return (unsigned)(q.rows_contig ? (q.rows + 7) / 8 : (q.rows + 255) / 256 * q.strips);
  };
  OzPrep<T> qa = oz_prep<T>(a, k, w.ea, w.part_a, w.ra, w.area_a), qb = oz_prep<T>(bT, k, w.eb, w.part_b, w.cb, w.area_b);
  qa.blocks = blocks(qa);
  qb.blocks = blocks(qb);
  oz_max<T><<<qa.blocks + qb.blocks, 256, 0, h->stream>>>(qa, qb, k, w.words);
  return nrs_after_launch(h, "oz_max");
}

// Scale of the fixed-point sums of up to k values below 1.
float oz_sum_scale(int64_t k) {
  float s = kSumScale;
  while ((double)s * (double)k >= 2147483648.0 && s > 1.0f) s *= 0.5f;
  return s;
}

template <typename T>
int launch_oz_est(nrs_handle* h, const OzOperand& a, const OzOperand& bT, int64_t k, int64_t kpad,
                  const OzScratch& w, bool pass2) {
  auto blocks = [&](const OzPrep<T>& q) {
    return (unsigned)(q.rows_contig ? (q.rows + 7) / 8
                                    : (q.rows + kSliceColN - 1) / kSliceColN * ((kpad + kSliceColK - 1) / kSliceColK));
  };
  OzPrep<T> qa = oz_prep<T>(a, k, w.ea, w.part_a, w.ra, w.area_a), qb = oz_prep<T>(bT, k, w.eb, w.part_b, w.cb, w.area_b);
  qa.blocks = blocks(qa);
  qb.blocks = blocks(qb);
  const float scale = oz_sum_scale(k);
  return nrs_cuda_check(h, nrs_launch_after(true, pass2 ? oz_est<T, true> : oz_est<T, false>, qa.blocks + qb.blocks, 256,
                                            0, h->stream, qa, qb, k, kpad, scale, w.words),
                        "oz_est");
}

// decide != null: the count is decided on the device under `rule`.
template <typename T>
int launch_oz_slice(nrs_handle* h, const OzOperand& a, const OzOperand& bT, int64_t k, int64_t kpad, int b, int S,
                    uint32_t* decide, const OzRule& rule, const OzScratch& w) {
  auto blocks = [&](const OzPrep<T>& q) {
    return (unsigned)(q.rows_contig
                          ? std::min<int64_t>((q.rows * (kpad / 8) + 255) / 256, (int64_t)h->num_sms * 8)
                          : (q.rows + kSliceColN - 1) / kSliceColN * ((kpad + kSliceColK - 1) / kSliceColK));
  };
  OzPrep<T> qa = oz_prep<T>(a, k, w.ea, w.part_a, w.ra, w.area_a), qb = oz_prep<T>(bT, k, w.eb, w.part_b, w.cb, w.area_b);
  qa.blocks = blocks(qa);
  qb.blocks = blocks(qb);
  const unsigned grid = qa.blocks + qb.blocks;
  auto kern = b == 8 ? oz_slice<T, 8> : b == 7 ? oz_slice<T, 7> : oz_slice<T, 6>;
  return nrs_cuda_check(h, nrs_launch_after(true, kern, grid, 256, 0, h->stream, qa, qb, k, kpad, S, decide, rule),
                        "oz_slice");
}

// CTAs of a pair launch (and its digit slots).
int pair_ctas(nrs_handle* h, int64_t tiles) { return 2 * (int)std::max<int64_t>(1, std::min<int64_t>(tiles, h->num_sms / 2)); }

// rows_a / rows_b: rows of the (stacked) slice buffers; P.kpad: their pitch.
template <bool EST, bool G, bool B8>
int launch_tc_b(nrs_handle* h, const void* sa, const void* sb, int S, const OzParams& P, int64_t rows_a,
                int64_t rows_b, cudaStream_t stream) {
  using Geo = OzGeom<EST, G>;
  CUtensorMap mapA, mapB;
  if (!make_slice_map(&mapA, sa, P.kpad, rows_a, S, OZ_BM) ||
      !make_slice_map(&mapB, sb, P.kpad, rows_b, S, Geo::LOAD_N))
    return nrs_fail(h, NRS_ERR_CUDA, "cuTensorMapEncodeTiled failed for the slices");
  // Set on every call: the attribute belongs to the current device's context.
  int st = nrs_cuda_check(h, cudaFuncSetAttribute(ozaki_tc_kernel<EST, G, B8>,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize, Geo::SMEM),
                          "cudaFuncSetAttribute(ozaki)");
  if (st) return st;
  const int n_tiles = P.n_tiles;
  if (n_tiles < 1) return NRS_OK;
  if constexpr (Geo::PAIR) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)pair_ctas(h, n_tiles));
    cfg.blockDim = dim3(OZ_THREADS);
    cfg.dynamicSmemBytes = Geo::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return nrs_cuda_check(h, cudaLaunchKernelEx(&cfg, ozaki_tc_kernel<EST, G, B8>, mapA, mapB, P), "ozaki_tc_kernel");
  }
  const int ctas = n_tiles < h->num_sms ? n_tiles : h->num_sms;
  // In one wave the early start saves ~3 us. CTAs that start early land on
  // whichever SM has room first, which scatters neighbouring tiles over the
  // dies: in several waves that costs more (f32 4096^3 on these tiles: 1.24
  // -> 1.27 ms). Tile lists follow a kernel that
  // does not let them in early.
  const bool after = !P.tiles && n_tiles <= h->num_sms;
  return nrs_cuda_check(h, nrs_launch_after(after, ozaki_tc_kernel<EST, G, B8>, (unsigned)ctas, OZ_THREADS,
                                            Geo::SMEM, stream, mapA, mapB, P),
                        EST ? "ozaki_tc_kernel<est>" : "ozaki_tc_kernel");
}
template <bool EST, bool G>
int launch_tc(nrs_handle* h, const void* sa, const void* sb, int S, const OzParams& P, int64_t rows_a,
              int64_t rows_b, cudaStream_t stream) {
  if (EST || P.digit_bits == 8) return launch_tc_b<EST, G, true>(h, sa, sb, S, P, rows_a, rows_b, stream);
  return launch_tc_b<EST, G, EST>(h, sa, sb, S, P, rows_a, rows_b, stream);
}

OzParams base_params(nrs_handle* h, int64_t m, int64_t n, int64_t k, int64_t kpad) {
  OzParams P{};
  P.m = m;
  P.n = n;
  P.k = k;
  P.kpad = kpad;
  P.tiles_m = (int)((m + OZ_BM - 1) / OZ_BM);
  P.tiles_n = (int)((n + OZ_BN - 1) / OZ_BN);
  P.group_m = 12;
  P.n_tiles = P.tiles_m * P.tiles_n;
  P.splits = 1;
  P.split_blocks = (int)((kpad + OZ_BK - 1) / OZ_BK);
  P.err = h->dev_error;
  return P;
}

// Elements between the rows of a slice: TMA needs multiples of 8; from 256 on
// of 64, so that the 128-byte rows of its boxes do not straddle sectors and
// lines (f64 5000^3: 6.82 ms with rows of 10000 bytes, 4.95 of 10112;
// 1999 x 1537 x 3001: 0.73 and 0.56). The
// pad is zero, and within the 64-wide K block that is computed anyway.
int64_t slice_pitch(int64_t k) { return k < 256 ? (k + 7) / 8 * 8 : (k + 63) / 64 * 64; }

// Limits of b-bit digits with S slices over kpad: S <= 16, every digit
// inside the 126 fraction bits (b S <= 126), int32-exact diagonal sums (at
// most kc S K-chunk sums of |x| <= 2^24 each, kc = ceil(kpad / 2^(26-2b)):
// kc S <= 127 for one problem, <= 120 for grouped launches, whose carried
// sums need the headroom), and the exact total inside a signed 128-bit
// integer (|total| < 2^(31 + b(S-1)) with b(S-1) <= 95).
constexpr int64_t kMaxChunkSlices = 127;
constexpr int64_t kMaxChunkSlicesGrouped = 120;
bool digits_fit(int b, int S, int64_t kpad, int64_t max_kcs) {
  const int64_t kc = std::max<int64_t>(1, (kpad + kChunkOf(b) - 1) / kChunkOf(b));
  return S >= 1 && S <= OZ_MAX_SLICES && b * S <= 126 && b * (S - 1) <= 95 && kc * S <= max_kcs;
}

// What a call's operands ask of a slice count (ozaki_count_holds): the bits
// that the spread needs and, for the pairs left out, target + log2 drop.
struct OzNeed {
  double bits, drop_bits;
};

// The least count for digits of b bits.
int slices_for(int b, const OzNeed& need) {
  int S = std::max(1, (int)std::ceil(need.bits / b - 1e-9));
  while (S <= OZ_MAX_SLICES && S > 1 && b * S < need.drop_bits + std::log2((double)(S - 1))) ++S;
  return S;
}

// Digit width and count: the widest b (8, 7, 6) whose least count is inside
// digits_fit's limits. false if no width qualifies.
bool choose_digits(int64_t kpad, const OzNeed& need, int* b, int* S, int* kchunks,
                   int64_t max_kcs = kMaxChunkSlices) {
  for (int cand = 8; cand >= 6; --cand) {
    const int s_c = slices_for(cand, need);
    const int64_t kc = (kpad + kChunkOf(cand) - 1) / kChunkOf(cand);
    if (digits_fit(cand, s_c, kpad, max_kcs)) {
      *b = cand;
      *S = s_c;
      *kchunks = (int)kc;
      return true;
    }
  }
  return false;
}

// Bits of the fixed-point operands that keep their rounding at FP64's unit
// roundoff relative to (|A||B|)_ij: bS >= 53 + log2 max_ij R_ij; 26 (24 and two
// guard bits) for f32.
constexpr int kTargetBits = 53, kTargetBits32 = 26;

struct SpreadResult {
  float rmax;
  uint32_t flags;  // bit 0: an operand holds Inf or NaN
  float dinv;      // 1 / the smallest nonzero (|A'||B'|)_ij
  bool finite() const { return std::isfinite((double)rmax) && std::isfinite((double)dinv); }
  OzNeed need(int target, int64_t k) const {
    const double drop = (double)dinv * (double)k / ozaki_drop_units_asked(target, (double)k);
    return OzNeed{target + (rmax > 1.0f ? std::log2((double)rmax) : 0.0), drop > 0.0 ? target + std::log2(drop) : 0.0};
  }
};

// Enqueues the spread estimate: exponents, estimate operands and one (pass
// 1) or three (pass 2) BF16 products into the decision words.
template <typename T>
int launch_estimate(nrs_handle* h, const OzOperand& a, const OzOperand& bT, int64_t m, int64_t n, int64_t k,
                    int64_t kpad, int pass, const OzScratch& w) {
  int st;
  if ((st = launch_oz_max<T>(h, a, bT, k, w))) return st;
  if ((st = launch_oz_est<T>(h, a, bT, k, kpad, w, pass == 2))) return st;
  OzParams P = base_params(h, m, n, k, kpad);
  P.slices = pass;
  P.kchunks = 1;
  P.n_pairs = pass == 1 ? 1 : 3;
  P.kchunk = (int)(((kpad + OZ_BK - 1) / OZ_BK) * OZ_BK);
  P.ra = w.ra;
  P.cb = w.cb;
  P.sum_unit = 1.0f / oz_sum_scale(k);
  P.est = w.words;
  return launch_tc<true, false>(h, w.area_a, w.area_b, pass, P, m, n, h->stream);
}

// The estimate with its result read back (one stream synchronisation).
int spread_estimate(nrs_handle* h, const OzOperand& a, const OzOperand& bT, bool f32, int64_t m, int64_t n, int64_t k,
                    int64_t kpad, int pass, SpreadResult* res) {
  int st;
  OzScratch w;
  uint8_t* ws = (uint8_t*)nrs_workspace(h, oz_scratch(m, n, kpad, pass, 0, nullptr, nullptr), &st);
  if (!ws) return st;
  oz_scratch(m, n, kpad, pass, 0, ws, &w);
  st = f32 ? launch_estimate<float>(h, a, bT, m, n, k, kpad, pass, w)
           : launch_estimate<double>(h, a, bT, m, n, k, kpad, pass, w);
  if (st) return st;
  cudaStream_t s = h->stream;
  uint32_t host[4] = {0, 0, 0, 0};
  static_assert(OZ_W_SPREAD == 0 && OZ_W_NONFINITE == 1 && OZ_W_DROP == 2 && OZ_W_HOLE == 3, "the words read back");
  if ((st = nrs_cuda_check(h, cudaMemcpyAsync(host, w.words, sizeof(host), cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync")))
    return st;
  if ((st = nrs_cuda_check(h, cudaStreamSynchronize(s), "cudaStreamSynchronize"))) return st;
  uint32_t derr = 0;
  if ((st = nrs_cuda_check(h, cudaMemcpy(&derr, h->dev_error, 4, cudaMemcpyDeviceToHost), "cudaMemcpy")))
    return st;
  if (derr) return nrs_fail(h, NRS_ERR_TIMEOUT, "ozaki spread estimate: a device-side bounded wait gave up");
  std::memcpy(&res->rmax, &host[OZ_W_SPREAD], 4);
  if (pass == 1 && host[OZ_W_HOLE]) res->rmax = HUGE_VALF;  // pass 2 counts only the k of nonzero products
  std::memcpy(&res->dinv, &host[OZ_W_DROP], 4);
  res->flags = host[OZ_W_NONFINITE];
  return NRS_OK;
}

// One problem runs either on CTA pairs with 256 x 256 tiles (the least panel
// traffic per flop) or on the grouped 128 x 128 geometry, either with K split
// into ranges whose f64 products are added in order, which fills the GPU at
// small sizes.
struct TcPlan {
  bool pair;
  int splits, split_blocks;
  double us;
};

// The form with the least modelled time (us). A 64-wide K block of one slice
// pair takes 0.22 us on a 128 x 128 tile and 0.34 us on a pair's 256 x 256
// one; a tile's fold and rounding 30 and 40 us; the ranges' slabs move at 3
// TB/s. Measured whole calls, us (128 x 128 tiles in 1, 2, 4 ranges / pairs in
// 1, 2, 4): f64 512^3 96, 79, 72 / 129, 103, 92; 1024^3 161, 134, 155 / 211,
// 163, 146; 1536^3 252, 276, 315 / 333, 244, 288; 2048^3 504, 547, 557 / 405,
// 458, 531; 4096^3 3006, 3088, - / 2544, 2524, -; 1024 x 8192 x 1024 981, 660,
// 682 / 1258, 796, 581; f32 2048^3 252, 305 / 223, 274.
TcPlan plan_tc(int64_t m, int64_t n, int64_t kpad, int S, int max_splits) {
  const double pairs = 0.5 * S * (S + 1);
  const int kb = (int)((kpad + OZ_BK - 1) / OZ_BK);
  const int64_t t128 = (m + 127) / 128 * ((n + 127) / 128), t256 = (m + 255) / 256 * ((n + 255) / 256);
  auto waves = [](int64_t tiles, int64_t at_once) { return (double)((tiles + at_once - 1) / at_once); };
  TcPlan best{true, 0, 0, 0.0};
  for (int z = 1; z <= max_splits && z <= kb; ++z) {
    const int blocks = (kb + z - 1) / z;
    const int splits = (kb + blocks - 1) / blocks;
    if (splits != z || (z > 1 && (double)z * (double)(m * n) * 8.0 > 256.0 * (1 << 20))) continue;
    const double join = z > 1 ? 3.0 + (double)z * (double)(m * n) * 8.0 / 3e6 : 0.0;
    const double one = waves(t128 * z, NRS_PLAN_SMS) * (pairs * blocks * 0.22 + 30.0) + join;
    const double two = waves(t256 * z, NRS_PLAN_SMS / 2) * (pairs * blocks * 0.34 + 40.0) + join;
    if (!best.splits || two < best.us) best = TcPlan{true, splits, blocks, two};
    if (one < best.us) best = TcPlan{false, splits, blocks, one};
  }
  return best;
}

// Digit slots of the slice products: a pair launch 16 bytes per element and
// CTA, the grouped geometry 8 (used beyond 9 slices).
size_t oz_slot_bytes(nrs_handle* h, const TcPlan& pl, int64_t m, int64_t n) {
  if (pl.pair) return (size_t)pair_ctas(h, (m + 255) / 256 * ((n + 255) / 256) * pl.splits) * OZ_BM * OZ_BN * 16;
  return (size_t)h->hw_sms * OZ_BM * OzGeom<false, true>::BN * OZ_DIGIT_BYTES;
}

// The slice products of one problem in the planned form (P from base_params).
int launch_products(nrs_handle* h, const TcPlan& pl, int S, OzParams P, const OzScratch& w) {
  using Pair = OzGeom<false, false>;
  const int bm = pl.pair ? Pair::BM : OZ_BM, bn = pl.pair ? Pair::BN : OzGeom<false, true>::BN;
  P.tiles_m = (int)((P.m + bm - 1) / bm);
  P.tiles_n = (int)((P.n + bn - 1) / bn);
  P.group_m = pl.pair ? 8 : 12;
  P.splits = pl.splits;
  P.split_blocks = pl.split_blocks;
  P.n_tiles = P.tiles_m * P.tiles_n * pl.splits;
  return pl.pair ? launch_tc<false, false>(h, w.area_a, w.area_b, S, P, P.m, P.n, h->stream)
                 : launch_tc<false, true>(h, w.area_a, w.area_b, S, P, P.m, P.n, h->stream);
}

int ozaki_run(nrs_handle* h, const OzOperand& a, const OzOperand& bT, int64_t m, int64_t n, int64_t k,
              int64_t kpad, int b, int S, double* C, int64_t ldc, bool accumulate) {
  int st;
  OzScratch w;
  TcPlan pl = plan_tc(m, n, kpad, S, 1);
  if (!digits_fit(b, S, kpad, kMaxChunkSlicesGrouped)) pl.pair = true;
  const size_t slots = oz_slot_bytes(h, pl, m, n);
  uint8_t* ws = (uint8_t*)nrs_workspace(h, oz_scratch(m, n, kpad, S, slots, nullptr, nullptr), &st);
  if (!ws) return st;
  oz_scratch(m, n, kpad, S, slots, ws, &w);
  if ((st = launch_oz_max<double>(h, a, bT, k, w))) return st;
  if ((st = launch_oz_slice<double>(h, a, bT, k, kpad, b, S, nullptr, OzRule{}, w))) return st;
  OzParams P = base_params(h, m, n, k, kpad);
  P.slices = S;
  P.ea = w.ea;
  P.eb = w.eb;
  P.acc = w.tail;
  P.C = C;
  P.ldc = ldc;
  P.digit_bits = b;
  P.kchunk = kChunkOf(b);
  P.accumulate = accumulate ? 1 : 0;
  return launch_products(h, pl, S, P, w);
}

// ---------------------------------------------------------------------------
// Plain GEMM calls on the tensor cores
// ---------------------------------------------------------------------------
// The slice GEMM as the everyday form of C = A*B: the slice count follows the
// operands' spread as in nrs_gemm_ozaki, but it is decided on the device, so
// the call neither synchronises nor copies anything back. The launches:
// oz_max, oz_est, the estimate product, oz_slice (decides), the slice
// products, and the plain FP64 / FP32 kernel, whose blocks return at once
// unless the count is 0 (Inf / NaN operands, sums that could overflow, or a
// spread beyond the slice limit).
// The most slices, whose planes the scratch always holds (2 bytes per operand
// element each). f32: 9 slices are 45 products, and the FP32 kernel is as fast
// (2048^3 573 us against 513, 4096^3 3.9 ms against 3.7).
template <typename T>
constexpr int kAutoMaxSlices = sizeof(T) == 8 ? 12 : 8;

template <typename T>
int tc_gemm(nrs_handle* h, const OzOperand& a, const OzOperand& bT, int64_t m, int64_t k, int64_t n, void* C,
            int64_t ldc, bool accumulate) {
  constexpr bool F32 = sizeof(T) == 4;
  const int64_t kpad = slice_pitch(k);
  // 8-bit digits up to K = 10240 (f32 15360), then 7-bit (exact int32 diagonal
  // sums for every count up to the limit)
  constexpr int most = kAutoMaxSlices<T>;
  const int b = digits_fit(8, most, kpad, kMaxChunkSlicesGrouped) ? 8 : 7;
  if (!digits_fit(b, most, kpad, kMaxChunkSlicesGrouped)) return NRS_ERR_UNSUPPORTED;
  int klog = 0;
  while (((int64_t)1 << klog) < k) ++klog;
  constexpr int target = F32 ? kTargetBits32 : kTargetBits;
  const OzRule rule{target, b, most, (float)((double)k / ozaki_drop_units(target)), (F32 ? 127 : 1023) - klog - 1};
  const TcPlan pl = plan_tc(m, n, kpad, F32 ? 4 : 7, 16);
  const int plain_splits = F32 ? 1 : nrs_dmma_splits(m, k, n);
  const int slabs = std::max(pl.splits > 1 ? pl.splits : 0, plain_splits > 1 ? plain_splits : 0);
  // Behind the slices: the digit slots, then the partial slabs.
  const size_t slots = oz_al(oz_slot_bytes(h, pl, m, n));
  const size_t tail = slots + (size_t)slabs * (size_t)(m * n) * 8;
  cudaStream_t s = h->stream;
  const size_t bytes = oz_scratch(m, n, kpad, most, tail, nullptr, nullptr);
  void* ws = nullptr;
  if (cudaMallocFromPoolAsync(&ws, bytes, h->pool, s) != cudaSuccess) {
    cudaGetLastError();  // no room: the plain kernel needs none
    return NRS_ERR_UNSUPPORTED;
  }
  OzScratch w;
  oz_scratch(m, n, kpad, most, tail, (uint8_t*)ws, &w);
  double* const slab = reinterpret_cast<double*>(w.tail + slots);
  auto run = [&]() -> int {
    int st;
    if ((st = launch_estimate<T>(h, a, bT, m, n, k, kpad, 1, w))) return st;
    if ((st = launch_oz_slice<T>(h, a, bT, k, kpad, b, 0, w.words, rule, w))) return st;
    OzParams P = base_params(h, m, n, k, kpad);
    P.count = w.words + OZ_W_COUNT;
    P.ea = w.ea;
    P.eb = w.eb;
    P.acc = w.tail;
    P.C = pl.splits > 1 ? slab : static_cast<double*>(C);
    P.ldc = ldc;
    P.digit_bits = b;
    P.kchunk = kChunkOf(b);
    P.accumulate = accumulate ? 1 : 0;
    P.f32 = F32 ? 1 : 0;
    st = launch_products(h, pl, most, P, w);
    if (st) return st;
    const int64_t rsa = a.rows_contig ? a.ld : 1, csa = a.rows_contig ? 1 : a.ld;
    const int64_t rsb = bT.rows_contig ? 1 : bT.ld, csb = bT.rows_contig ? bT.ld : 1;
    return nrs_plain_gemm_unless(h, F32 ? NRS_F32 : NRS_F64, m, k, n, a.p, rsa, csa, bT.p, rsb, csb, C, ldc,
                                 accumulate, P.count, slab, pl.splits);
  };
  const int st = run();
  cudaFreeAsync(ws, s);
  return st;
}

// ---------------------------------------------------------------------------
// Grouped launch: many f64 problems in one pass of each kernel
// ---------------------------------------------------------------------------
// The problems' slices are stacked: problem p owns rows [rowoff, rowoff + m)
// of the A slices and [coloff, coloff + n) of the B^T slices, all with the
// group's pitch KP (the largest kpad, a multiple of 64); columns [k, kpad) of
// its rows are zero and columns beyond its kpad are never read. One launch
// of each pre-processing kernel covers every problem through a chunk table,
// and one persistent tensor-core launch covers every tile.
struct OzIn {
  const void* A;  // double or float, as the group's element type T
  int64_t lda;
  const void* B;
  int64_t ldb;
  int64_t m, n, k, kpad;
  int64_t rowoff, coloff;
};
struct OzChunk {
  int32_t prob, r0, k0, pad;  // problem, first row (column), first k
};

// The high word of |x| as a double, whose top bits are the exponent (T: double
// or float, the group's element type; floats widen exactly).
template <typename T>
__device__ __forceinline__ uint32_t g_high_bits(T x) {
  return (uint32_t)__double2hiint((double)x) & 0x7FFFFFFFu;
}

// Column maxima of every B: 32 columns x 256 k per block, 8 threads per column
// (2048 problems of 16..512: 85 us with 256-column blocks, half of whose
// threads had no column, 70 so), atomicMax into a zeroed array.
template <typename T>
__global__ void __launch_bounds__(256)
    g_col_max_bits(const OzIn* __restrict__ in, const OzChunk* __restrict__ ch, unsigned long long* __restrict__ colmax) {
  __shared__ uint32_t part[8][32];
  const OzChunk c = ch[blockIdx.x];
  const OzIn q = in[c.prob];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t col = (int64_t)c.r0 + tx;
  const int64_t r1 = (c.k0 + kColStrip) < q.k ? (c.k0 + kColStrip) : q.k;
  uint32_t mx = 0;
  if (col < q.n) {
    const T* p = static_cast<const T*>(q.B) + col;
#pragma unroll 8
    for (int64_t i = c.k0 + ty; i < r1; i += 8) mx = max(mx, g_high_bits(p[i * q.ldb]));
  }
  part[ty][tx] = mx;
  __syncthreads();
  if (ty == 0 && col < q.n) {
#pragma unroll
    for (int r = 1; r < 8; ++r) mx = max(mx, part[r][tx]);
    atomicMax(&colmax[q.coloff + col], (unsigned long long)mx << 32);
  }
}

// Row exponents and slices of every A: a block takes 8 rows of one problem.
// Each warp finds two rows' exponents; then a thread slices 8 consecutive k of
// one row (zero beyond k, up to the problem's kpad), whose second read hits
// the caches. A block's chain of dependent loads (chunk, problem, row, slices)
// bounds it, so blocks are small and nine fit an SM. (2048 problems of 16..512:
// 97 + 263 us with the exponents in their own launch, 357 fused in blocks of
// 256 threads, 261 in blocks of 128.)
template <typename T, int b, bool SMALL>
__global__ void __launch_bounds__(128)
    g_slice_rows(const OzIn* __restrict__ in, const OzChunk* __restrict__ ch, int* __restrict__ ea, int S,
                 int64_t pitch, int64_t plane, uint16_t* __restrict__ out) {
  __shared__ int row_e[8];
  const OzChunk c = ch[blockIdx.x];
  const OzIn q = in[c.prob];
  const T* const Aq = static_cast<const T*>(q.A) + (int64_t)c.r0 * q.lda;
  {
    const int r = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool ok[2] = {c.r0 + r < q.m, c.r0 + r + 4 < q.m};
    uint32_t mx[2] = {0, 0};
#pragma unroll 4
    for (int64_t j = lane; j < q.k; j += 32) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (ok[i]) mx[i] = max(mx[i], g_high_bits(Aq[(r + 4 * i) * q.lda + j]));
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t m = __reduce_max_sync(0xffffffffu, mx[i]);
      if (lane == 0 && ok[i]) {
        const int e = (m >> 20) == 0 ? -1021 : (int)(m >> 20) - 1022;
        row_e[r + 4 * i] = e;
        ea[q.rowoff + c.r0 + r + 4 * i] = e;
      }
    }
  }
  __syncthreads();
  const bool vec = (reinterpret_cast<uintptr_t>(q.A) & 15) == 0 && (q.lda * sizeof(T)) % 16 == 0;
  const uint32_t groups = (uint32_t)(q.kpad / 8);
  const unsigned __int128 C = digit_offset(S, b);
  const uint64_t C64 = ozaki_offset64(S, b);
  for (uint32_t w = threadIdx.x; w < 8 * groups; w += blockDim.x) {
    const uint32_t r = w / groups;
    const int64_t row = (int64_t)c.r0 + r, j0 = (int64_t)(w - r * groups) * 8;
    if (row >= q.m) break;  // w only grows: every later item is beyond m too
    const int e = row_e[r];
    T x[8];
    load_run(Aq + r * q.lda + j0, vec, q.k - j0, x);
    uint16_t* o = out + (q.rowoff + row) * pitch + j0;
    if constexpr (SMALL) {
      OzakiZ64 Z[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) Z[t] = ozaki_z64(x[t], e, b, S, C64);
#pragma unroll
      for (int t = 0; t < OZ_MAX_SLICES; ++t) {
        if (t < S) {
          uint32_t pk[4];
#pragma unroll
          for (int hh = 0; hh < 4; ++hh)
            pk[hh] = bf16_of_int(ozaki_digit64<b>(Z[2 * hh], t)) |
                     (bf16_of_int(ozaki_digit64<b>(Z[2 * hh + 1], t)) << 16);
          *reinterpret_cast<uint4*>(o + (int64_t)t * plane) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        }
      }
    } else {
      unsigned __int128 Z[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) Z[t] = (unsigned __int128)fixed126(x[t], e) + C;
#pragma unroll
      for (int t = 0; t < OZ_MAX_SLICES; ++t) {
        if (t < S) {
          uint32_t pk[4];
#pragma unroll
          for (int hh = 0; hh < 4; ++hh)
            pk[hh] = bf16_of_int(digit_at<b>(Z[2 * hh], t)) | (bf16_of_int(digit_at<b>(Z[2 * hh + 1], t)) << 16);
          *reinterpret_cast<uint4*>(o + (int64_t)t * plane) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        }
      }
    }
  }
}

// B^T slices of every problem: slice_cols' 64 k x 32 n transposing tile.
template <typename T, int b, bool SMALL>
__global__ void __launch_bounds__(256)
    g_slice_cols(const OzIn* __restrict__ in, const OzChunk* __restrict__ ch, const int* __restrict__ eb, int S,
                 int64_t pitch, int64_t plane, uint16_t* __restrict__ out) {
  extern __shared__ uint32_t tile[];  // [S][32][33]
  const OzChunk c = ch[blockIdx.x];
  const OzIn q = in[c.prob];
  const int64_t k0 = c.k0, n0 = c.r0;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const unsigned __int128 C = digit_offset(S, b);
  const uint64_t C64 = ozaki_offset64(S, b);
  const T* const Bq = static_cast<const T*>(q.B);
  {
    const int64_t nn = n0 + tx;
    const int e = nn < q.n ? eb[q.coloff + nn] : 0;
#pragma unroll
    for (int r = 0; r < kSliceColK / 16; ++r) {
      const int w = ty + 8 * r;
      const int64_t kk = k0 + 2 * w;
      const T x0 = kk < q.k && nn < q.n ? Bq[kk * q.ldb + nn] : T(0);
      const T x1 = kk + 1 < q.k && nn < q.n ? Bq[(kk + 1) * q.ldb + nn] : T(0);
      if constexpr (SMALL) {
        const OzakiZ64 Z0 = ozaki_z64(x0, e, b, S, C64), Z1 = ozaki_z64(x1, e, b, S, C64);
#pragma unroll
        for (int t = 0; t < OZ_MAX_SLICES; ++t)
          if (t < S)
            tile[(t * kSliceColN + tx) * kSliceColPitch + w] =
                bf16_of_int(ozaki_digit64<b>(Z0, t)) | (bf16_of_int(ozaki_digit64<b>(Z1, t)) << 16);
      } else {
        const unsigned __int128 Z0 = (unsigned __int128)fixed126(x0, e) + C;
        const unsigned __int128 Z1 = (unsigned __int128)fixed126(x1, e) + C;
#pragma unroll
        for (int t = 0; t < OZ_MAX_SLICES; ++t)
          if (t < S)
            tile[(t * kSliceColN + tx) * kSliceColPitch + w] =
                bf16_of_int(digit_at<b>(Z0, t)) | (bf16_of_int(digit_at<b>(Z1, t)) << 16);
      }
    }
  }
  __syncthreads();
  const int r = threadIdx.x >> 3, cc = threadIdx.x & 7;
  const int64_t nn = n0 + r, kk = k0 + cc * 8;
  if (nn < q.n && kk < q.kpad) {
    for (int t = 0; t < S; ++t) {
      const uint32_t* src = tile + (t * kSliceColN + r) * kSliceColPitch + cc * 4;
      *reinterpret_cast<uint4*>(out + (int64_t)t * plane + (q.coloff + nn) * pitch + kk) =
          make_uint4(src[0], src[1], src[2], src[3]);
    }
  }
}

}  // namespace

// f64 and f32 GEMMs for which the slice GEMM is the faster form; NRS_ERR_UNSUPPORTED:
// not one of them (nothing was enqueued). The rule compares both forms'
// modelled times: the FP64 tensor path's 1.05 TFLOP/s on 32-wide tiles
// against plan_tc's. Both sides measured (us, DMMA / slices): 256^3 47 / 62,
// 384^3 124 / 65, 512^3 279 / 70, 1024^3 1983 / 130, 2048^3 15661 / 405,
// 4096^3 124903 / 2560, 3000 x 2000 x 10 379 / 148, 64 x 4096 x 64 91 / 100.
// f32 against the FP32 kernels (us): 1024^3 77 / 90, 1280^3 155 / 112,
// 1536^3 184 / 134, 2048^3 418 / 222, 4096^3 3214 / 1120 (error 4e-9 of
// (|A||B|)_ij against the FMA chains' 3e-7).
bool nrs_tc_gemm_pays(int dtype, int64_t m, int64_t k, int64_t n) {
  if (dtype != NRS_F64 && dtype != NRS_F32) return false;
  const bool f32 = dtype == NRS_F32;
  if (m > (1LL << 24) || n > (1LL << 24) || k > (1LL << 24)) return false;
  const double mk = (double)m * k, kn = (double)k * n;
  const double plain_us = f32 ? nrs_plain_f32_us(m, k, n)
                              : (double)((m + 31) / 32 * 32) * (double)((n + 31) / 32 * 32) * (double)k * 2.0 / 1.05e6 + 10.0;
  if (plain_us < 60.0) return false;
  // exponents, estimate, slicing: six launches, 40 (f32: 16) bytes per
  // operand element
  const int S = f32 ? 4 : 7;
  const double tc_us = 30.0 + (mk + kn) * (f32 ? 16.0 : 40.0) / 3e6 +
                       plan_tc(m, n, slice_pitch(k), S, 16).us * (1.0 + 2.0 / (S * (S + 1)));
  return tc_us <= 0.9 * plain_us;
}

int nrs_tc_gemm_auto(nrs_handle* h, int dtype, int64_t m, int64_t k, int64_t n, const void* A, int64_t lda, bool ta,
                     const void* B, int64_t ldb, bool tb, void* C, int64_t ldc, bool accumulate) {
  if (!h->pool || !nrs_tc_gemm_pays(dtype, m, k, n)) return NRS_ERR_UNSUPPORTED;
  // Under stream capture the plain kernel runs, as its launches hold no
  // allocation.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(h->stream, &cap) != cudaSuccess) {
    cudaGetLastError();
    return NRS_ERR_UNSUPPORTED;
  }
  if (cap != cudaStreamCaptureStatusNone) return NRS_ERR_UNSUPPORTED;
  // A workspace cannot grow during a capture: a call outside one leaves the
  // room that the FP64 kernel's K ranges take when the same call is captured
  // (no room: only that capture is refused).
  const int splits = dtype == NRS_F64 ? nrs_dmma_splits(m, k, n) : 1;
  if (splits > 1) {
    int st;
    if (!nrs_workspace(h, (size_t)splits * (size_t)(m * n) * sizeof(double), &st)) h->last_error.clear();
  }
  const OzOperand a{A, lda, m, !ta};
  const OzOperand bT{B, ldb, n, tb};
  return dtype == NRS_F32 ? tc_gemm<float>(h, a, bT, m, k, n, C, ldc, accumulate)
             : tc_gemm<double>(h, a, bT, m, k, n, C, ldc, accumulate);
}

extern "C" int nrs_gemm_ozaki(nrs_handle* h, int64_t m, int64_t k, int64_t n, const double* A,
                              int64_t lda, const double* B, int64_t ldb, double* C, int64_t ldc,
                              unsigned flags, int slices, nrs_ozaki_info* info) {
  if (!h) return NRS_ERR_INVALID;
  h->last_error.clear();
  if (m < 0 || k < 0 || n < 0) return nrs_fail(h, NRS_ERR_SHAPE, "negative GEMM dimension");
  if (flags & ~(NRS_GEMM_ACCUMULATE | NRS_GEMM_TRANS_A | NRS_GEMM_TRANS_B))
    return nrs_fail(h, NRS_ERR_INVALID, "unknown GEMM flag");
  const bool ta = flags & NRS_GEMM_TRANS_A, tb = flags & NRS_GEMM_TRANS_B;
  const bool accumulate = flags & NRS_GEMM_ACCUMULATE;
  if (ldc < (n > 0 ? n : 1)) return nrs_fail(h, NRS_ERR_SHAPE, "ldc < n");
  if (lda < ((ta ? m : k) > 0 ? (ta ? m : k) : 1)) return nrs_fail(h, NRS_ERR_SHAPE, "lda too small");
  if (ldb < ((tb ? k : n) > 0 ? (tb ? k : n) : 1)) return nrs_fail(h, NRS_ERR_SHAPE, "ldb too small");
  if (slices < 0 || slices > OZ_MAX_SLICES)
    return nrs_fail(h, NRS_ERR_INVALID, "slices must be 0 (auto) or 1..16");
  const int64_t kpad = slice_pitch(k);
  if (info) std::memset(info, 0, sizeof(*info));
  int b = 0, S = 0, kchunks = 0;
  if (slices > 0) {
    // Widest digits whose int32 diagonal sums stay exact for this K and S.
    for (int cand = 8; cand >= 6 && !b; --cand) {
      const int kc = (int)((kpad + kChunkOf(cand) - 1) / kChunkOf(cand));
      if (digits_fit(cand, slices, kpad, kMaxChunkSlices)) {
        b = cand;
        S = slices;
        kchunks = kc;
      }
    }
    if (!b)
      return nrs_fail(h, NRS_ERR_TOO_LARGE,
                      "k too large for this slice count (ceil(k / 16384) * S must be < 128)");
  }
  if (m == 0 || n == 0) return NRS_OK;
  if (k == 0) {
    if (accumulate) return NRS_OK;
    return nrs_gemm(h, NRS_F64, m, 0, n, A, lda, B, ldb, C, ldc, 0, NRS_GEMM_GENERIC);
  }
  if (!A || !B || !C) return nrs_fail(h, NRS_ERR_INVALID, "null operand");
  int st = nrs_cuda_check(h, cudaSetDevice(h->device), "cudaSetDevice");
  if (st) return st;
  if (m > (1LL << 31) || n > (1LL << 31) || kpad > (1LL << 31))
    return nrs_fail(h, NRS_ERR_TOO_LARGE, "dimension beyond 2^31");
  const OzOperand a{A, lda, m, !ta};
  const OzOperand bT{B, ldb, n, tb};

  auto fallback = [&](const char*) {
    // Native FP64 (DMMA) GEMM: non-finite operands, or a spread that no
    // slice count within the limits covers.
    if (info) {
      info->slices = 0;
      info->products = 0;
      info->est_rel_error = 0.0;
    }
    return nrs_gemm(h, NRS_F64, m, k, n, A, lda, B, ldb, C, ldc, flags, NRS_GEMM_DMMA);
  };

  double spread = 0.0, dropped = 0.0;
  if (slices == 0) {
    SpreadResult r{};
    if ((st = spread_estimate(h, a, bT, false, m, n, k, kpad, 1, &r))) return st;
    if (r.flags & 1u) return fallback("non-finite operand");
    if (!(r.finite() && choose_digits(kpad, r.need(kTargetBits, k), &b, &S, &kchunks))) {
      // The pass-1 numerator counts every k; pass 2 counts only the k where
      // the other operand is nonzero (sparse and structured operands).
      if ((st = spread_estimate(h, a, bT, false, m, n, k, kpad, 2, &r))) return st;
      if (!(r.finite() && choose_digits(kpad, r.need(kTargetBits, k), &b, &S, &kchunks))) {
        if (info) info->spread = std::isfinite((double)r.rmax) ? (double)r.rmax : HUGE_VAL;
        return fallback("spread beyond the slice limits");
      }
    }
    spread = r.rmax;
    dropped = (double)(S - 1) * (double)k * (double)r.dinv;
  }
  if (info) {
    info->slices = S;
    info->products = S * (S + 1) / 2 * (kchunks > 0 ? kchunks : 1);
    info->slice_bits = b;
    info->k_chunk = kChunkOf(b);
    info->spread = spread;
    // auto: 2^-(bS) (R_max and the pairs left out), and the final rounding;
    // explicit: relative to rowmax|A| colmax|B| k, as no spread was measured
    info->est_rel_error = slices == 0 ? std::ldexp(std::max(spread, 1.0) + dropped, -b * S) + std::ldexp(1.0, -53)
                                      : std::ldexp(S + 1.0, -b * S);
  }
  return ozaki_run(h, a, bT, m, n, k, kpad, b, S, C, ldc, accumulate);
}

// ---------------------------------------------------------------------------
// Grouped launch: host side
// ---------------------------------------------------------------------------
struct nrs_ozaki_group {
  int S = 0, b = 0;
  int f32 = 0;  // element type of the group's problems: float (1) or double (0)
  int64_t pitch = 0, rows_a = 0, rows_b = 0, n_tiles = 0;
  int64_t n_rowch = 0, n_colch = 0, n_slcol = 0;
  void* arena = nullptr;
  OzIn* d_in = nullptr;
  OzChunk *d_rowch = nullptr, *d_colch = nullptr, *d_slcol = nullptr;
  OzProb* d_probs = nullptr;
  OzTile* d_tiles = nullptr;
  int *d_ea = nullptr, *d_eb = nullptr;
  unsigned long long* d_colmax = nullptr;
  uint16_t *d_sa = nullptr, *d_sb = nullptr;
  uint8_t* d_acc = nullptr;
};

void nrs_ozaki_group_free(nrs_ozaki_group* g) {
  if (!g) return;
  cudaFree(g->arena);
  delete g;
}

int nrs_ozaki_group_info(const nrs_ozaki_group* g, int* slices, int* bits, int64_t* tiles) {
  if (!g) return NRS_ERR_INVALID;
  if (slices) *slices = g->S;
  if (bits) *bits = g->b;
  if (tiles) *tiles = g->n_tiles;
  return NRS_OK;
}

// The row-major GEMMs of element type `dtype` (NRS_F64 or NRS_F32) as one
// group. Slice count for `slices` = 0: each problem's spread measured now
// (one read-back each); the group takes the largest count that one of them
// needs. Problems whose spread no count covers, or
// with Inf / NaN, are left out (they stay on the persistent kernel's DMMA or
// FP32 tiles). digit_bits 0 = the widest width the group's K allows.
int nrs_ozaki_group_build(nrs_handle* h, int64_t count, const nrs_gemm_desc* d, int dtype, int slices,
                          int digit_bits, int* accepted, nrs_ozaki_group** out) {
  *out = nullptr;
  if (slices < 0 || slices > OZ_MAX_SLICES) return nrs_fail(h, NRS_ERR_INVALID, "slices must be 0 (auto) or 1..16");
  if (digit_bits != 0 && (digit_bits < 6 || digit_bits > 8))
    return nrs_fail(h, NRS_ERR_INVALID, "digit bits must be 0 (widest) or 6..8");
  std::vector<int64_t> idx;
  int64_t kp_max = 0;
  for (int64_t i = 0; i < count; ++i) {
    accepted[i] = 0;
    const nrs_gemm_desc& g = d[i];
    if (g.dtype != dtype || (g.flags & (NRS_GEMM_TRANS_A | NRS_GEMM_TRANS_B)) || g.m <= 0 || g.n <= 0 || g.k <= 0)
      continue;
    idx.push_back(i);
    kp_max = std::max(kp_max, (g.k + OZ_BK - 1) / OZ_BK * OZ_BK);
  }
  if (idx.empty()) return NRS_OK;
  const bool f32 = dtype == NRS_F32;
  const int target = f32 ? kTargetBits32 : kTargetBits;
  OzNeed most{(double)target, 0.0};
  std::vector<int64_t> keep;
  for (int64_t i : idx) {
    const nrs_gemm_desc& g = d[i];
    if (slices > 0) {
      keep.push_back(i);
      continue;
    }
    const int64_t kpad1 = slice_pitch(g.k);
    SpreadResult r{};
    const OzOperand a{g.A, g.lda, g.m, true}, bT{g.B, g.ldb, g.n, false};
    int st = spread_estimate(h, a, bT, f32, g.m, g.n, g.k, kpad1, 1, &r);
    if (st) return st;
    if (r.flags & 1u) continue;
    int bb, SS, kc;
    if (!(r.finite() && choose_digits(kp_max, r.need(target, g.k), &bb, &SS, &kc, kMaxChunkSlicesGrouped))) {
      if ((st = spread_estimate(h, a, bT, f32, g.m, g.n, g.k, kpad1, 2, &r))) return st;
      if (!(r.finite() && choose_digits(kp_max, r.need(target, g.k), &bb, &SS, &kc, kMaxChunkSlicesGrouped)))
        continue;
    }
    const OzNeed need = r.need(target, g.k);
    most.bits = std::max(most.bits, need.bits);
    most.drop_bits = std::max(most.drop_bits, need.drop_bits);
    keep.push_back(i);
  }
  if (keep.empty()) return NRS_OK;
  int b = 0, S = 0, kc_max = 0;
  if (digit_bits) {
    // a given width: S from the bits (or as given), if the width's limits hold
    const int s_c = slices > 0 ? slices : slices_for(digit_bits, most);
    if (digits_fit(digit_bits, s_c, kp_max, kMaxChunkSlicesGrouped)) {
      b = digit_bits;
      S = s_c;
    } else {
      return NRS_OK;  // this width cannot carry the bits: all stay on DMMA
    }
  } else if (slices > 0) {
    for (int cand = 8; cand >= 6 && !b; --cand) {
      const int kc = (int)((kp_max + kChunkOf(cand) - 1) / kChunkOf(cand));
      if (digits_fit(cand, slices, kp_max, kMaxChunkSlicesGrouped)) {
        b = cand;
        S = slices;
        kc_max = kc;
      }
    }
    if (!b) return nrs_fail(h, NRS_ERR_TOO_LARGE, "k too large for this slice count");
  } else if (!choose_digits(kp_max, most, &b, &S, &kc_max, kMaxChunkSlicesGrouped)) {
    return NRS_OK;  // nothing qualifies together: all stay on DMMA
  }
  (void)kc_max;
  // Layout: offsets, chunk tables, tiles (most work first: the persistent
  // kernel hands tiles out round-robin).
  std::vector<OzIn> ins;
  std::vector<OzProb> probs;
  std::vector<OzChunk> rowch, colch, slcol;
  struct TileW {
    double w;
    OzTile t;
  };
  std::vector<TileW> tiles;
  int64_t rowoff = 0, coloff = 0;
  for (int64_t i : keep) {
    const nrs_gemm_desc& g = d[i];
    const int64_t kpad = (g.k + OZ_BK - 1) / OZ_BK * OZ_BK;
    const int p = (int)ins.size();
    ins.push_back(OzIn{g.A, g.lda, g.B, g.ldb, g.m, g.n, g.k, kpad, rowoff, coloff});
    const int kc = (int)((kpad + kChunkOf(b) - 1) / kChunkOf(b));
    probs.push_back(OzProb{g.m, g.n, kpad, rowoff, coloff, g.C, g.ldc, kc, S * (S + 1) / 2 * kc,
                           (g.flags & NRS_GEMM_ACCUMULATE) ? 1 : 0, f32 ? 1 : 0});
    for (int64_t r = 0; r < g.m; r += 8) rowch.push_back(OzChunk{p, (int32_t)r, 0, 0});
    for (int64_t c0 = 0; c0 < g.n; c0 += 32)
      for (int64_t k0 = 0; k0 < g.k; k0 += kColStrip) colch.push_back(OzChunk{p, (int32_t)c0, (int32_t)k0, 0});
    for (int64_t c0 = 0; c0 < g.n; c0 += kSliceColN)
      for (int64_t k0 = 0; k0 < kpad; k0 += kSliceColK) slcol.push_back(OzChunk{p, (int32_t)c0, (int32_t)k0, 0});
    constexpr int kBN = OzGeom<false, true>::BN;
    const int tm_n = (int)((g.m + OZ_BM - 1) / OZ_BM), tn_n = (int)((g.n + kBN - 1) / kBN);
    for (int a = 0; a < tm_n; ++a)
      for (int c = 0; c < tn_n; ++c) tiles.push_back({(double)kpad * (S * (S + 1) / 2), OzTile{p, a, c, 0}});
    rowoff += g.m;
    coloff += g.n;
  }
  std::stable_sort(tiles.begin(), tiles.end(), [](const TileW& x, const TileW& y) { return x.w > y.w; });
  std::vector<OzTile> tl(tiles.size());
  for (size_t i = 0; i < tiles.size(); ++i) tl[i] = tiles[i].t;
  if (rowoff > (1LL << 31) || coloff > (1LL << 31) || (int64_t)tl.size() > (1LL << 30))
    return NRS_OK;  // beyond the tensor maps' coordinate range: stay on DMMA
  auto al = [](size_t v) { return (v + 255) & ~size_t(255); };
  const size_t b_in = al(ins.size() * sizeof(OzIn)), b_rc = al(rowch.size() * sizeof(OzChunk)),
               b_cc = al(colch.size() * sizeof(OzChunk)), b_sc = al(slcol.size() * sizeof(OzChunk)),
               b_pr = al(probs.size() * sizeof(OzProb)), b_tl = al(tl.size() * sizeof(OzTile)),
               b_ea = al((size_t)rowoff * 4), b_eb = al((size_t)coloff * 4), b_cm = al((size_t)coloff * 8),
               b_sa = al((size_t)S * rowoff * kp_max * 2), b_sb = al((size_t)S * coloff * kp_max * 2),
               b_acc = al((size_t)h->hw_sms * OZ_BM * OzGeom<false, true>::BN * OZ_DIGIT_BYTES);  // a digit slot per CTA
  const size_t total = b_in + b_rc + b_cc + b_sc + b_pr + b_tl + b_ea + b_eb + b_cm + b_sa + b_sb + b_acc;
  nrs_ozaki_group* G = new nrs_ozaki_group();
  if (cudaMalloc(&G->arena, total) != cudaSuccess) {
    cudaGetLastError();
    delete G;
    return nrs_fail(h, NRS_ERR_ALLOC, "grouped Ozaki buffers");
  }
  uint8_t* q = (uint8_t*)G->arena;
  auto take = [&](size_t bytes) {
    uint8_t* p = q;
    q += bytes;
    return p;
  };
  G->d_in = (OzIn*)take(b_in);
  G->d_rowch = (OzChunk*)take(b_rc);
  G->d_colch = (OzChunk*)take(b_cc);
  G->d_slcol = (OzChunk*)take(b_sc);
  G->d_probs = (OzProb*)take(b_pr);
  G->d_tiles = (OzTile*)take(b_tl);
  G->d_ea = (int*)take(b_ea);
  G->d_eb = (int*)take(b_eb);
  G->d_colmax = (unsigned long long*)take(b_cm);
  G->d_sa = (uint16_t*)take(b_sa);
  G->d_sb = (uint16_t*)take(b_sb);
  G->d_acc = take(b_acc);
  G->S = S;
  G->b = b;
  G->f32 = f32 ? 1 : 0;
  G->pitch = kp_max;
  G->rows_a = rowoff;
  G->rows_b = coloff;
  G->n_tiles = (int64_t)tl.size();
  G->n_rowch = (int64_t)rowch.size();
  G->n_colch = (int64_t)colch.size();
  G->n_slcol = (int64_t)slcol.size();
  cudaError_t e = cudaSuccess;
  auto up = [&](void* dst, const void* src, size_t bytes) {
    if (!e && bytes) e = cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
  };
  up(G->d_in, ins.data(), ins.size() * sizeof(OzIn));
  up(G->d_rowch, rowch.data(), rowch.size() * sizeof(OzChunk));
  up(G->d_colch, colch.data(), colch.size() * sizeof(OzChunk));
  up(G->d_slcol, slcol.data(), slcol.size() * sizeof(OzChunk));
  up(G->d_probs, probs.data(), probs.size() * sizeof(OzProb));
  up(G->d_tiles, tl.data(), tl.size() * sizeof(OzTile));
  if (e) {
    nrs_ozaki_group_free(G);
    return nrs_cuda_check(h, e, "cudaMemcpy(grouped Ozaki tables)");
  }
  for (int64_t i : keep) accepted[i] = 1;
  *out = G;
  return NRS_OK;
}

template <typename T, int b, bool SMALL>
int group_slices_s(nrs_handle* h, nrs_ozaki_group* G, cudaStream_t s) {
  const int64_t plane_a = G->rows_a * G->pitch, plane_b = G->rows_b * G->pitch;
  g_slice_rows<T, b, SMALL><<<(unsigned)G->n_rowch, 128, 0, s>>>(G->d_in, G->d_rowch, G->d_ea, G->S, G->pitch,
                                                                 plane_a, G->d_sa);
  const int smem = (int)((size_t)G->S * kSliceColN * kSliceColPitch * 4);
  int st = nrs_cuda_check(
      h, cudaFuncSetAttribute(g_slice_cols<T, b, SMALL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
      "cudaFuncSetAttribute(g_slice_cols)");
  if (st) return st;
  g_slice_cols<T, b, SMALL><<<(unsigned)G->n_slcol, 256, smem, s>>>(G->d_in, G->d_slcol, G->d_eb, G->S, G->pitch,
                                                                   plane_b, G->d_sb);
  return nrs_after_launch(h, "grouped ozaki slicing");
}
template <typename T, int b>
int group_slices(nrs_handle* h, nrs_ozaki_group* G, cudaStream_t s) {
  return b * G->S <= 64 ? group_slices_s<T, b, true>(h, G, s) : group_slices_s<T, b, false>(h, G, s);
}

template <typename T>
int group_prepare(nrs_handle* h, nrs_ozaki_group* G, cudaStream_t s) {
  g_col_max_bits<T><<<(unsigned)G->n_colch, 256, 0, s>>>(G->d_in, G->d_colch, G->d_colmax);
  exponents_from_bits<<<(unsigned)((G->rows_b + 255) / 256), 256, 0, s>>>(G->d_colmax, G->rows_b, G->d_eb);
  int st = nrs_after_launch(h, "grouped ozaki exponents");
  if (st) return st;
  return G->b == 8 ? group_slices<T, 8>(h, G, s) : G->b == 7 ? group_slices<T, 7>(h, G, s)
                                                             : group_slices<T, 6>(h, G, s);
}

// Enqueues the whole group on `s` (no host synchronisation).
int nrs_ozaki_group_launch(nrs_handle* h, nrs_ozaki_group* G, cudaStream_t s) {
  if (!G || G->n_tiles == 0) return NRS_OK;
  int st = nrs_cuda_check(h, cudaMemsetAsync(G->d_colmax, 0, (size_t)G->rows_b * 8, s), "cudaMemsetAsync");
  if (st) return st;
  st = G->f32 ? group_prepare<float>(h, G, s) : group_prepare<double>(h, G, s);
  if (st) return st;
  OzParams P{};
  P.kpad = G->pitch;
  P.slices = G->S;
  P.group_m = 1;
  P.ea = G->d_ea;
  P.eb = G->d_eb;
  P.acc = G->d_acc;
  P.digit_bits = G->b;
  P.kchunk = kChunkOf(G->b);
  P.err = h->dev_error;
  P.tiles = G->d_tiles;
  P.probs = G->d_probs;
  P.n_tiles = (int)G->n_tiles;
  return launch_tc<false, true>(h, G->d_sa, G->d_sb, G->S, P, G->rows_a, G->rows_b, s);
}

extern "C" int nrs_gemm_ozaki_grouped(nrs_handle* h, int64_t count, const nrs_gemm_desc* descs, int slices,
                                      int* on_tensor_cores, nrs_ozaki_info* info) {
  if (!h || count < 0 || (count && !descs)) return NRS_ERR_INVALID;
  h->last_error.clear();
  int st = nrs_cuda_check(h, cudaSetDevice(h->device), "cudaSetDevice");
  if (st) return st;
  for (int64_t i = 0; i < count; ++i) {
    const nrs_gemm_desc& g = descs[i];
    if (g.dtype != NRS_F64) return nrs_fail(h, NRS_ERR_DTYPE, "grouped Ozaki takes f64 GEMMs");
    if (g.flags & ~(NRS_GEMM_ACCUMULATE | NRS_GEMM_TRANS_A | NRS_GEMM_TRANS_B))
      return nrs_fail(h, NRS_ERR_INVALID, "unknown GEMM flag");
    const bool ta = g.flags & NRS_GEMM_TRANS_A, tb = g.flags & NRS_GEMM_TRANS_B;
    if (g.m < 0 || g.k < 0 || g.n < 0) return nrs_fail(h, NRS_ERR_SHAPE, "negative GEMM dimension");
    if (g.ldc < (g.n > 0 ? g.n : 1) || g.lda < ((ta ? g.m : g.k) > 0 ? (ta ? g.m : g.k) : 1) ||
        g.ldb < ((tb ? g.k : g.n) > 0 ? (tb ? g.k : g.n) : 1))
      return nrs_fail(h, NRS_ERR_SHAPE, "leading dimension too small");
    if (g.m * g.n > 0 && (!g.C || (g.k > 0 && (!g.A || !g.B)))) return nrs_fail(h, NRS_ERR_INVALID, "null operand");
  }
  std::vector<int> acc((size_t)count);
  nrs_ozaki_group* G = nullptr;
  if ((st = nrs_ozaki_group_build(h, count, descs, NRS_F64, slices, 0, acc.data(), &G))) return st;
  if (info) {
    std::memset(info, 0, sizeof(*info));
    if (G) {
      info->slices = G->S;
      info->slice_bits = G->b;
      info->k_chunk = kChunkOf(G->b);
      info->products = (int32_t)G->n_tiles;
    }
  }
  // the problems the group does not take run one by one on DMMA
  for (int64_t i = 0; i < count && st == NRS_OK; ++i) {
    if (on_tensor_cores) on_tensor_cores[i] = acc[i];
    if (!acc[i]) {
      const nrs_gemm_desc& g = descs[i];
      st = nrs_gemm(h, NRS_F64, g.m, g.k, g.n, g.A, g.lda, g.B, g.ldb, g.C, g.ldc, g.flags, NRS_GEMM_DMMA);
    }
  }
  if (st == NRS_OK && G) st = nrs_ozaki_group_launch(h, G, h->stream);
  if (G) {
    cudaStreamSynchronize(h->stream);  // the group's buffers are freed below
    nrs_ozaki_group_free(G);
  }
  return st;
}

