// Plain GEMM: C := A*B (or C += A*B), the GPU form of kernels::gemm::gemm_2d
// (src/kernels/gemm.rs:246).
//
//  * dmma_gemm   : f64 on the FP64 tensor path, mma.sync.m8n8k4.f64 fragments
//                  from shared-memory tiles (GB300's FP64 rate is the bound).
//  * simt_gemm   : f32 / f64 register-tiled CUDA-core GEMM.
//  * generic_gemm: one thread per C element, any dtype (integers wrap like
//                  gemm_generic, src/kernels/gemm.rs:408). Integer products of
//                  a tile or more run on SIMT tiles (the same wrapped sums).
//  * batched_gemm: every panel of an N-D product in one launch, on the same
//                  tiles.
//
// Operands are addressed with (row, col) element strides, so transposed views
// need no copy (the reference copies them in kernels::borrow::operand).
// Overwrite contract: C is written, never read, unless ACCUMULATE is set, in
// which case C += (A*B) with the product rounded first (matmul_to computes a
// temporary and adds it, src/array/operations_optimized.rs:385).
#include <algorithm>
#include <cmath>
#include <type_traits>

#include <cooperative_groups.h>

#include "gemm_tiles.cuh"

using namespace nrs_tiles;
namespace cg = cooperative_groups;

namespace {

// blockIdx.z takes k-values [z*kc, min(k, (z+1)*kc)). With one chunk the
// tile goes to C; with several, chunk z writes its product to the partial
// slab P + z*m*n (row pitch n) and splitk_finish adds the slabs.
template <int BM, int BN, int WM, int WN>
__global__ void __launch_bounds__(WM * WN * 32)
    dmma_gemm(int64_t m, int64_t n, int64_t k, int64_t kc, const double* __restrict__ A, int64_t rsa,
              int64_t csa, const double* __restrict__ B, int64_t rsb, int64_t csb,
              double* __restrict__ C, int64_t ldc, int accumulate, double* __restrict__ P,
              const uint32_t* __restrict__ unless) {
  launch_wait();
  launch_next();
  if (unless && *unless) return;
  using Tile = Dmma<BM, BN, WM, WN>;
  __shared__ __align__(16) uint8_t smem[Tile::kSmem];
  Tile t;
  const int64_t m0 = (int64_t)blockIdx.y * BM, n0 = (int64_t)blockIdx.x * BN;
  const int64_t k0 = (int64_t)blockIdx.z * kc, k1 = (k0 + kc < k) ? k0 + kc : k;
  t.run(A, rsa, csa, B, rsb, csb, m, n, m0, n0, k0, k1, smem);
  if (gridDim.z == 1)
    tile_store<double>(t, C, ldc, m, n, m0, n0, accumulate != 0);
  else
    tile_store<double>(t, P + (int64_t)blockIdx.z * m * n, n, m, n, m0, n0, false);
}

// C := p_0 + p_1 + ... + p_{S-1} (slab order), or C += that sum: the product
// is rounded (to T) before it meets C, as without the split. With `choice`,
// the slab count is `splits_if` where *choice != 0, else `splits`; one slab
// means C is already written.
template <typename T>
__global__ void splitk_finish(const double* __restrict__ P, int splits, int64_t m, int64_t n,
                              T* __restrict__ C, int64_t ldc, int accumulate, const uint32_t* __restrict__ choice,
                              int splits_if) {
  launch_wait();
  if (choice && *choice) splits = splits_if;
  if (splits <= 1) return;
  const int64_t mn = m * n;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < mn;
       e += (int64_t)gridDim.x * blockDim.x) {
    double v = P[e];
    for (int z = 1; z < splits; ++z) v += P[z * mn + e];
    T* c = C + (e / n) * ldc + (e % n);
    *c = accumulate ? *c + (T)v : (T)v;
  }
}

// DMMA tiling for an m x n x k product on `sms` SMs: 32x32 or 64x64 tiles and
// the number of k chunks (multiples of 16, at least 64 values each when split)
// that minimise the busiest SM's share of the work, ceil(ctas / sms) x the
// work of one CTA, a split charged 1% (its partial slabs and the finish).
// Measured at 256^3-2048^3: per flop the two tiles run within 4% of each
// other (32x32 ahead), and the CTAs' pipeline fill overlaps across the many
// CTAs an SM holds, so whole-wave balance is what decides.
struct DmmaPlan {
  int tile;
  int splits;
  int64_t kc;
};
DmmaPlan plan_dmma(int64_t m, int64_t n, int64_t k, int sms) {
#if defined(NRS_DMMA_TILE) && defined(NRS_DMMA_SPLITS)  // fixed plan, for measuring the model
  {
    int64_t kc = (k + NRS_DMMA_SPLITS - 1) / NRS_DMMA_SPLITS;
    kc = (kc + 15) / 16 * 16;
    return DmmaPlan{NRS_DMMA_TILE, (int)((k + kc - 1) / kc), kc};
  }
#endif
  DmmaPlan best{32, 1, k};
  double best_cost = 1e300;
  for (int tile : {32, 64}) {
    const double ntiles = (double)((m + tile - 1) / tile) * (double)((n + tile - 1) / tile);
    const double w = tile == 64 ? 4.0 : 1.0;
    for (int s = 1; s <= 16; ++s) {
      int64_t kc = (k + s - 1) / s;
      kc = (kc + 15) / 16 * 16;
      if (s > 1 && kc < 64) break;
      const int splits = (int)((k + kc - 1) / kc);
      if (splits != s) continue;
      if (splits > 1 && (double)splits * (double)m * (double)n * 8.0 > 256.0 * (1 << 20)) break;
      const double cost = std::ceil(ntiles * splits / sms) * w * ((double)kc / (double)k) * (splits > 1 ? 1.01 : 1.0);
      if (cost < best_cost - 1e-12) {
        best_cost = cost;
        best = DmmaPlan{tile, splits, kc};
      }
    }
  }
  return best;
}

template <typename T, int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), (BM * BN >= 128 * 128 ? 2 : 1))
    simt_gemm(int64_t m, int64_t n, int64_t k, const T* __restrict__ A, int64_t rsa, int64_t csa,
              const T* __restrict__ B, int64_t rsb, int64_t csb, T* __restrict__ C, int64_t ldc,
              int accumulate, const uint32_t* __restrict__ unless) {
  launch_wait();
  launch_next();
  if (unless && *unless) return;
  using Tile = Simt<T, BM, BN, BK, TM, TN>;
  __shared__ __align__(16) uint8_t smem[Tile::kSmem];
  Tile t;
  const int64_t m0 = (int64_t)blockIdx.y * BM, n0 = (int64_t)blockIdx.x * BN;
  t.run(A, rsa, csa, B, rsb, csb, m, n, m0, n0, 0, k, smem);
  tile_store<T>(t, C, ldc, m, n, m0, n0, accumulate != 0);
}

// K split over a cluster of `splits` CTAs: CTA `rank` takes k-values
// [rank*kc, min(k, (rank+1)*kc)) and leaves its product in shared memory; then
// every CTA adds a share of the tile's elements over the ranks in order
// (through distributed shared memory) and writes them. One launch and no
// scratch, so it needs no workspace shared between streams and runs under
// capture.
template <typename T, int BM, int NT, typename Tile>
__device__ __forceinline__ void cluster_sum_store(const Tile& t, T* part, int rank, int splits, T* C, int64_t ldc,
                                                  int64_t m, int64_t n, int64_t m0, int64_t n0, bool accumulate) {
#pragma unroll
  for (int e = 0; e < Tile::kPerThread; ++e) {
    int r, c;
    t.coords(e, r, c);
    part[r * BM + c] = t.value(e);
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const int share = BM * BM / splits;
  for (int i = threadIdx.x; i < share; i += NT) {
    const int idx = rank * share + i;
    const int64_t gi = m0 + idx / BM, gj = n0 + idx % BM;
    if (gi >= m || gj >= n) continue;
    T v = cluster.map_shared_rank(part, 0)[idx];
    for (int z = 1; z < splits; ++z) v = tile_add(v, cluster.map_shared_rank(part, z)[idx]);
    T* c = C + gi * ldc + gj;
    *c = accumulate ? tile_add(*c, v) : v;
  }
  cluster.sync();  // a CTA's shared memory outlives its readers
}

// A 64 x 64 tile with K split over a cluster of gridDim.z CTAs.
constexpr int kSplitTile = 64;
template <typename T>
using SplitTile = Simt<T, kSplitTile, kSplitTile, 16, 4, 4>;
constexpr int kSplitThreads = SplitTile<float>::NT;
template <typename T>
__global__ void __launch_bounds__(kSplitThreads, sizeof(T) == 4 ? 3 : 2)
    simt_gemm_split(int64_t m, int64_t n, int64_t k, int64_t kc, const T* __restrict__ A, int64_t rsa, int64_t csa,
                    const T* __restrict__ B, int64_t rsb, int64_t csb, T* __restrict__ C, int64_t ldc,
                    int accumulate, const uint32_t* __restrict__ unless) {
  using Tile = SplitTile<T>;
  static_assert(Tile::kSmem >= kSplitTile * kSplitTile * (int)sizeof(T), "the partial tile reuses the operand buffers");
  launch_wait();
  launch_next();
  if (unless && *unless) return;  // (the same word for every CTA of the cluster)
  __shared__ __align__(16) uint8_t smem[Tile::kSmem];
  Tile t;
  const int64_t m0 = (int64_t)blockIdx.y * kSplitTile, n0 = (int64_t)blockIdx.x * kSplitTile;
  const int64_t k0 = (int64_t)blockIdx.z * kc, k1 = (k0 + kc < k) ? k0 + kc : k;
  t.run(A, rsa, csa, B, rsb, csb, m, n, m0, n0, k0, k1, smem);
  const int splits = (int)gridDim.z;
  if (splits == 1) {
    tile_store<T>(t, C, ldc, m, n, m0, n0, accumulate != 0);
    return;
  }
  // (run() ends with a barrier)
  cluster_sum_store<T, kSplitTile, kSplitThreads>(t, reinterpret_cast<T*>(smem), (int)blockIdx.z, splits, C, ldc, m, n,
                                                  m0, n0, accumulate != 0);
}

// Generic GEMM: one thread per C element, k ascending, one rounding per op.
template <typename T> __device__ __forceinline__ T gmul(T a, T b) { return a * b; }
template <typename T> __device__ __forceinline__ T gadd(T a, T b) { return a + b; }
template <> __device__ __forceinline__ int64_t gmul(int64_t a, int64_t b) {
  return (int64_t)((unsigned long long)a * (unsigned long long)b);
}
template <> __device__ __forceinline__ int64_t gadd(int64_t a, int64_t b) {
  return (int64_t)((unsigned long long)a + (unsigned long long)b);
}
template <> __device__ __forceinline__ int32_t gmul(int32_t a, int32_t b) {
  return (int32_t)((unsigned)a * (unsigned)b);
}
template <> __device__ __forceinline__ int32_t gadd(int32_t a, int32_t b) {
  return (int32_t)((unsigned)a + (unsigned)b);
}
template <> __device__ __forceinline__ double gmul(double a, double b) { return __dmul_rn(a, b); }
template <> __device__ __forceinline__ double gadd(double a, double b) { return __dadd_rn(a, b); }
template <> __device__ __forceinline__ float gmul(float a, float b) { return __fmul_rn(a, b); }
template <> __device__ __forceinline__ float gadd(float a, float b) { return __fadd_rn(a, b); }

template <typename T>
__global__ void generic_gemm(int64_t m, int64_t n, int64_t k, const T* __restrict__ A, int64_t rsa,
                             int64_t csa, const T* __restrict__ B, int64_t rsb, int64_t csb,
                             T* __restrict__ C, int64_t ldc, int accumulate) {
  const int64_t total = m * n;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx / n, j = idx % n;
    T acc = T(0);
    for (int64_t p = 0; p < k; ++p) acc = gadd(acc, gmul(A[i * rsa + p * csa], B[p * rsb + j * csb]));
    T* c = C + i * ldc + j;
    *c = accumulate ? gadd(*c, acc) : acc;
  }
}

// Every panel of a batch: blockIdx.z + z0 is the panel's row-major index
// over the batch dimensions, whose strides place its operands.
constexpr int kMaxBatchDims = NRS_UFUNC_MAX_DIMS;
struct BatchDims {
  int n;
  int64_t size[kMaxBatchDims], a[kMaxBatchDims], b[kMaxBatchDims];
};
// SPLIT: K over clusters of `splits` CTAs along x (few panels with long sums:
// 2 x (64 x 4096 x 64) f64 1239 -> 159 us, which one CTA per tile adds 256
// k tiles for).
template <typename T, typename Tile, int BM, int NT, bool SPLIT>
__global__ void __launch_bounds__(NT)
    batched_gemm(const __grid_constant__ BatchDims g, int64_t z0, int64_t m, int64_t n, int64_t k, int splits,
                 int64_t kc, const T* __restrict__ A, int64_t rsa, int64_t csa, const T* __restrict__ B, int64_t rsb,
                 int64_t csb, T* __restrict__ C) {
  constexpr int kPart = SPLIT ? BM * BM * (int)sizeof(T) : 0;  // the partial tile reuses the operand buffers
  __shared__ __align__(16) uint8_t smem[Tile::kSmem > kPart ? Tile::kSmem : kPart];
  const int64_t z = z0 + blockIdx.z;
  int64_t rem = z, ao = 0, bo = 0;
  for (int d = g.n - 1; d >= 0; --d) {
    const int64_t c = rem % g.size[d];
    rem /= g.size[d];
    ao += c * g.a[d];
    bo += c * g.b[d];
  }
  Tile t;
  const int rank = SPLIT ? (int)(blockIdx.x % (unsigned)splits) : 0;
  const int64_t m0 = (int64_t)blockIdx.y * BM, n0 = (int64_t)(SPLIT ? blockIdx.x / (unsigned)splits : blockIdx.x) * BM;
  const int64_t k0 = rank * kc, k1 = SPLIT && k0 + kc < k ? k0 + kc : k;
  t.run(A + ao, rsa, csa, B + bo, rsb, csb, m, n, m0, n0, k0, k1, smem);
  T* const Cz = C + z * m * n;
  if constexpr (SPLIT)
    cluster_sum_store<T, BM, NT>(t, reinterpret_cast<T*>(smem), rank, splits, Cz, n, m, n, m0, n0, false);
  else
    tile_store<T>(t, Cz, n, m, n, m0, n0, false);
}

template <typename T>
__global__ void zero_fill_2d(T* C, int64_t m, int64_t n, int64_t ldc) {
  const int64_t total = m * n;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x)
    C[(idx / n) * ldc + idx % n] = T(0);
}

dim3 tiles(int64_t m, int64_t n, int bm, int bn) {
  return dim3((unsigned)((n + bn - 1) / bn), (unsigned)((m + bm - 1) / bm));
}

}  // namespace

namespace {

void launch_dmma(nrs_handle* h, const DmmaPlan& pl, int64_t m, int64_t k, int64_t n, const double* A, int64_t rsa,
                 int64_t csa, const double* B, int64_t rsb, int64_t csb, double* C, int64_t ldc, int acc, double* P,
                 const uint32_t* unless) {
  dim3 g = tiles(m, n, pl.tile, pl.tile);
  g.z = (unsigned)pl.splits;
  if (pl.tile == 64)
    nrs_launch_after(unless != nullptr, dmma_gemm<64, 64, 2, 4>, g, 256, 0, h->stream, m, n, k, pl.kc, A, rsa, csa, B,
                     rsb, csb, C, ldc, acc, P, unless);
  else
    nrs_launch_after(unless != nullptr, dmma_gemm<32, 32, 2, 2>, g, 128, 0, h->stream, m, n, k, pl.kc, A, rsa, csa, B,
                     rsb, csb, C, ldc, acc, P, unless);
}

int finish_grid(nrs_handle* h, int64_t m, int64_t n) {
  const int64_t blocks = (m * n + 255) / 256;
  return (int)(blocks < (int64_t)h->num_sms * 8 ? blocks : (int64_t)h->num_sms * 8);
}

// f32 GEMMs by themselves: 128 x 128 tiles, or 64 x 64 tiles with K split over
// up to 8 CTAs of a cluster (whole 16-wide k tiles, at least 64 values each),
// whichever the busiest SM finishes first (planned for NRS_PLAN_SMS, as the
// split decides the rounding). Measured (us, before with 32 x 32 or 128 x 128
// tiles / now): 300 x 1000 x 257 35 / 20, 512^3 29 / 19, 1024^3 124 / 76,
// 64 x 4096 x 64 115 / 29, 3000 x 2000 x 10 65 / 35.
struct F32Plan {
  int tile;
  int splits;
  int64_t kc;
  double us;
};
// 64 x 64 tiles alone; us as for f32.
F32Plan plan_split(int64_t m, int64_t n, int64_t k) {
  auto waves = [](double ctas) { return std::ceil(ctas / NRS_PLAN_SMS); };
  F32Plan best{64, 1, k, 1e300};
  const double t64 = (double)((m + 63) / 64) * (double)((n + 63) / 64);
  for (int z = 1; z <= 8; z *= 2) {
    const int64_t kc = ((k + z - 1) / z + 15) / 16 * 16;
    if (z > 1 && (kc < 64 || (k + kc - 1) / kc != z)) break;
    const double us = 4.0 + waves(t64 * z) * (double)kc * (64.0 * 64.0 / 1.0e5) + (z > 1 ? 2.0 : 0.0);
    if (us < best.us) best = F32Plan{64, z, kc, us};
  }
  return best;
}
F32Plan plan_f32(int64_t m, int64_t n, int64_t k) {
  const double t128 = (double)((m + 127) / 128) * (double)((n + 127) / 128);
  const F32Plan large{128, 1, k, 4.0 + std::ceil(t128 / NRS_PLAN_SMS) * (double)k * (128.0 * 128.0 / 1.45e5)};
  const F32Plan split = plan_split(m, n, k);
  return split.us < large.us ? split : large;
}

template <typename T>
void launch_simt_split(nrs_handle* h, const F32Plan& pl, int64_t m, int64_t k, int64_t n, const T* A, int64_t rsa,
                       int64_t csa, const T* B, int64_t rsb, int64_t csb, T* C, int64_t ldc, int acc,
                       const uint32_t* unless) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = tiles(m, n, kSplitTile, kSplitTile);
  cfg.gridDim.z = (unsigned)pl.splits;
  cfg.blockDim = dim3(kSplitThreads);
  cfg.stream = h->stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 1;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = (unsigned)pl.splits;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, simt_gemm_split<T>, m, n, k, pl.kc, A, rsa, csa, B, rsb, csb, C, ldc, acc, unless);
}

void launch_simt_f32(nrs_handle* h, bool large, int64_t m, int64_t k, int64_t n, const float* A, int64_t rsa,
                     int64_t csa, const float* B, int64_t rsb, int64_t csb, float* C, int64_t ldc, int acc,
                     const uint32_t* unless) {
  if (large)
    nrs_launch_after(unless != nullptr, simt_gemm<float, 128, 128, 8, 8, 8>, tiles(m, n, 128, 128), 256, 0, h->stream, m,
                     n, k, A, rsa, csa, B, rsb, csb, C, ldc, acc, unless);
  else
    simt_gemm<float, 32, 32, 16, 2, 2><<<tiles(m, n, 32, 32), 256, 0, h->stream>>>(m, n, k, A, rsa, csa, B, rsb, csb,
                                                                                   C, ldc, acc, unless);
}

void launch_auto_f32(nrs_handle* h, int64_t m, int64_t k, int64_t n, const float* A, int64_t rsa, int64_t csa,
                     const float* B, int64_t rsb, int64_t csb, float* C, int64_t ldc, int acc,
                     const uint32_t* unless) {
  const F32Plan pl = plan_f32(m, n, k);
  if (pl.tile == 128)
    launch_simt_f32(h, true, m, k, n, A, rsa, csa, B, rsb, csb, C, ldc, acc, unless);
  else
    launch_simt_split(h, pl, m, k, n, A, rsa, csa, B, rsb, csb, C, ldc, acc, unless);
}

// i64 products of row-major operands, modelled (us). One thread per element:
// 1.98 products per ns and 0.33 elements per ns, or 0.17 us per k of one
// thread's chain; 64 x 64 tiles 0.17 us per k and wave, K padded to 16.
// Measured (us, one thread per element / tiles): 64 x 20000 x 64 3313 / 479,
// 512^3 92 / 55, 8000 x 16 x 8000 714 / 381, 20000 x 100 x 100 106 / 100.
double generic_i64_us(int64_t m, int64_t n, int64_t k) {
  const double mn = (double)m * (double)n;
  return 4.0 + std::max(mn * (double)k / 1.98e6 + mn / 3.3e5, 0.17 * (double)k);
}
double tiled_i64_us(int64_t m, int64_t n, int64_t k) {
  const F32Plan pl = plan_split(m, n, k);
  const double ctas = (double)((m + 63) / 64) * (double)((n + 63) / 64) * pl.splits;
  return 4.0 + std::ceil(ctas / NRS_PLAN_SMS) * (double)((pl.kc + 15) / 16 * 16) * 0.17;
}

bool grid_too_large(int64_t m, int64_t n) { return (n + 31) / 32 > 0x7fffffffLL || (m + 31) / 32 > 65535; }

}  // namespace

double nrs_plain_f32_us(int64_t m, int64_t k, int64_t n) { return plan_f32(m, n, k).us; }

int nrs_dmma_splits(int64_t m, int64_t k, int64_t n) { return plan_dmma(m, n, k, NRS_PLAN_SMS).splits; }

int nrs_plain_gemm_unless(nrs_handle* h, int dtype, int64_t m, int64_t k, int64_t n, const void* A, int64_t rsa,
                          int64_t csa, const void* B, int64_t rsb, int64_t csb, void* C, int64_t ldc,
                          bool accumulate, const uint32_t* unless, double* slab, int tc_splits) {
  const int acc = accumulate ? 1 : 0;
  if (dtype == NRS_F64) {
    const DmmaPlan pl = plan_dmma(m, n, k, NRS_PLAN_SMS);
    launch_dmma(h, pl, m, k, n, (const double*)A, rsa, csa, (const double*)B, rsb, csb, (double*)C, ldc, acc, slab,
                unless);
    if (pl.splits > 1 || tc_splits > 1)
      nrs_launch_after(true, splitk_finish<double>, finish_grid(h, m, n), 256, 0, h->stream, slab, pl.splits, m, n,
                       (double*)C, ldc, acc, unless, tc_splits);
  } else {
    launch_auto_f32(h, m, k, n, (const float*)A, rsa, csa, (const float*)B, rsb, csb, (float*)C, ldc, acc, unless);
    if (tc_splits > 1)
      nrs_launch_after(true, splitk_finish<float>, finish_grid(h, m, n), 256, 0, h->stream, slab, 1, m, n, (float*)C,
                       ldc, acc, unless, tc_splits);
  }
  return nrs_after_launch(h, "plain GEMM behind the slice products");
}

// Launches one plain GEMM. Sizes are validated by the caller.
int nrs_plain_gemm_launch(nrs_handle* h, int dtype, int64_t m, int64_t k, int64_t n,
                          const void* A, int64_t rsa, int64_t csa, const void* B, int64_t rsb,
                          int64_t csb, void* C, int64_t ldc, bool accumulate, int variant) {
  const int acc = accumulate ? 1 : 0;
  cudaStream_t s = h->stream;
  if (grid_too_large(m, n)) variant = NRS_GEMM_GENERIC;
  if (variant == NRS_GEMM_AUTO) {
    if (dtype == NRS_F64) variant = NRS_GEMM_DMMA;
    else if (dtype != NRS_F32 && m * n < 1024) variant = NRS_GEMM_GENERIC;
  }
  // Integers from a 32 x 32 C on: tiles read each operand element once per 64
  // products, one thread per element reads two per product; a split K fills
  // the GPU (i64, us, one thread per element / tiles: 1000^3 657 / 308,
  // 300 x 1000 x 257 174 / 57). For i64 the padding of narrow and of shallow
  // products can cost more than that (2^20 x 64 x 16 542 / 1189,
  // 4096 x 1 x 4096 64 / 99).
  if (variant == NRS_GEMM_AUTO && dtype == NRS_I64 && csa == 1 && csb == 1 && generic_i64_us(m, n, k) < tiled_i64_us(m, n, k))
    variant = NRS_GEMM_GENERIC;
  if (variant == NRS_GEMM_AUTO && dtype == NRS_I64) {
    launch_simt_split(h, plan_split(m, n, k), m, k, n, (const int64_t*)A, rsa, csa, (const int64_t*)B, rsb, csb,
                      (int64_t*)C, ldc, acc, nullptr);
    return nrs_after_launch(h, "simt_gemm_split<i64>");
  }
  if (variant == NRS_GEMM_AUTO && dtype == NRS_I32) {
    launch_simt_split(h, plan_split(m, n, k), m, k, n, (const int32_t*)A, rsa, csa, (const int32_t*)B, rsb, csb,
                      (int32_t*)C, ldc, acc, nullptr);
    return nrs_after_launch(h, "simt_gemm_split<i32>");
  }
  if (variant == NRS_GEMM_AUTO) {
    launch_auto_f32(h, m, k, n, (const float*)A, rsa, csa, (const float*)B, rsb, csb, (float*)C, ldc, acc, nullptr);
    return nrs_after_launch(h, "simt_gemm<f32>");
  }
  if (variant == NRS_GEMM_DMMA && dtype == NRS_F64) {
    // The k split decides the rounding: plan for a fixed SM count.
    const DmmaPlan pl = plan_dmma(m, n, k, NRS_PLAN_SMS);
    double* P = nullptr;
    if (pl.splits > 1) {
      int st;
      P = (double*)nrs_workspace(h, (size_t)pl.splits * (size_t)(m * n) * sizeof(double), &st);
      if (!P) return st;
    }
    launch_dmma(h, pl, m, k, n, (const double*)A, rsa, csa, (const double*)B, rsb, csb, (double*)C, ldc, acc, P,
                nullptr);
    if (pl.splits > 1)
      splitk_finish<double><<<finish_grid(h, m, n), 256, 0, s>>>(P, pl.splits, m, n, (double*)C, ldc, acc, nullptr, 0);
    return nrs_after_launch(h, "dmma_gemm");
  }
  if ((variant == NRS_GEMM_SIMT || variant == NRS_GEMM_SIMT_SMALL) && dtype == NRS_F32) {
    launch_simt_f32(h, variant == NRS_GEMM_SIMT, m, k, n, (const float*)A, rsa, csa, (const float*)B, rsb, csb,
                    (float*)C, ldc, acc, nullptr);
    return nrs_after_launch(h, "simt_gemm<f32>");
  }
  if (variant == NRS_GEMM_SIMT && dtype == NRS_F64) {
    simt_gemm<double, 64, 64, 8, 4, 4><<<tiles(m, n, 64, 64), 256, 0, s>>>(
        m, n, k, (const double*)A, rsa, csa, (const double*)B, rsb, csb, (double*)C, ldc, acc, nullptr);
    return nrs_after_launch(h, "simt_gemm<f64,64>");
  }
  if (variant != NRS_GEMM_GENERIC && variant != NRS_GEMM_DMMA && variant != NRS_GEMM_SIMT &&
      variant != NRS_GEMM_SIMT_SMALL)
    return nrs_fail(h, NRS_ERR_INVALID, "unknown GEMM variant");
  if (variant != NRS_GEMM_GENERIC)
    return nrs_fail(h, NRS_ERR_DTYPE, "variant not available for this dtype");
  int64_t blocks = (m * n + 255) / 256;
  int grid = (int)(blocks < (int64_t)h->num_sms * 16 ? blocks : (int64_t)h->num_sms * 16);
  switch (dtype) {
    case NRS_F32:
      generic_gemm<float><<<grid, 256, 0, s>>>(m, n, k, (const float*)A, rsa, csa, (const float*)B, rsb, csb, (float*)C, ldc, acc);
      break;
    case NRS_F64:
      generic_gemm<double><<<grid, 256, 0, s>>>(m, n, k, (const double*)A, rsa, csa, (const double*)B, rsb, csb, (double*)C, ldc, acc);
      break;
    case NRS_I64:
      generic_gemm<int64_t><<<grid, 256, 0, s>>>(m, n, k, (const int64_t*)A, rsa, csa, (const int64_t*)B, rsb, csb, (int64_t*)C, ldc, acc);
      break;
    default:
      generic_gemm<int32_t><<<grid, 256, 0, s>>>(m, n, k, (const int32_t*)A, rsa, csa, (const int32_t*)B, rsb, csb, (int32_t*)C, ldc, acc);
      break;
  }
  return nrs_after_launch(h, "generic_gemm");
}

extern "C" int nrs_gemm(nrs_handle* h, int dtype, int64_t m, int64_t k, int64_t n, const void* A,
                        int64_t lda, const void* B, int64_t ldb, void* C, int64_t ldc,
                        unsigned flags, int variant) {
  if (!h) return NRS_ERR_INVALID;
  h->last_error.clear();
  if (m < 0 || k < 0 || n < 0) return nrs_fail(h, NRS_ERR_SHAPE, "negative GEMM dimension");
  if (!nrs_dtype_size(dtype)) return nrs_fail(h, NRS_ERR_DTYPE, "unknown dtype");
  if (flags & ~(NRS_GEMM_ACCUMULATE | NRS_GEMM_TRANS_A | NRS_GEMM_TRANS_B))
    return nrs_fail(h, NRS_ERR_INVALID, "unknown GEMM flag");
  if (variant < NRS_GEMM_AUTO || variant > NRS_GEMM_SIMT_SMALL)
    return nrs_fail(h, NRS_ERR_INVALID, "unknown GEMM variant");
  const bool ta = flags & NRS_GEMM_TRANS_A, tb = flags & NRS_GEMM_TRANS_B;
  // Leading-dimension checks (the reference checks slice lengths, :250).
  if (ldc < (n > 0 ? n : 1)) return nrs_fail(h, NRS_ERR_SHAPE, "ldc < n");
  if (lda < ((ta ? m : k) > 0 ? (ta ? m : k) : 1)) return nrs_fail(h, NRS_ERR_SHAPE, "lda too small");
  if (ldb < ((tb ? k : n) > 0 ? (tb ? k : n) : 1)) return nrs_fail(h, NRS_ERR_SHAPE, "ldb too small");
  if (m == 0 || n == 0) return NRS_OK;  // nothing to overwrite
  if (!C) return nrs_fail(h, NRS_ERR_INVALID, "null C");
  int st = nrs_cuda_check(h, cudaSetDevice(h->device), "cudaSetDevice");
  if (st) return st;
  const bool accumulate = flags & NRS_GEMM_ACCUMULATE;
  if (k == 0) {
    if (accumulate) return NRS_OK;  // C += 0
    int grid = h->num_sms * 4;
    switch (dtype) {
      case NRS_F32: zero_fill_2d<float><<<grid, 256, 0, h->stream>>>((float*)C, m, n, ldc); break;
      case NRS_F64: zero_fill_2d<double><<<grid, 256, 0, h->stream>>>((double*)C, m, n, ldc); break;
      case NRS_I64: zero_fill_2d<int64_t><<<grid, 256, 0, h->stream>>>((int64_t*)C, m, n, ldc); break;
      default: zero_fill_2d<int32_t><<<grid, 256, 0, h->stream>>>((int32_t*)C, m, n, ldc); break;
    }
    return nrs_after_launch(h, "zero_fill_2d");
  }
  if (!A || !B) return nrs_fail(h, NRS_ERR_INVALID, "null A or B");
  if (variant == NRS_GEMM_AUTO && !grid_too_large(m, n)) {
    st = nrs_tc_gemm_auto(h, dtype, m, k, n, A, lda, ta, B, ldb, tb, C, ldc, accumulate);
    if (st != NRS_ERR_UNSUPPORTED) return st;
  }
  const int64_t rsa = ta ? 1 : lda, csa = ta ? lda : 1;
  const int64_t rsb = tb ? 1 : ldb, csb = tb ? ldb : 1;
  return nrs_plain_gemm_launch(h, dtype, m, k, n, A, rsa, csa, B, rsb, csb, C, ldc, accumulate,
                               variant);
}

namespace {

// 64 x 64 tiles (weight 4) or 32 x 32, and K in ranges of at least 64 values
// over clusters of up to 8 CTAs while the batch does not fill the GPU: the form
// whose busiest SM has less to do (a split costs about 32 k-values of a tile).
struct BatchPlan {
  bool large;
  int splits;
  int64_t kc;
};
BatchPlan plan_batched(int64_t m, int64_t n, int64_t k, int64_t batch) {
  BatchPlan best{true, 1, k};
  double least = 1e300;
  for (int tile : {64, 32}) {
    const double ctas = (double)((m + tile - 1) / tile) * (double)((n + tile - 1) / tile) * (double)batch;
    for (int z = 1; z <= 8; z *= 2) {
      const int64_t kc = z > 1 ? ((k + z - 1) / z + 15) / 16 * 16 : k;
      if (z > 1 && (kc < 64 || (k + kc - 1) / kc != z || ctas * z >= 2.0 * NRS_PLAN_SMS)) break;
      const double cost = std::ceil(ctas * z / NRS_PLAN_SMS) * (tile == 64 ? 4.0 : 1.0) * ((double)kc + (z > 1 ? 32.0 : 0.0));
      if (cost < least) {
        least = cost;
        best = BatchPlan{tile == 64, z, kc};
      }
    }
  }
  return best;
}

template <typename T, typename Tile, int BM, int NT>
void launch_batched(nrs_handle* h, const BatchDims& g, const BatchPlan& pl, int64_t batch, int64_t m, int64_t k,
                    int64_t n, const void* A, int64_t rsa, int64_t csa, const void* B, int64_t rsb, int64_t csb,
                    void* C) {
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(NT);
  cfg.stream = h->stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)pl.splits;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = pl.splits > 1 ? 1 : 0;
  auto kern = pl.splits > 1 ? batched_gemm<T, Tile, BM, NT, true> : batched_gemm<T, Tile, BM, NT, false>;
  for (int64_t z0 = 0; z0 < batch; z0 += 65535) {
    cfg.gridDim = tiles(m, n, BM, BM);
    cfg.gridDim.x *= (unsigned)pl.splits;
    cfg.gridDim.z = (unsigned)(batch - z0 < 65535 ? batch - z0 : 65535);
    cudaLaunchKernelEx(&cfg, kern, g, z0, m, n, k, pl.splits, pl.kc, (const T*)A, rsa, csa, (const T*)B, rsb, csb,
                       (T*)C);
  }
}

}  // namespace

extern "C" int nrs_gemm_batched(nrs_handle* h, int dtype, int batch_ndim, const int64_t* batch_shape, int64_t m,
                                int64_t k, int64_t n, const void* A, const int64_t* a_strides, int64_t lda,
                                const void* B, const int64_t* b_strides, int64_t ldb, void* C, unsigned flags) {
  if (!h) return NRS_ERR_INVALID;
  h->last_error.clear();
  if (batch_ndim < 0 || batch_ndim > kMaxBatchDims || (batch_ndim && (!batch_shape || !a_strides || !b_strides)))
    return nrs_fail(h, NRS_ERR_INVALID, "bad batch dimensions");
  if (m < 0 || k < 0 || n < 0) return nrs_fail(h, NRS_ERR_SHAPE, "negative GEMM dimension");
  const size_t es = nrs_dtype_size(dtype);
  if (!es) return nrs_fail(h, NRS_ERR_DTYPE, "unknown dtype");
  if (flags & ~(NRS_GEMM_TRANS_A | NRS_GEMM_TRANS_B)) return nrs_fail(h, NRS_ERR_INVALID, "unknown GEMM flag");
  const bool ta = flags & NRS_GEMM_TRANS_A, tb = flags & NRS_GEMM_TRANS_B;
  if (lda < ((ta ? m : k) > 0 ? (ta ? m : k) : 1)) return nrs_fail(h, NRS_ERR_SHAPE, "lda too small");
  if (ldb < ((tb ? k : n) > 0 ? (tb ? k : n) : 1)) return nrs_fail(h, NRS_ERR_SHAPE, "ldb too small");
  BatchDims g{};
  g.n = batch_ndim;
  int64_t batch = 1;
  for (int d = 0; d < batch_ndim; ++d) {
    if (batch_shape[d] < 0) return nrs_fail(h, NRS_ERR_SHAPE, "negative dimension");
    if (a_strides[d] < 0 || b_strides[d] < 0) return nrs_fail(h, NRS_ERR_STRIDE, "negative stride");
    g.size[d] = batch_shape[d];
    g.a[d] = a_strides[d];
    g.b[d] = b_strides[d];
    batch *= batch_shape[d];
  }
  if (batch == 0 || m == 0 || n == 0) return NRS_OK;
  if (!C || (k > 0 && (!A || !B))) return nrs_fail(h, NRS_ERR_INVALID, "null operand");
  if (k == 0) return nrs_gemm(h, dtype, batch * m, 0, n, A, 1, B, n, C, n, 0, NRS_GEMM_AUTO);
  int st = nrs_cuda_check(h, cudaSetDevice(h->device), "cudaSetDevice");
  if (st) return st;
  // A panel that fills the GPU by itself has the single product's choice of
  // kernels (slice products among them).
  const bool fills = (double)((m + 127) / 128) * (double)((n + 127) / 128) >= NRS_PLAN_SMS ||
                     (dtype == NRS_F64 && nrs_tc_gemm_pays(NRS_F64, m, k, n));
  if (batch == 1 || fills || grid_too_large(m, n)) {
    const size_t panel = (size_t)m * (size_t)n * es;
    for (int64_t z = 0; z < batch; ++z) {
      int64_t rem = z, ao = 0, bo = 0;
      for (int d = batch_ndim - 1; d >= 0; --d) {
        const int64_t c = rem % g.size[d];
        rem /= g.size[d];
        ao += c * g.a[d];
        bo += c * g.b[d];
      }
      if ((st = nrs_gemm(h, dtype, m, k, n, (const uint8_t*)A + ao * (int64_t)es, lda,
                         (const uint8_t*)B + bo * (int64_t)es, ldb, (uint8_t*)C + z * panel, n, flags, NRS_GEMM_AUTO)))
        return st;
    }
    return NRS_OK;
  }
  const int64_t rsa = ta ? 1 : lda, csa = ta ? lda : 1;
  const int64_t rsb = tb ? 1 : ldb, csb = tb ? ldb : 1;
  const BatchPlan pl = plan_batched(m, n, k, batch);
  // One launch over (tiles, panels); a 32 x 96 x 80 x 112 f64 batch: 1.45 ms
  // as a plan built per call from one descriptor per panel, 0.07 ms here (the FP64
  // pipe takes 0.06 for the padded tiles).
#define NRS_BATCH(T, TILE, BM, NT) \
  launch_batched<T, TILE, BM, NT>(h, g, pl, batch, m, k, n, A, rsa, csa, B, rsb, csb, C)
  using F32L = Simt<float, 64, 64, 16, 4, 4>;
  using F32S = Simt<float, 32, 32, 16, 2, 2>;
  using F64L = Dmma<64, 64, 2, 4>;
  using F64S = Dmma<32, 32, 2, 2>;
  using I64L = Simt<int64_t, 64, 64, 8, 4, 4>;
  using I64S = Simt<int64_t, 32, 32, 16, 2, 2>;
  using I32L = Simt<int32_t, 64, 64, 16, 4, 4>;
  using I32S = Simt<int32_t, 32, 32, 16, 2, 2>;
  switch (dtype) {
    case NRS_F32: pl.large ? NRS_BATCH(float, F32L, 64, 256) : NRS_BATCH(float, F32S, 32, 256); break;
    case NRS_F64: pl.large ? NRS_BATCH(double, F64L, 64, 256) : NRS_BATCH(double, F64S, 32, 128); break;
    case NRS_I64: pl.large ? NRS_BATCH(int64_t, I64L, 64, 256) : NRS_BATCH(int64_t, I64S, 32, 256); break;
    default: pl.large ? NRS_BATCH(int32_t, I32L, 64, 256) : NRS_BATCH(int32_t, I32S, 32, 256); break;
  }
#undef NRS_BATCH
  return nrs_after_launch(h, "batched_gemm");
}

// ---------------------------------------------------------------------------
// Pipe-rate probes: the denominators for the GEMM rooflines on this device.
// ---------------------------------------------------------------------------
namespace {

// Every warp issues `iters` rounds of 8 independent m8n8k4 DMMA chains
// (8 x 512 flops per round) from registers; the operands change with the
// thread so nothing folds at compile time, and the result is stored only if
// it is NaN (never) so the chains stay live.
__global__ void __launch_bounds__(256) dmma_rate(int64_t iters, double seed, double* sink) {
  double a = seed + threadIdx.x * 1e-3, b = 1.0 - a * 1e-3;
  double d[8][2];
#pragma unroll
  for (int c = 0; c < 8; ++c) d[c][0] = d[c][1] = 0.0;
  for (int64_t i = 0; i < iters; ++i) {
#pragma unroll
    for (int c = 0; c < 8; ++c) dmma_m8n8k4(d[c][0], d[c][1], a, b);
  }
  double s = 0.0;
#pragma unroll
  for (int c = 0; c < 8; ++c) s += d[c][0] + d[c][1];
  if (s != s) sink[threadIdx.x] = s;
}

// FP32 FMA rate: 8 independent FMA chains per thread.
__global__ void __launch_bounds__(256) ffma_rate(int64_t iters, float seed, float* sink) {
  float x[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) x[c] = seed + (float)(threadIdx.x + c) * 1e-3f;
  const float a = 0.999f, b = 1e-4f;
  for (int64_t i = 0; i < iters; ++i) {
#pragma unroll
    for (int c = 0; c < 8; ++c) x[c] = fmaf(x[c], a, b);
  }
  float s = 0.0f;
#pragma unroll
  for (int c = 0; c < 8; ++c) s += x[c];
  if (s != s) sink[threadIdx.x] = s;
}

}  // namespace

extern "C" int nrs_probe_peak(nrs_handle* h, int kind, double* tflops) {
  if (!h || !tflops) return NRS_ERR_INVALID;
  if (kind != NRS_PEAK_FP64_DMMA && kind != NRS_PEAK_FP32_FMA)
    return nrs_fail(h, NRS_ERR_INVALID, "unknown probe kind");
  h->last_error.clear();
  int st = nrs_cuda_check(h, cudaSetDevice(h->device), "cudaSetDevice");
  if (st) return st;
  void* sink = nrs_workspace(h, 4096, &st);
  if (!sink) return st;
  // 32 warps per SM; long enough (tens of ms) that launch overhead is noise.
  const int blocks = h->num_sms * 4;
  const int64_t iters = kind == NRS_PEAK_FP64_DMMA ? 4096 : (1 << 20);
  cudaEvent_t e0, e1;
  if ((st = nrs_cuda_check(h, cudaEventCreate(&e0), "cudaEventCreate"))) return st;
  if ((st = nrs_cuda_check(h, cudaEventCreate(&e1), "cudaEventCreate"))) {
    cudaEventDestroy(e0);
    return st;
  }
  float best_ms = 1e30f;
  for (int rep = 0; rep < 4 && st == NRS_OK; ++rep) {  // first launch is a warm-up
    cudaEventRecord(e0, h->stream);
    if (kind == NRS_PEAK_FP64_DMMA)
      dmma_rate<<<blocks, 256, 0, h->stream>>>(iters, 0.5, (double*)sink);
    else
      ffma_rate<<<blocks, 256, 0, h->stream>>>(iters, 0.5f, (float*)sink);
    cudaEventRecord(e1, h->stream);
    st = nrs_cuda_check(h, cudaEventSynchronize(e1), "probe");
    float ms = 0.0f;
    if (st == NRS_OK) st = nrs_cuda_check(h, cudaEventElapsedTime(&ms, e0, e1), "cudaEventElapsedTime");
    if (st == NRS_OK && rep > 0 && ms < best_ms) best_ms = ms;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (st) return st;
  const double warps = (double)blocks * 8.0;
  const double flops = kind == NRS_PEAK_FP64_DMMA ? warps * (double)iters * 8.0 * 512.0
                                                  : warps * 32.0 * (double)iters * 8.0 * 2.0;
  *tflops = flops / (best_ms * 1e-3) / 1e12;
  return NRS_OK;
}
