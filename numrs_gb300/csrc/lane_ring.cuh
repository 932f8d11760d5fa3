// Sequential lane folds over views that TMA cannot address: rows or columns
// whose pitch or base is not a multiple of 16 bytes, lanes of any strides,
// and few lanes. Shared by the axis reductions (reduce.cu) and the running
// folds (scan.cu).
//
// One block of four warps owns 32 lanes. A folding warp (one lane per thread)
// walks the axis through a ring of shared-memory tiles; three moving warps
// fill the ring with element-sized cp.async copies (coalesced along the axis
// for rows, across lanes otherwise, whatever the alignment), several tiles
// ahead of the fold, and, for running folds, write the folded tiles back.
// A per-element transform (the squared deviations of a variance) is the
// moving warps' work, so that it runs on their SM partitions while the
// folding warp's partition carries only the ordered adds: an f64 add takes 64
// cycles of a partition, so three FP64 operations per element in the folding
// warp made a step 202 cycles.
//
// Before it, these views ran one thread per lane with strided loads
// (9973 x 12001 f64: row std 4.00 -> 1.41 ms, row max 7.70 -> 0.97 ms; f32 row
// sum 0.67 -> 0.15 ms).
//
// Every wait is bounded; on give-up the block records the error word, waits
// for its own copies and returns.
#pragma once
#include <type_traits>

#include "nrs_internal.cuh"

namespace nrs_ring {

constexpr int kLanes = 32;
constexpr int kThreads = 128;
constexpr int kMovers = 96;       // threads of the three moving warps
constexpr int kStages = 4;
constexpr int kXformLag = 2;      // tiles loaded ahead of the transform

// Axis positions per tile: 512 bytes of a lane, for the most bytes in flight,
// while every block is resident at that size (three per SM), else 256 bytes
// and six blocks per SM (19456 x 12001 f64 row sums: 1173 us as two waves of
// the larger tile).
inline int tile_len(int esize, int64_t n_lanes, int sms) {
  return ((n_lanes + kLanes - 1) / kLanes <= (int64_t)3 * sms ? 512 : 256) / esize;
}
// Shared tile layout: ROWS [lane][len + 1] (a thread reads its own row: the
// odd pitch keeps the 32 threads on different banks), else [position][lane].
__host__ __device__ constexpr int tile_elems(bool rows, int len) { return kLanes * (rows ? len + 1 : len); }
inline size_t smem_bytes(int esize, bool rows, int len) { return (size_t)kStages * tile_elems(rows, len) * esize; }

template <int N>
NRS_DEV void cp_async_n(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(N) : "memory");
}
// Arrives on `bar` once all of this thread's earlier cp.async have landed.
NRS_DEV void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
NRS_DEV void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
NRS_DEV void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
NRS_DEV void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Kept dimensions of a lane problem, outer to inner.
template <int DIMS>
struct LaneDims {
  int n;
  int64_t size[DIMS], xstride[DIMS], ostride[DIMS];
};

// Fold: the policy of the folding warp (one object per thread = lane).
//   kStore               tiles are written back to out (running folds)
//   kXform               movers apply xform(v, param, odd) to every element,
//                        with the lane's parameter; odd alternates
//   block<N>(v, j)       folds N consecutive values (positions j ...); with
//                        kStore the values become the prefixes
//   one(v, j)            the same for one value
//   finish(lane)         after the last position
template <typename T, bool ROWS, typename Fold, int DIMS>
__device__ __forceinline__ void run(const T* __restrict__ x, const LaneDims<DIMS>& g, int64_t n_lanes, int64_t alen,
                                    int64_t xastride, T* __restrict__ out, int64_t oastride,
                                    const T* __restrict__ param, int len, uint32_t* err, uint32_t site,
                                    Fold& fold) {
  const int pitch = ROWS ? len + 1 : kLanes;
  const int tile_size = tile_elems(ROWS, len);
  extern __shared__ __align__(16) uint8_t ring_smem[];
  T* const tiles = reinterpret_cast<T*>(ring_smem);
  __shared__ uint64_t full[kStages], done[kStages];
  __shared__ int64_t xoff[kLanes], ooff[kLanes];
  __shared__ T lane_param[kLanes];
  __shared__ int abort_flag, slot_min, fold_warp;

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int64_t l0 = (int64_t)blockIdx.x * kLanes;
  const int live = (int)(n_lanes - l0 < kLanes ? n_lanes - l0 : kLanes);
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], kMovers);
      mbar_init(&done[s], 1);
    }
    fence_mbar_init();
    abort_flag = 0;
    slot_min = 1 << 20;
    fold_warp = 4;
  }
  if (tid < kLanes) {
    // lanes past the last one stand for the first (their results are dropped)
    int64_t rem = l0 + (tid < live ? tid : 0), xb = 0, ob = 0;
    const int64_t o = rem;
    for (int d = g.n - 1; d >= 0; --d) {
      const int64_t c = rem % g.size[d];
      rem /= g.size[d];
      xb += c * g.xstride[d];
      ob += c * g.ostride[d];
    }
    xoff[tid] = xb;
    ooff[tid] = ob;
    if (Fold::kXform) lane_param[tid] = param[o];
  }
  __syncthreads();
  // The folding warp: blocks that share an SM fold on different partitions
  // (warp slots map to partitions modulo 4; the choice only affects speed).
  uint32_t slot;
  asm volatile("mov.u32 %0, %%warpid;" : "=r"(slot));
  if (lane == 0) atomicMin(&slot_min, (int)slot);
  __syncthreads();
  if (lane == 0 && (slot & 3u) == (((uint32_t)slot_min >> 2) & 3u)) atomicMin(&fold_warp, warp);
  __syncthreads();
  const int fw = fold_warp < 4 ? fold_warp : 0;

  volatile int* const aborted = &abort_flag;
  auto bounded = [&](uint64_t* bar, uint32_t phase) -> bool {
    for (uint32_t i = 0; i < NRS_WAIT_LIMIT; ++i) {
      if (mbar_try_wait(bar, phase)) return true;
      if (*aborted) return false;
    }
    *aborted = 1;
    atomicOr(err, NRS_DEVERR_REDUCE_TMA | (site << 8));
    return false;
  };
  const int64_t n_tiles = (alen + len - 1) / len;

  if (warp == fw) {
    // ---------------- fold ----------------
    // Blocks of N values, the next block's loads issued before the current
    // one is folded (a block's own loads in front of its chain of adds cost
    // 20 of 84 cycles per f64 step).
    constexpr int N = 8;
    uint32_t s = 0, ph = 0;
    bool ok = true;
    for (int64_t i = 0; i < n_tiles; ++i) {
      if (!bounded(&full[s], ph)) {
        ok = false;
        break;
      }
      // (threads past the last lane follow the first and store nothing)
      const int ml = lane < live ? lane : 0;
      T* const mine = tiles + (size_t)s * tile_size + (ROWS ? ml * pitch : ml);
      const int64_t j0 = i * len;
      const int cnt = (int)(alen - j0 < len ? alen - j0 : len);
      const int whole = cnt & ~(N - 1);
      auto read = [&](int e, T (&v)[N]) {
#pragma unroll
        for (int q = 0; q < N; ++q) v[q] = mine[ROWS ? e + q : (e + q) * kLanes];
      };
      auto work = [&](int e, T (&v)[N]) {
        fold.template block<N>(v, j0 + e);
        if (Fold::kStore && lane < live) {
#pragma unroll
          for (int q = 0; q < N; ++q) mine[ROWS ? e + q : (e + q) * kLanes] = v[q];
        }
      };
      T v0[N], v1[N];
      if (whole) read(0, v0);
      int e = 0;
#pragma unroll 1
      for (; e < whole; e += 2 * N) {
        if (e + N < whole) read(e + N, v1);
        work(e, v0);
        if (e + N >= whole) break;
        if (e + 2 * N < whole) read(e + 2 * N, v0);
        work(e + N, v1);
      }
      e = whole;
      for (; e < cnt; ++e) {
        T* const p = mine + (ROWS ? e : e * kLanes);
        T v = *p;
        fold.one(v, j0 + e);
        if (Fold::kStore && lane < live) *p = v;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&done[s]);
      if (++s == kStages) {
        s = 0;
        ph ^= 1;
      }
    }
    if (ok && lane < live) fold.finish(l0 + lane);
    return;
  }

  // ---------------- move ----------------
  const int mw = warp < fw ? warp : warp - 1;  // 0, 1, 2
  // A thread's elements of a tile: rows (positions) mw, mw + 3, ...; the same
  // ones for loading, transforming and storing, so that it needs no barrier
  // for its own elements. Its row offsets stay in registers and whole tiles
  // run unrolled (with both taken from memory in a loop, a copy cost 100
  // cycles of the warp).
  constexpr int kRows = (kLanes + 2) / 3;
  constexpr int FULL = 512 / (int)sizeof(T);
  int64_t xrow[ROWS ? kRows : 1];
#pragma unroll
  for (int k = 0; k < (ROWS ? kRows : 1); ++k) xrow[k] = xoff[ROWS ? (mw + 3 * k < kLanes ? mw + 3 * k : 0) : lane];
  // f(tile element index, lane, axis offset in the tile, the lane's input
  // offset, parity of the element among the thread's)
  auto walk_len = [&](auto whole_len, int cnt, auto f) {
    constexpr int LEN = decltype(whole_len)::value;
    if (ROWS) {
#pragma unroll
      for (int k = 0; k < kRows; ++k) {
        const int r = mw + 3 * k;
        if (r >= live) break;
#pragma unroll
        for (int q = 0; q < LEN; q += 32)
          if (q + lane < cnt) f(r * (LEN + 1) + q + lane, r, q + lane, xrow[ROWS ? k : 0], (k ^ (q / 32)) & 1);
      }
    } else if (lane < live) {
#pragma unroll 8
      for (int e = mw; e < cnt; e += 3) f(e * kLanes + lane, lane, e, xrow[0], e & 1);
    }
  };
  auto walk = [&](int64_t i, auto f) {
    const int64_t left = alen - i * len;
    const int cnt = (int)(left < len ? left : len);
    if (len == FULL) walk_len(std::integral_constant<int, FULL>{}, cnt, f);
    else walk_len(std::integral_constant<int, FULL / 2>{}, cnt, f);
  };
  auto load = [&](int64_t i, uint32_t s) {
    const uint32_t base = smem_u32(tiles + (size_t)s * tile_size);
    const T* const xt = x + i * len * (ROWS ? 1 : xastride);
    walk(i, [&](int at, int, int e, int64_t off, int) {
      cp_async_n<sizeof(T)>(base + (uint32_t)(at * sizeof(T)), xt + off + (ROWS ? (int64_t)e : e * xastride));
    });
  };
  uint32_t s = 0, ph = 1;         // slot to fill, phase of its earlier done
  int64_t i = 0;
  const int64_t last = n_tiles + (Fold::kStore ? kStages : Fold::kXform ? kXformLag : 0);
  for (; i < last; ++i) {
    if (i >= kStages && i < n_tiles + kStages) {  // tile i - kStages has been folded
      if ((Fold::kStore || i < n_tiles) && !bounded(&done[s], ph)) break;
      if (Fold::kStore)
        walk(i - kStages, [&](int at, int r, int e, int64_t, int) {
          out[ooff[r] + ((i - kStages) * len + e) * oastride] = tiles[(size_t)s * tile_size + at];
        });
    }
    if (i < n_tiles) load(i, s);
    if (Fold::kXform) {
      cp_async_commit();
      if (i >= kXformLag) {
        cp_async_wait<kXformLag>();  // this thread's elements of tile i - lag
        const int64_t t = i - kXformLag;
        const uint32_t ts = (uint32_t)(t % kStages);
        T* const tile = tiles + (size_t)ts * tile_size;
        walk(t, [&](int at, int r, int, int64_t, int odd) { tile[at] = Fold::xform(tile[at], lane_param[r], odd); });
        mbar_arrive(&full[ts]);
      }
    } else if (i < n_tiles) {
      cp_async_arrive(&full[s]);
    }
    if (++s == kStages) {
      s = 0;
      ph ^= 1;
    }
  }
  cp_async_wait_all();
}

}  // namespace nrs_ring
