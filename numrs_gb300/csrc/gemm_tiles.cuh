// Block-level GEMM tile bodies shared by the standalone GEMM kernels
// (gemm.cu) and the persistent grouped kernel (grouped.cu), so both produce
// bit-identical results for the same tile shape.
//
// A tile computes acc = A[m0:m0+BM, k0:k1] * B[k0:k1, n0:n0+BN] with
// (row, col) element strides, into registers; `tile_store` writes (or adds)
// it to C. Shared memory comes from the caller (a raw byte buffer).
#pragma once

#include "nrs_internal.cuh"

namespace nrs_tiles {

__device__ __forceinline__ void dmma_m8n8k4(double& d0, double& d1, double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// ---------------------------------------------------------------------------
// FP64 DMMA tile: warp grid WM x WN, warp tile (BM/WM) x (BN/WN) built from
// m8n8k4 fragments; k-major shared tiles with a pitch of BM+8 / BN+8 doubles
// so a fragment load touches each bank pair at most twice (256 B minimum).
// ---------------------------------------------------------------------------
template <int BM, int BN, int WM, int WN>
struct Dmma {
  static constexpr int BK = 16;
  static constexpr int NT = WM * WN * 32;
  static constexpr int TM = BM / WM, TN = BN / WN;
  static constexpr int FM = TM / 8, FN = TN / 8;
  static constexpr int PA = BM + 8, PB = BN + 8;
  static constexpr int LA = BM * BK / NT, LB = BN * BK / NT;
  static constexpr int kSmem = 2 * BK * (PA + PB) * 8;
  double acc[FM][FN][2];

  __device__ __forceinline__ void run(const double* __restrict__ A, int64_t rsa, int64_t csa,
                                      const double* __restrict__ B, int64_t rsb, int64_t csb,
                                      int64_t m, int64_t n, int64_t m0, int64_t n0, int64_t k0,
                                      int64_t k1, uint8_t* smem) {
    double(*As)[BK][PA] = reinterpret_cast<double(*)[BK][PA]>(smem);
    double(*Bs)[BK][PB] = reinterpret_cast<double(*)[BK][PB]>(smem + 2 * BK * PA * 8);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp / WN, wn = warp % WN;
    const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
    for (int i = 0; i < FM; ++i)
#pragma unroll
      for (int j = 0; j < FN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    double ra[LA], rb[LB];
    auto load = [&](int64_t kt) {
#pragma unroll
      for (int i = 0; i < LA; ++i) {
        int e = tid + i * NT;
        int r = e / BK, kk = e % BK;
        int64_t gi = m0 + r, gk = kt + kk;
        ra[i] = (gi < m && gk < k1) ? A[gi * rsa + gk * csa] : 0.0;
      }
#pragma unroll
      for (int i = 0; i < LB; ++i) {
        int e = tid + i * NT;
        int kk = e / BN, c = e % BN;
        int64_t gk = kt + kk, gj = n0 + c;
        rb[i] = (gk < k1 && gj < n) ? B[gk * rsb + gj * csb] : 0.0;
      }
    };
    auto store = [&](int buf) {
#pragma unroll
      for (int i = 0; i < LA; ++i) {
        int e = tid + i * NT;
        As[buf][e % BK][e / BK] = ra[i];
      }
#pragma unroll
      for (int i = 0; i < LB; ++i) {
        int e = tid + i * NT;
        Bs[buf][e / BN][e % BN] = rb[i];
      }
    };
    const int64_t ktiles = (k1 - k0 + BK - 1) / BK;
    if (ktiles > 0) {
      load(k0);
      store(0);
    }
    __syncthreads();
    for (int64_t kt = 0; kt < ktiles; ++kt) {
      const int buf = (int)(kt & 1);
      if (kt + 1 < ktiles) load(k0 + (kt + 1) * BK);
#pragma unroll
      for (int ks = 0; ks < BK; ks += 4) {
        double af[FM], bf[FN];
#pragma unroll
        for (int i = 0; i < FM; ++i) af[i] = As[buf][ks + t4][wm * TM + i * 8 + g];
#pragma unroll
        for (int j = 0; j < FN; ++j) bf[j] = Bs[buf][ks + t4][wn * TN + j * 8 + g];
#pragma unroll
        for (int i = 0; i < FM; ++i)
#pragma unroll
          for (int j = 0; j < FN; ++j) dmma_m8n8k4(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
      }
      if (kt + 1 < ktiles) store(buf ^ 1);
      __syncthreads();
    }
  }

  // Element (r, c) of the tile held by this thread, e = 0 .. FM*FN*2-1.
  __device__ __forceinline__ void coords(int e, int& r, int& c) const {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = warp / WN, wn = warp % WN;
    const int i = e / (FN * 2), j = (e / 2) % FN, h = e & 1;
    r = wm * TM + i * 8 + (lane >> 2);
    c = wn * TN + j * 8 + 2 * (lane & 3) + h;
  }
  __device__ __forceinline__ double value(int e) const {
    const int i = e / (FN * 2), j = (e / 2) % FN, h = e & 1;
    return acc[i][j][h];
  }
  static constexpr int kPerThread = FM * FN * 2;
};

// ---------------------------------------------------------------------------
// SIMT register tile (f32 / f64). f32 tiles with TM, TN multiples of 4: thread
// (tr, tc) owns TM/4 groups of 4 consecutive rows, group g at
// g*(BM/(TM/4)) + 4*tr (columns likewise), so each k step reads its A and B
// fragments as 16-byte shared loads (TM/4 + TN/4 of them per TM*TN FMAs).
// Otherwise thread (tr, tc) owns rows tr + i*(BM/TM), cols tc + j*(BN/TN).
// Either way every C element is the same k-ordered FMA chain, so the mapping
// does not change a bit of the result.
// ---------------------------------------------------------------------------
// One operand's shared tile [BK][ROWS + 4] (k-major): element (row, k) of the
// operand at p[row * rs + k * ks], rs or ks being 1 (or neither: scalar
// loads). A thread moves vectors of V elements along whichever dimension is
// contiguous, so that a warp's loads cover whole sectors for either layout
// (with the fixed k-fastest mapping an operand that is contiguous along its
// rows took one sector per element: a 300 x 1000 x 257 f32 product with a
// transposed B 66 us). Addresses advance by a constant per k tile.
template <typename T, int ROWS, int BK, int NT>
struct SimtLoader {
  static constexpr int PER = ROWS * BK / NT;  // elements per thread
  static constexpr int V = PER < 16 / (int)sizeof(T) ? PER : 16 / (int)sizeof(T);
  static constexpr int N = PER / V;
  static_assert(PER >= 1 && PER % V == 0 && BK % V == 0 && ROWS % V == 0, "tile / thread split");
  T reg[N][V];
  const T* p[N];
  int row[N], kk[N];
  int64_t step, rstep;  // of a k tile; between a vector's elements along rows
  int64_t left;         // rows of the operand from the tile's first row on
  bool kfast, vec;

  __device__ __forceinline__ void init(const T* base, int64_t rs, int64_t ks_, int64_t rows, int64_t r0, int64_t k0) {
    kfast = ks_ == 1;
    step = (int64_t)BK * ks_;
    left = rows - r0;
    const T* tile = base + r0 * rs + k0 * ks_;
    // every vector of the tile is aligned when its first one and the pitch are
    vec = (kfast || rs == 1) && (reinterpret_cast<uintptr_t>(tile) % (V * sizeof(T))) == 0 &&
          ((kfast ? rs : ks_) % V) == 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int e = threadIdx.x + i * NT;
      row[i] = kfast ? e / (BK / V) : (e % (ROWS / V)) * V;
      kk[i] = kfast ? (e % (BK / V)) * V : e / (ROWS / V);
      p[i] = tile + (int64_t)row[i] * rs + (int64_t)kk[i] * ks_;
    }
    rstep = kfast ? 0 : rs;
  }

  // Loads the k tile whose first k is `kleft` before the end, then moves on.
  __device__ __forceinline__ void load(int64_t kleft) {
    const int rl = left < ROWS ? (int)left : ROWS, kl = kleft < BK ? (int)kleft : BK;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const bool whole = kfast ? (row[i] < rl && kk[i] + V <= kl) : (kk[i] < kl && row[i] + V <= rl);
      if (vec && whole) {
        if constexpr (V * sizeof(T) == 16) {
          const uint4 u = *reinterpret_cast<const uint4*>(p[i]);
          memcpy(reg[i], &u, 16);
        } else if constexpr (V * sizeof(T) == 8) {
          const uint2 u = *reinterpret_cast<const uint2*>(p[i]);
          memcpy(reg[i], &u, 8);
        } else {
          reg[i][0] = *p[i];
        }
      } else {
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const bool in = kfast ? (row[i] < rl && kk[i] + v < kl) : (kk[i] < kl && row[i] + v < rl);
          reg[i][v] = in ? p[i][kfast ? v : v * rstep] : T(0);
        }
      }
      p[i] += step;
    }
  }
  __device__ __forceinline__ void store(T (*sm)[ROWS + 4]) const {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (!kfast && V * sizeof(T) == 16) {
        uint4 u;
        memcpy(&u, reg[i], 16);
        *reinterpret_cast<uint4*>(&sm[kk[i]][row[i]]) = u;
      } else {
#pragma unroll
        for (int v = 0; v < V; ++v) sm[kfast ? kk[i] + v : kk[i]][kfast ? row[i] : row[i] + v] = reg[i][v];
      }
    }
  }
};

// a * b + c: one rounding for floats, wrapping for integers.
__device__ __forceinline__ float tile_fma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double tile_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ int64_t tile_fma(int64_t a, int64_t b, int64_t c) {
  return (int64_t)((unsigned long long)a * (unsigned long long)b + (unsigned long long)c);
}
__device__ __forceinline__ int32_t tile_fma(int32_t a, int32_t b, int32_t c) {
  return (int32_t)((unsigned)a * (unsigned)b + (unsigned)c);
}
__device__ __forceinline__ float tile_add(float a, float b) { return a + b; }
__device__ __forceinline__ double tile_add(double a, double b) { return a + b; }
__device__ __forceinline__ int64_t tile_add(int64_t a, int64_t b) {
  return (int64_t)((unsigned long long)a + (unsigned long long)b);
}
__device__ __forceinline__ int32_t tile_add(int32_t a, int32_t b) { return (int32_t)((unsigned)a + (unsigned)b); }

template <typename T, int BM, int BN, int BK, int TM, int TN>
struct Simt {
  static constexpr int NT = (BM / TM) * (BN / TN);
  static constexpr int kSmem = 2 * BK * ((BM + 4) + (BN + 4)) * (int)sizeof(T);
  static constexpr bool kVec = sizeof(T) == 4 && TM % 4 == 0 && TN % 4 == 0;
  T acc[TM][TN];
  // Row (column) of fragment element i (j) for thread row tr (column tc).
  static __device__ __forceinline__ int row_of(int tr, int i) {
    return kVec ? (i / 4) * (BM / (TM / 4)) + 4 * tr + (i % 4) : tr + i * (BM / TM);
  }
  static __device__ __forceinline__ int col_of(int tc, int j) {
    return kVec ? (j / 4) * (BN / (TN / 4)) + 4 * tc + (j % 4) : tc + j * (BN / TN);
  }

  __device__ __forceinline__ void run(const T* __restrict__ A, int64_t rsa, int64_t csa,
                                      const T* __restrict__ B, int64_t rsb, int64_t csb,
                                      int64_t m, int64_t n, int64_t m0, int64_t n0, int64_t k0,
                                      int64_t k1, uint8_t* smem) {
    T(*As)[BK][BM + 4] = reinterpret_cast<T(*)[BK][BM + 4]>(smem);
    T(*Bs)[BK][BN + 4] = reinterpret_cast<T(*)[BK][BN + 4]>(smem + 2 * BK * (BM + 4) * sizeof(T));
    const int tid = threadIdx.x;
    const int tr = tid / (BN / TN), tc = tid % (BN / TN);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = T(0);
    SimtLoader<T, BM, BK, NT> la;
    SimtLoader<T, BN, BK, NT> lb;
    la.init(A, rsa, csa, m, m0, k0);
    lb.init(B, csb, rsb, n, n0, k0);
    const int64_t ktiles = (k1 - k0 + BK - 1) / BK;
    int64_t kleft = k1 - k0;
    if (ktiles > 0) {
      la.load(kleft);
      lb.load(kleft);
      la.store(As[0]);
      lb.store(Bs[0]);
    }
    __syncthreads();
    for (int64_t kt = 0; kt < ktiles; ++kt) {
      const int buf = (int)(kt & 1);
      kleft -= BK;
      if (kt + 1 < ktiles) {
        la.load(kleft);
        lb.load(kleft);
      }
#pragma unroll
      for (int kk = 0; kk < BK; ++kk) {
        T a[TM], b[TN];
        if constexpr (kVec) {
#pragma unroll
          for (int g = 0; g < TM / 4; ++g) {
            const uint4 v = *reinterpret_cast<const uint4*>(&As[buf][kk][row_of(tr, 4 * g)]);
            memcpy(&a[4 * g], &v, 16);
          }
#pragma unroll
          for (int g = 0; g < TN / 4; ++g) {
            const uint4 v = *reinterpret_cast<const uint4*>(&Bs[buf][kk][col_of(tc, 4 * g)]);
            memcpy(&b[4 * g], &v, 16);
          }
        } else {
#pragma unroll
          for (int i = 0; i < TM; ++i) a[i] = As[buf][kk][row_of(tr, i)];
#pragma unroll
          for (int j = 0; j < TN; ++j) b[j] = Bs[buf][kk][col_of(tc, j)];
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = tile_fma(a[i], b[j], acc[i][j]);
      }
      if (kt + 1 < ktiles) {
        la.store(As[buf ^ 1]);
        lb.store(Bs[buf ^ 1]);
      }
      __syncthreads();
    }
  }
  __device__ __forceinline__ void coords(int e, int& r, int& c) const {
    const int tid = threadIdx.x;
    const int tr = tid / (BN / TN), tc = tid % (BN / TN);
    r = row_of(tr, e / TN);
    c = col_of(tc, e % TN);
  }
  __device__ __forceinline__ T value(int e) const { return acc[e / TN][e % TN]; }
  static constexpr int kPerThread = TM * TN;
};

// Writes (or, with accumulate, adds -- product rounded first) the tile to C.
template <typename T, typename Tile>
__device__ __forceinline__ void tile_store(const Tile& t, T* __restrict__ C, int64_t ldc, int64_t m,
                                           int64_t n, int64_t m0, int64_t n0, bool accumulate) {
#pragma unroll
  for (int e = 0; e < Tile::kPerThread; ++e) {
    int r, c;
    t.coords(e, r, c);
    const int64_t gi = m0 + r, gj = n0 + c;
    if (gi < m && gj < n) {
      T* p = C + gi * ldc + gj;
      const T v = (T)t.value(e);
      *p = accumulate ? tile_add(*p, v) : v;
    }
  }
}

}  // namespace nrs_tiles
