// Elementwise ufunc programs and the fused y = exp(a*x + b) kernel.
//
// The reference's elementwise kernels take closures
// (kernels::elementwise::binary_serial, src/kernels/elementwise.rs:51) and
// ExprNode trees (src/expr/owned.rs:204). Across a C ABI they become postfix
// programs over a value stack. Every op rounds once (MUL then ADD is two
// roundings, never contracted into an FMA: the reference documents this at
// src/expr/fused_eval.rs:17-21), so results match a scalar evaluation of the
// same closure element for element; ln/sqrt and the f32 exp are CUDA's, the
// f64 exp is nrs_exp_fixed (f64_exp.cuh).
#include <cmath>
#include <cstring>
#include <type_traits>

#include "f64_exp.cuh"
#include "nrs_internal.cuh"

namespace {

struct Prog {
  int len;
  int has_exp;
  int32_t code[NRS_UFUNC_MAX_OPS];
  int32_t arg[NRS_UFUNC_MAX_OPS];
  double scalar[NRS_UFUNC_MAX_OPS];
};

struct Geometry {
  int ndim;
  int n_inputs;
  int64_t shape[NRS_UFUNC_MAX_DIMS];
  int64_t in_stride[NRS_UFUNC_MAX_INPUTS][NRS_UFUNC_MAX_DIMS];
  int64_t out_stride[NRS_UFUNC_MAX_DIMS];
  const void* in[NRS_UFUNC_MAX_INPUTS];
};

constexpr int kStack = 8;

// Codes that only optimise() writes (the evaluators of up to kMaxIn inputs
// know them): multiply the top of the stack by the scalar +-2^arg (f64);
// and the binary operations op whose right operand is input k (X_IN + 4 op +
// k), a scalar or the top itself (X_SCALAR, X_SELF + op).
enum { NRS_OP_X_SCALE2 = 100, NRS_OP_X_IN = 128, NRS_OP_X_SCALAR = 192, NRS_OP_X_SELF = 224 };
inline __host__ __device__ bool is_binary(int c) { return (c >= NRS_OP_ADD && c <= NRS_OP_DIV) || c == NRS_OP_MAX || c == NRS_OP_MIN; }

// Non-contracting arithmetic.
template <typename T> __device__ __forceinline__ T radd(T a, T b);
template <typename T> __device__ __forceinline__ T rsub(T a, T b);
template <typename T> __device__ __forceinline__ T rmul(T a, T b);
template <typename T> __device__ __forceinline__ T rdiv(T a, T b);
template <> __device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
template <> __device__ __forceinline__ float rsub(float a, float b) { return __fsub_rn(a, b); }
template <> __device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
template <> __device__ __forceinline__ float rdiv(float a, float b) { return __fdiv_rn(a, b); }
template <> __device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
template <> __device__ __forceinline__ double rsub(double a, double b) { return __dsub_rn(a, b); }
template <> __device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
template <> __device__ __forceinline__ double rdiv(double a, double b) { return __ddiv_rn(a, b); }
#define NRS_INT_OPS(T, U)                                                                      \
  template <> __device__ __forceinline__ T radd(T a, T b) { return (T)((U)a + (U)b); }         \
  template <> __device__ __forceinline__ T rsub(T a, T b) { return (T)((U)a - (U)b); }         \
  template <> __device__ __forceinline__ T rmul(T a, T b) { return (T)((U)a * (U)b); }         \
  template <> __device__ __forceinline__ T rdiv(T a, T b) {                                    \
    return (b == 0 || (b == (T)-1 && a == (T)((U)1 << (sizeof(T) * 8 - 1)))) ? (T)0 : a / b;   \
  }
NRS_INT_OPS(int64_t, unsigned long long)
NRS_INT_OPS(int32_t, unsigned)

// exp(f64): the fixed-point form, whose table of 2^(j/256) each block builds
// in shared memory (exp_table_init, 256 threads); results that are not
// normal take CUDA's exp.
__device__ __forceinline__ uint64_t* exp_table() {
  __shared__ uint64_t table[kNrsExpTable];
  return table;
}
template <typename T>
__device__ __forceinline__ void exp_table_init(bool used) {
  if constexpr (std::is_same<T, double>::value) {
    if (!used) return;  // (uniform)
    for (int j = threadIdx.x; j < kNrsExpTable; j += blockDim.x) exp_table()[j] = nrs_exp_entry(j);
    __syncthreads();
  }
}
// |x| >= 32 and NaN (a call, so that the common path's registers and code do
// not carry it); from -708.5 down and 710 up no result is normal.
__device__ __noinline__ double exp_far(double v) {
  const uint32_t hi = (uint32_t)__double2hiint(v);
  if (hi >= 0xC0862400u || (hi & 0x7FFFFFFFu) >= 0x40863000u) return exp(v);
  bool special;
  const double r = nrs_exp_fixed(v, exp_table(), special);
  return special ? exp(v) : r;
}
// Results that are 0 or Inf whatever the low bits: x <= -746 or x >= 710. (The
// arguments of a Gaussian over spread-out points and of masked scores are mostly
// such. 8192^2 of -Inf: 2347 us through exp_far, 2138 before the fixed-point
// form.)
__device__ __forceinline__ bool exp_flat(double v, double& r) {
  const uint64_t u = (uint64_t)__double_as_longlong(v);
  const bool zero = u - 0xC087500000000000ull <= 0xFFF0000000000000ull - 0xC087500000000000ull;
  const bool inf = u - 0x4086300000000000ull <= 0x7FF0000000000000ull - 0x4086300000000000ull;
  r = zero ? 0.0 : inf ? __longlong_as_double(0x7FF0000000000000ll) : r;
  return zero | inf;
}
template <int W>
__device__ __forceinline__ void exp_vec(double (&v)[W]) {
  double r[W];
  unsigned special = 0;
#pragma unroll
  for (int e = 0; e < W; ++e) {
    bool far;
    r[e] = nrs_exp_near(v[e], exp_table(), far);
    special |= (unsigned)far << e;
  }
  if (special) {
    bool flat = false;  // (tested first: arguments between 32 and 710 do not pay for it)
#pragma unroll
    for (int e = 0; e < W; ++e) flat |= ((uint32_t)__double2hiint(v[e]) & 0x7FFFFFFFu) >= 0x40863000u;
    if (flat) {
#pragma unroll
      for (int e = 0; e < W; ++e) special &= ~((unsigned)exp_flat(v[e], r[e]) << e);
    }
#pragma unroll 1
    for (int e = 0; special >> e; ++e) {
      if (!((special >> e) & 1)) continue;
      double x = v[0];
#pragma unroll
      for (int q = 1; q < W; ++q) x = q == e ? v[q] : x;
      x = exp_far(x);
#pragma unroll
      for (int q = 0; q < W; ++q) r[q] = q == e ? x : r[q];
    }
  }
#pragma unroll
  for (int e = 0; e < W; ++e) v[e] = r[e];
}
// (a call: the compiler would otherwise multiply in either case and select)
__device__ __noinline__ double mul_far(double x, double s) { return __dmul_rn(x, s); }
// x * s for s = +-2^k: an exponent-field add (the FP64 pipe is the slow one)
// while x and the product are normal, else the multiplication.
__device__ __forceinline__ double scale2(double x, int k, double s) {
  const uint32_t hi = (uint32_t)__double2hiint(x);
  const int be = (int)((hi >> 20) & 0x7FFu);
  if ((unsigned)(be - 1) < 2046u && (unsigned)(be + k - 1) < 2046u)
    return __hiloint2double((int)((hi + ((uint32_t)k << 20)) ^ ((uint32_t)__double2hiint(s) & 0x80000000u)),
                            __double2loint(x));
  return mul_far(x, s);
}

template <typename T>
__device__ __forceinline__ T unary(int code, T v) {
  if constexpr (std::is_floating_point<T>::value) {
    switch (code) {
      case NRS_OP_NEG: return -v;
      case NRS_OP_ABS: return fabs(v);
      case NRS_OP_SQRT: return sqrt(v);
      case NRS_OP_EXP:
        if constexpr (std::is_same<T, double>::value) {
          double w[1] = {v};
          exp_vec(w);
          return w[0];
        } else {
          return exp(v);
        }
      default: return log(v);
    }
  } else {
    switch (code) {
      case NRS_OP_NEG: return rsub<T>(T(0), v);
      default: return v < 0 ? rsub<T>(T(0), v) : v;
    }
  }
}

template <typename T>
__device__ __forceinline__ T binop(int code, T a, T b) {
  switch (code) {
    case NRS_OP_ADD: return radd(a, b);
    case NRS_OP_SUB: return rsub(a, b);
    case NRS_OP_MUL: return rmul(a, b);
    case NRS_OP_DIV: return rdiv(a, b);
    case NRS_OP_MAX:
      if constexpr (std::is_floating_point<T>::value) return (a != a || a > b) ? a : b;
      else return a > b ? a : b;
    default:
      if constexpr (std::is_floating_point<T>::value) return (a != a || a < b) ? a : b;
      else return a < b ? a : b;
  }
}

// ---------------------------------------------------------------------------
// Evaluators. An evaluator maps W elements of every input to W results:
// run<W>(in[kIn][W], res[W]). Everything stays in registers. The program
// is the same for every thread, so its op codes, input numbers and stack
// depth are warp-uniform: each step is decoded once per W elements and
// dispatched with a uniform switch whose cases touch the register arrays at
// compile-time indices only (a dynamic index would move them to local
// memory, a per-element select chain would cost ~8 instructions per slot).
// The top of the stack lives in `acc`; slots below it in `st`.
// ---------------------------------------------------------------------------
constexpr int kMaxIn = 4;  // inputs the register evaluators handle

#define NRS_SLOT_CASES(X) X(0) X(1) X(2) X(3) X(4) X(5) X(6)
static_assert(kStack - 1 == 7, "NRS_SLOT_CASES lists the kStack - 1 slots below the top");

// st has SL slots (the program's depth - 1, rounded up to 1, 3 or 7).
template <typename T, int SL, int W>
__device__ __forceinline__ void slot_store(T (&st)[SL][W], int slot, const T (&v)[W]) {
  switch (slot) {
#define NRS_STORE(S)                                                            \
  case S:                                                                       \
    if constexpr (S < SL) {                                                     \
      _Pragma("unroll") for (int e = 0; e < W; ++e) st[S < SL ? S : 0][e] = v[e]; \
    }                                                                           \
    break;
    NRS_SLOT_CASES(NRS_STORE)
#undef NRS_STORE
  }
}
template <typename T, int SL, int W>
__device__ __forceinline__ void slot_load(const T (&st)[SL][W], int slot, T (&v)[W]) {
  switch (slot) {
#define NRS_LOAD(S)                                                             \
  case S:                                                                       \
    if constexpr (S < SL) {                                                     \
      _Pragma("unroll") for (int e = 0; e < W; ++e) v[e] = st[S < SL ? S : 0][e]; \
    }                                                                           \
    break;
    NRS_SLOT_CASES(NRS_LOAD)
#undef NRS_LOAD
  }
}
template <typename T, int NI, int W>
__device__ __forceinline__ void input_load(const T (&in)[NI][W], int k, T (&v)[W]) {
  switch (k) {
#define NRS_IN(S) \
  case S:         \
    if constexpr (S < NI) {                                                         \
      _Pragma("unroll") for (int e = 0; e < W; ++e) v[e] = in[S < NI ? S : 0][e]; \
    }                                                                               \
    break;
    NRS_IN(0) NRS_IN(1) NRS_IN(2) NRS_IN(3)
#undef NRS_IN
  }
}
template <typename T, int W, bool EXP64>
__device__ __forceinline__ void unary_vec(int code, T (&acc)[W]) {
  if constexpr (std::is_same<T, double>::value && EXP64) {
    if (code == NRS_OP_EXP) {
      exp_vec(acc);
      return;
    }
  }
  switch (code) {
#define NRS_UN(C) \
  case C:         \
    _Pragma("unroll") for (int e = 0; e < W; ++e) acc[e] = unary<T>(C, acc[e]); break;
    case NRS_OP_EXP:  // (f64: handled above)
      if constexpr (!std::is_same<T, double>::value) {
#pragma unroll
        for (int e = 0; e < W; ++e) acc[e] = unary<T>(NRS_OP_EXP, acc[e]);
      }
      break;
    NRS_UN(NRS_OP_NEG) NRS_UN(NRS_OP_ABS) NRS_UN(NRS_OP_SQRT) NRS_UN(NRS_OP_LN)
#undef NRS_UN
  }
}
// acc = lhs (op) acc
template <typename T, int W>
__device__ __forceinline__ void binary_vec(int code, const T (&lhs)[W], T (&acc)[W]) {
  switch (code) {
#define NRS_BIN(C) \
  case C:          \
    _Pragma("unroll") for (int e = 0; e < W; ++e) acc[e] = binop<T>(C, lhs[e], acc[e]); break;
    NRS_BIN(NRS_OP_ADD) NRS_BIN(NRS_OP_SUB) NRS_BIN(NRS_OP_MUL) NRS_BIN(NRS_OP_DIV)
    NRS_BIN(NRS_OP_MAX) NRS_BIN(NRS_OP_MIN)
#undef NRS_BIN
  }
}

// acc = acc (op) input k / scalar / acc for the codes optimise() wrote: one
// uniform switch whose cases read both operands where they are (through the
// stack an operand moves twice, four register moves per element and operation).
#define NRS_FUSED_OPS(X) X(NRS_OP_ADD) X(NRS_OP_SUB) X(NRS_OP_MUL) X(NRS_OP_DIV) X(NRS_OP_MAX) X(NRS_OP_MIN)
template <int NI, typename T, int W>
__device__ __forceinline__ void fused_vec(int code, T s, const T (&in)[NI][W], T (&acc)[W]) {
  switch (code) {
#define NRS_FUSED_IN(C, K)                                                                                          \
  case NRS_OP_X_IN + 4 * (C) + (K):                                                                                 \
    if constexpr ((K) < NI) {                                                                                       \
      _Pragma("unroll") for (int e = 0; e < W; ++e) acc[e] = binop<T>(C, acc[e], in[(K) < NI ? (K) : 0][e]); \
    }                                                                                                               \
    break;
#define NRS_FUSED(C)                                                                                     \
  NRS_FUSED_IN(C, 0) NRS_FUSED_IN(C, 1) NRS_FUSED_IN(C, 2) NRS_FUSED_IN(C, 3)                            \
  case NRS_OP_X_SCALAR + (C):                                                                            \
    _Pragma("unroll") for (int e = 0; e < W; ++e) acc[e] = binop<T>(C, acc[e], s);                 \
    break;                                                                                               \
  case NRS_OP_X_SELF + (C):                                                                              \
    _Pragma("unroll") for (int e = 0; e < W; ++e) acc[e] = binop<T>(C, acc[e], acc[e]);            \
    break;
    NRS_FUSED_OPS(NRS_FUSED)
#undef NRS_FUSED
#undef NRS_FUSED_IN
  }
}

// The general program (validated on the host: depth 1..D, inputs
// < n_inputs, ends with one value). D (2, 4 or 8) bounds the stack the
// program reaches, so a shallow program holds only D - 1 slots in registers.
// NI: inputs held in registers. EXP64: an f64 program with an exp.
template <typename T, int D, int NI, bool EXP64 = false>
struct ProgEval {
  static constexpr int kIn = NI;
  // 16-byte vectors per thread step in the vector kernels, those evaluated
  // together, and resident blocks: shallow programs are bound by their
  // decoding (a step of 8 doubles or 16 floats pays it once), deep ones by
  // registers, and exp by the latency of its dependent integer chain, which
  // more warps hide. Measured at 8192^2 (us; one, two vectors per step and
  // now): f32 a*b+c 179, 187, 169; f32 gauss 380, 183, 145; f64 a*b+c 439,
  // 399, 381; f64 gauss with 2, 3, 4 blocks 507, 480, 473.
  static constexpr int kUnroll = D <= 2 && !EXP64 ? 4 : D <= 4 ? 2 : 1;
  static constexpr int kGroup = D <= 2 || sizeof(T) == 8 ? kUnroll : 1;
  static constexpr int kBlocks = D > 4 ? 1 : EXP64 ? (D <= 2 && NI <= 2 ? 4 : 2) : D <= 2 || sizeof(T) == 8 ? 2 : 3;
  Prog prog;
  __device__ __forceinline__ void init() const { exp_table_init<T>(EXP64); }
  template <int W>
  __device__ __forceinline__ void run(const T (&in)[kIn][W], T (&res)[W]) const {
    T acc[W], lhs[W], st[D - 1][W];
    int depth = 0;  // values on the stack, acc included
    for (int pc = 0; pc < prog.len; ++pc) {
      const int code = prog.code[pc];
      if (code >= NRS_OP_X_IN) {
        fused_vec<NI>(code, (T)prog.scalar[pc], in, acc);
      } else if (code == NRS_OP_INPUT || code == NRS_OP_SCALAR) {
        if (depth > 0) slot_store(st, depth - 1, acc);
        ++depth;
        if (code == NRS_OP_INPUT) {
          input_load(in, prog.arg[pc], acc);
        } else {
          const T s = (T)prog.scalar[pc];
#pragma unroll
          for (int e = 0; e < W; ++e) acc[e] = s;
        }
      } else if (code >= NRS_OP_NEG && code <= NRS_OP_LN) {
        unary_vec<T, W, EXP64>(code, acc);
      } else if (code == NRS_OP_X_SCALE2) {
        if constexpr (std::is_same<T, double>::value) {
#pragma unroll
          for (int e = 0; e < W; ++e) acc[e] = scale2(acc[e], prog.arg[pc], prog.scalar[pc]);
        }
      } else {
        --depth;
        slot_load(st, depth - 1, lhs);
        binary_vec(code, lhs, acc);
      }
    }
#pragma unroll
    for (int e = 0; e < W; ++e) res[e] = acc[e];
  }
};

// `inputs[0] op inputs[1]`: the operators and binary closures.
template <typename T, int OP>
struct BinEval {
  static constexpr int kIn = 2;
  static constexpr int kUnroll = 4, kGroup = sizeof(T) == 8 ? 2 : 1, kBlocks = 1;
  __device__ __forceinline__ void init() const {}
  template <int W>
  __device__ __forceinline__ void run(const T (&in)[kIn][W], T (&res)[W]) const {
#pragma unroll
    for (int e = 0; e < W; ++e) res[e] = binop<T>(OP, in[0][e], in[1][e]);
  }
};

// A unary operation of one input.
template <typename T, int OP>
struct UnEval {
  static constexpr int kIn = 1;
  static constexpr int kUnroll = 4, kGroup = sizeof(T) == 8 ? 2 : 1, kBlocks = 1;
  __device__ __forceinline__ void init() const { exp_table_init<T>(OP == NRS_OP_EXP); }
  template <int W>
  __device__ __forceinline__ void run(const T (&in)[kIn][W], T (&res)[W]) const {
#pragma unroll
    for (int e = 0; e < W; ++e) res[e] = in[0][e];
    unary_vec<T, W, OP == NRS_OP_EXP>(OP, res);
  }
};

// Any strides, one element per thread, full index decode (small inner dims).
template <typename T, typename Eval>
__global__ void __launch_bounds__(256)
    ufunc_decode(Eval ev, Geometry g, int64_t n, T* __restrict__ out) {
  ev.init();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t off[Eval::kIn] = {};
    int64_t ooff = 0;
    int64_t rem = i;
    for (int d = g.ndim - 1; d >= 0; --d) {
      const int64_t c = rem % g.shape[d];
      rem /= g.shape[d];
      ooff += c * g.out_stride[d];
#pragma unroll
      for (int k = 0; k < Eval::kIn; ++k) off[k] += c * g.in_stride[k][d];
    }
    T v[Eval::kIn][1], r[1];
#pragma unroll
    for (int k = 0; k < Eval::kIn; ++k)
      v[k][0] = k < g.n_inputs ? static_cast<const T*>(g.in[k])[off[k]] : T(0);
    ev.template run<1>(v, r);
    out[ooff] = r[0];
  }
}

// Broadcast / strided views with a long last dimension: a CTA takes one
// row (all dims but the last) at a time, decodes its offsets once and walks
// the row with plain strided increments.
template <typename T, typename Eval>
__global__ void __launch_bounds__(256)
    ufunc_rows(Eval ev, Geometry g, int64_t rows, T* __restrict__ out) {
  ev.init();
  const int last = g.ndim - 1;
  const int64_t inner = g.shape[last];
  for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
    int64_t off[Eval::kIn] = {};
    int64_t ooff = 0;
    int64_t rem = r;
    for (int d = last - 1; d >= 0; --d) {
      const int64_t c = rem % g.shape[d];
      rem /= g.shape[d];
      ooff += c * g.out_stride[d];
#pragma unroll
      for (int k = 0; k < Eval::kIn; ++k) off[k] += c * g.in_stride[k][d];
    }
    for (int64_t j = threadIdx.x; j < inner; j += blockDim.x) {
      T v[Eval::kIn][1], res[1];
#pragma unroll
      for (int k = 0; k < Eval::kIn; ++k)
        v[k][0] = k < g.n_inputs ? static_cast<const T*>(g.in[k])[off[k] + j * g.in_stride[k][last]] : T(0);
      ev.template run<1>(v, res);
      out[ooff + j * g.out_stride[last]] = res[0];
    }
  }
}

// Broadcast rows with 16-byte vectors: the last dimension has stride 1 in
// the output and stride 1 or 0 in every input (a broadcast row or column),
// every row starts 16-byte aligned and the row length is a multiple of the
// vector width (the host checks all three). A stride-0 input is one value
// per row, loaded once.
template <typename T, typename Eval>
__global__ void __launch_bounds__(256, Eval::kBlocks)
    ufunc_rows_vec(Eval ev, Geometry g, int64_t rows, T* __restrict__ out) {
  using V = typename std::conditional<sizeof(T) == 4, int4, longlong2>::type;
  constexpr int PER = 16 / sizeof(T);
  ev.init();
  const int last = g.ndim - 1;
  const int64_t nv = g.shape[last] / PER;
  for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
    int64_t off[Eval::kIn] = {};
    int64_t ooff = 0;
    int64_t rem = r;
    for (int d = last - 1; d >= 0; --d) {
      const int64_t c = rem % g.shape[d];
      rem /= g.shape[d];
      ooff += c * g.out_stride[d];
#pragma unroll
      for (int k = 0; k < Eval::kIn; ++k) off[k] += c * g.in_stride[k][d];
    }
    T bcast[Eval::kIn];
#pragma unroll
    for (int k = 0; k < Eval::kIn; ++k)
      bcast[k] = (k < g.n_inputs && g.in_stride[k][last] == 0) ? static_cast<const T*>(g.in[k])[off[k]] : T(0);
    // U vectors per thread step, all loads issued before any compute, which
    // takes them in G groups of W elements.
    constexpr int U = Eval::kUnroll, G = U / Eval::kGroup, W = Eval::kGroup * PER;
    for (int64_t j = threadIdx.x; j < nv; j += (int64_t)blockDim.x * U) {
      T x[G][Eval::kIn][W];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t jj = j + (int64_t)u * blockDim.x;
#pragma unroll
        for (int k = 0; k < Eval::kIn; ++k) {
          T* const xv = &x[u / (U / G)][k][u % (U / G) * PER];
          if (jj < nv && k < g.n_inputs && g.in_stride[k][last] != 0) {
            const V q = __ldcs(reinterpret_cast<const V*>(static_cast<const T*>(g.in[k]) + off[k]) + jj);
            memcpy(xv, &q, 16);
          } else {
#pragma unroll
            for (int e = 0; e < PER; ++e) xv[e] = bcast[k];
          }
        }
      }
#pragma unroll
      for (int i = 0; i < G; ++i) {
        if (j + (int64_t)i * (U / G) * blockDim.x >= nv) break;
        T res[W];
        ev.template run<W>(x[i], res);
#pragma unroll
        for (int u = 0; u < U / G; ++u) {
          const int64_t jj = j + (int64_t)(i * (U / G) + u) * blockDim.x;
          if (jj >= nv) break;
          V q;
          memcpy(&q, res + u * PER, 16);
          __stcs(reinterpret_cast<V*>(out + ooff) + jj, q);
        }
      }
    }
  }
}

// Same-shape contiguous, 16-byte aligned inputs and output (the common
// `&a + &b` of binary_serial): 16 bytes of every input per thread step.
template <typename T, typename Eval>
__global__ void __launch_bounds__(256, Eval::kBlocks)
    ufunc_flat_vec(Eval ev, Geometry g, int64_t n, T* __restrict__ out) {
  using V = typename std::conditional<sizeof(T) == 4, int4, longlong2>::type;
  constexpr int PER = 16 / sizeof(T);
  ev.init();
  const int64_t nv = n / PER;
  // A block covers U * blockDim consecutive vectors per step (coalesced for
  // each u); all loads are issued before any compute.
  constexpr int U = Eval::kUnroll, G = U / Eval::kGroup, W = Eval::kGroup * PER;
  const int64_t step = (int64_t)gridDim.x * blockDim.x * U;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x * U + threadIdx.x; i < nv; i += step) {
    T x[G][Eval::kIn][W];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t ii = i + (int64_t)u * blockDim.x;
#pragma unroll
      for (int k = 0; k < Eval::kIn; ++k) {
        T* const xv = &x[u / (U / G)][k][u % (U / G) * PER];
        if (ii < nv && k < g.n_inputs) {
          const V q = __ldcs(reinterpret_cast<const V*>(g.in[k]) + ii);
          memcpy(xv, &q, 16);
        } else {
#pragma unroll
          for (int e = 0; e < PER; ++e) xv[e] = T(0);
        }
      }
    }
#pragma unroll
    for (int gi = 0; gi < G; ++gi) {
      if (i + (int64_t)gi * (U / G) * blockDim.x >= nv) break;
      T res[W];
      ev.template run<W>(x[gi], res);
#pragma unroll
      for (int u = 0; u < U / G; ++u) {
        const int64_t ii = i + (int64_t)(gi * (U / G) + u) * blockDim.x;
        if (ii >= nv) break;
        V q;
        memcpy(&q, res + u * PER, 16);
        __stcs(reinterpret_cast<V*>(out) + ii, q);
      }
    }
  }
  // scalar tail (< PER elements)
  const int64_t t = nv * PER + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t < n) {
    T v[Eval::kIn][1], r[1];
#pragma unroll
    for (int k = 0; k < Eval::kIn; ++k) v[k][0] = k < g.n_inputs ? static_cast<const T*>(g.in[k])[t] : T(0);
    ev.template run<1>(v, r);
    out[t] = r[0];
  }
}

// Programs with more than kMaxIn inputs: the stack interpreter over up to 8
// inputs with a full index decode per element.
template <typename T>
__global__ void __launch_bounds__(256)
    ufunc_generic(Prog prog, Geometry g, int64_t n, T* __restrict__ out) {
  exp_table_init<T>(prog.has_exp);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t off[NRS_UFUNC_MAX_INPUTS];
    int64_t ooff = 0;
#pragma unroll
    for (int k = 0; k < NRS_UFUNC_MAX_INPUTS; ++k) off[k] = 0;
    int64_t rem = i;
    for (int d = g.ndim - 1; d >= 0; --d) {
      int64_t c = rem % g.shape[d];
      rem /= g.shape[d];
      ooff += c * g.out_stride[d];
      for (int k = 0; k < g.n_inputs; ++k) off[k] += c * g.in_stride[k][d];
    }
    T st[kStack];
    int sp = 0;
    for (int pc = 0; pc < prog.len; ++pc) {
      const int code = prog.code[pc];
      if (code == NRS_OP_INPUT) {
        st[sp++] = static_cast<const T*>(g.in[prog.arg[pc]])[off[prog.arg[pc]]];
      } else if (code == NRS_OP_SCALAR) {
        st[sp++] = (T)prog.scalar[pc];
      } else if (code >= NRS_OP_NEG && code <= NRS_OP_LN) {
        st[sp - 1] = unary<T>(code, st[sp - 1]);
      } else {
        T b = st[--sp];
        st[sp - 1] = binop<T>(code, st[sp - 1], b);
      }
    }
    out[ooff] = st[0];
  }
}

// y = exp((a*x) + b), contiguous, 16-byte vectors, streaming loads/stores
// (every byte is touched once, so keep it from displacing L2 contents).
__device__ __forceinline__ float ea(float x, float a, float b) {
  return expf(__fadd_rn(__fmul_rn(a, x), b));
}
__device__ __forceinline__ double ea(double x, double a, double b) {
  double v[1] = {__dadd_rn(__dmul_rn(a, x), b)};
  exp_vec(v);
  return v[0];
}
template <int N>
__device__ __forceinline__ void ea_vec(float (&x)[N], float a, float b) {
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = ea(x[i], a, b);
}
template <int N>
__device__ __forceinline__ void ea_vec(double (&x)[N], double a, double b) {
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = __dadd_rn(__dmul_rn(a, x[i]), b);
  exp_vec(x);
}

template <typename T>
__global__ void __launch_bounds__(256)
    exp_affine_vec(const T* __restrict__ x, int64_t n, T a, T b, T* __restrict__ y) {
  using V = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
  constexpr int PER = 16 / sizeof(T);
  constexpr int UNROLL = sizeof(T) == 4 ? 4 : 2;
  exp_table_init<T>(true);
  const int64_t nv = n / PER;
  const V* xv = reinterpret_cast<const V*>(x);
  V* yv = reinterpret_cast<V*>(y);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  for (; i + (UNROLL - 1) * stride < nv; i += UNROLL * stride) {
    T e[UNROLL * PER];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const V v = __ldcs(xv + i + u * stride);
      memcpy(e + u * PER, &v, 16);
    }
    // (f64: one group of chains for all vectors; f32 stores each as it is
    // ready: 3480 x 4050 21.9 -> 21.5 us)
    if constexpr (sizeof(T) == 8) ea_vec(e, a, b);
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      if constexpr (sizeof(T) == 4) ea_vec(reinterpret_cast<T(&)[PER]>(e[u * PER]), a, b);
      V v;
      memcpy(&v, e + u * PER, 16);
      __stcs(yv + i + u * stride, v);
    }
  }
  for (; i < nv; i += stride) {
    V v = __ldcs(xv + i);
    T e[PER];
    memcpy(e, &v, 16);
    ea_vec(e, a, b);
    memcpy(&v, e, 16);
    __stcs(yv + i, v);
  }
  // scalar tail
  const int64_t t = nv * PER + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t < n) y[t] = ea(x[t], a, b);
}

template <typename T>
__global__ void exp_affine_scalar(const T* __restrict__ x, int64_t n, T a, T b, T* __restrict__ y) {
  exp_table_init<T>(true);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    y[i] = ea(x[i], a, b);
}

template <typename T>
int launch_exp_affine(nrs_handle* h, int64_t n, const T* x, T a, T b, T* y) {
  if (n == 0) return NRS_OK;
  const bool aligned = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
  int grid = h->num_sms * 8;
  if (aligned) {
    int64_t nv = n / (16 / (int64_t)sizeof(T));
    int64_t need = (nv + 255) / 256;
    if (need < grid) grid = (int)(need > 0 ? need : 1);
    exp_affine_vec<T><<<grid, 256, 0, h->stream>>>(x, n, a, b, y);
  } else {
    exp_affine_scalar<T><<<grid, 256, 0, h->stream>>>(x, n, a, b, y);
  }
  return nrs_after_launch(h, "exp_affine");
}

enum class Access { kFlat, kRowsVec, kStrided };

// Picks the access pattern: flat vectors, vector row walks, scalar row walks,
// or a full decode.
template <typename T, typename Eval>
int launch_eval(nrs_handle* h, const Eval& ev, const Geometry& g, int64_t n, Access acc, void* out) {
  if (n == 0) return NRS_OK;
  const int cap = h->num_sms * 8;
  if (acc == Access::kFlat) {
    const int64_t per_block = 256 * (int64_t)Eval::kUnroll;
    const int64_t need = (n / (16 / (int64_t)sizeof(T)) + per_block - 1) / per_block + 1;
    const int grid = (int)(need < cap ? need : cap);
    ufunc_flat_vec<T, Eval><<<grid, 256, 0, h->stream>>>(ev, g, n, (T*)out);
    return nrs_after_launch(h, "ufunc_flat_vec");
  }
  if (acc == Access::kRowsVec) {
    const int64_t rows = n / g.shape[g.ndim - 1];
    const int grid = (int)(rows < (int64_t)h->num_sms * 16 ? rows : (int64_t)h->num_sms * 16);
    ufunc_rows_vec<T, Eval><<<grid, 256, 0, h->stream>>>(ev, g, rows, (T*)out);
    return nrs_after_launch(h, "ufunc_rows_vec");
  }
  if (g.ndim >= 1 && g.shape[g.ndim - 1] >= 256) {
    const int64_t rows = n / g.shape[g.ndim - 1];
    const int grid = (int)(rows < (int64_t)h->num_sms * 16 ? rows : (int64_t)h->num_sms * 16);
    ufunc_rows<T, Eval><<<grid, 256, 0, h->stream>>>(ev, g, rows, (T*)out);
    return nrs_after_launch(h, "ufunc_rows");
  }
  const int64_t need = (n + 255) / 256;
  const int grid = (int)(need < (int64_t)h->num_sms * 16 ? need : (int64_t)h->num_sms * 16);
  ufunc_decode<T, Eval><<<grid, 256, 0, h->stream>>>(ev, g, n, (T*)out);
  return nrs_after_launch(h, "ufunc_decode");
}

// The same value with fewer operations and stack moves: a binary operation
// whose operands are the same subprogram evaluates it once (d*d of a squared
// difference), an f64 multiplication by a scalar +-2^k becomes an exponent
// add, and an input, scalar or duplicate that an operation consumes at once is
// part of it. Bits do not change. Returns the program's depth. Measured,
// 8192^2 f64 exp((x - mu)^2 * -0.5): 10 codes to 5.
int optimise(Prog& p, bool f64) {
  Prog q{};
  q.has_exp = p.has_exp;
  auto put = [&](int code, int32_t arg, double scalar) {
    q.code[q.len] = code;
    q.arg[q.len] = arg;
    q.scalar[q.len] = scalar;
    ++q.len;
  };
  int start[kStack + 1], depth = 0;  // first code of each stack value in q
  auto same = [&](int a, int b, int n) {
    for (int i = 0; i < n; ++i)
      if (q.code[a + i] != q.code[b + i] || q.arg[a + i] != q.arg[b + i] ||
          std::memcmp(&q.scalar[a + i], &q.scalar[b + i], sizeof(double)) != 0)
        return false;
    return true;
  };
  auto power = [&](int at, int* k) {  // a normal +-2^k scalar
    if (!f64 || q.code[at] != NRS_OP_SCALAR) return false;
    const double s = q.scalar[at];
    const double m = std::frexp(s, k);
    --*k;
    return std::fabs(m) == 0.5 && *k >= -1022 && *k <= 1023;
  };
  for (int i = 0; i < p.len; ++i) {
    const int c = p.code[i];
    if (c == NRS_OP_INPUT || c == NRS_OP_SCALAR) {
      start[depth++] = q.len;
      put(c, p.arg[i], p.scalar[i]);
      continue;
    }
    if (c >= NRS_OP_NEG && c <= NRS_OP_LN) {
      put(c, p.arg[i], p.scalar[i]);
      continue;
    }
    const int l = start[depth - 2], r = start[depth - 1], nl = r - l, nr = q.len - r;
    int k;
    --depth;
    if (c == NRS_OP_MUL && nr == 1 && power(r, &k)) {
      const double s = q.scalar[r];
      --q.len;
      put(NRS_OP_X_SCALE2, k, s);
    } else if (c == NRS_OP_MUL && nl == 1 && power(l, &k)) {
      const double s = q.scalar[l];
      for (int t = l; t + 1 < q.len; ++t) {
        q.code[t] = q.code[t + 1];
        q.arg[t] = q.arg[t + 1];
        q.scalar[t] = q.scalar[t + 1];
      }
      --q.len;
      put(NRS_OP_X_SCALE2, k, s);
    } else if (nl == nr && same(l, r, nl)) {
      q.len = r;
      put(NRS_OP_X_SELF + c, 0, 0.0);
    } else if (nr == 1 && q.code[r] == NRS_OP_INPUT) {
      q.code[r] = NRS_OP_X_IN + 4 * c + q.arg[r];
    } else if (nr == 1 && q.code[r] == NRS_OP_SCALAR) {
      q.code[r] = NRS_OP_X_SCALAR + c;
    } else {
      put(c, p.arg[i], p.scalar[i]);
    }
  }
  int d = 0, most = 0;
  for (int i = 0; i < q.len; ++i) {
    const int c = q.code[i];
    if (c == NRS_OP_INPUT || c == NRS_OP_SCALAR) ++d;
    else if (is_binary(c)) --d;
    most = d > most ? d : most;
  }
  p = q;
  return most;
}

template <typename T, bool EXP64>
int launch_depth(nrs_handle* h, const Prog& p, int depth, const Geometry& g, int64_t n, Access flat, void* out) {
  if (depth <= 2 && g.n_inputs <= 2) return launch_eval<T>(h, ProgEval<T, 2, 2, EXP64>{p}, g, n, flat, out);
  if (depth <= 2 && g.n_inputs == 3) return launch_eval<T>(h, ProgEval<T, 2, 3, EXP64>{p}, g, n, flat, out);
  if (depth <= 4) return launch_eval<T>(h, ProgEval<T, 4, kMaxIn, EXP64>{p}, g, n, flat, out);
  return launch_eval<T>(h, ProgEval<T, kStack, kMaxIn, EXP64>{p}, g, n, flat, out);
}

// Dispatch on the program's shape: a lone binary op gets its own functor.
template <typename T>
int launch_program(nrs_handle* h, Prog& p, int depth, const Geometry& g, int64_t n, Access flat,
                   void* out) {
  if (g.n_inputs > kMaxIn) {
    const int64_t need = (n + 255) / 256;
    const int grid = (int)(need < (int64_t)h->num_sms * 16 ? need : (int64_t)h->num_sms * 16);
    ufunc_generic<T><<<grid, 256, 0, h->stream>>>(p, g, n, (T*)out);
    return nrs_after_launch(h, "ufunc_generic");
  }
  if (p.len == 3 && p.code[0] == NRS_OP_INPUT && p.arg[0] == 0 && p.code[1] == NRS_OP_INPUT &&
      p.arg[1] == 1) {
    switch (p.code[2]) {
      case NRS_OP_ADD: return launch_eval<T>(h, BinEval<T, NRS_OP_ADD>{}, g, n, flat, out);
      case NRS_OP_SUB: return launch_eval<T>(h, BinEval<T, NRS_OP_SUB>{}, g, n, flat, out);
      case NRS_OP_MUL: return launch_eval<T>(h, BinEval<T, NRS_OP_MUL>{}, g, n, flat, out);
      case NRS_OP_DIV: return launch_eval<T>(h, BinEval<T, NRS_OP_DIV>{}, g, n, flat, out);
      default: break;
    }
  }
  if constexpr (std::is_floating_point<T>::value) {
    if (p.len == 2 && p.code[0] == NRS_OP_INPUT && p.arg[0] == 0) {
      switch (p.code[1]) {
        case NRS_OP_EXP: return launch_eval<T>(h, UnEval<T, NRS_OP_EXP>{}, g, n, flat, out);
        case NRS_OP_LN: return launch_eval<T>(h, UnEval<T, NRS_OP_LN>{}, g, n, flat, out);
        case NRS_OP_SQRT: return launch_eval<T>(h, UnEval<T, NRS_OP_SQRT>{}, g, n, flat, out);
        default: break;
      }
    }
  }
  depth = optimise(p, std::is_same<T, double>::value);
  if constexpr (std::is_same<T, double>::value) {
    if (p.has_exp) return launch_depth<T, true>(h, p, depth, g, n, flat, out);
  }
  return launch_depth<T, false>(h, p, depth, g, n, flat, out);
}

}  // namespace

extern "C" int nrs_exp_affine(nrs_handle* h, int dtype, int64_t n, const void* x, double a,
                              double b, void* y) {
  if (!h || n < 0 || (n && (!x || !y))) return NRS_ERR_INVALID;
  h->last_error.clear();
  int st = nrs_cuda_check(h, cudaSetDevice(h->device), "cudaSetDevice");
  if (st) return st;
  if (dtype == NRS_F32)
    return launch_exp_affine<float>(h, n, (const float*)x, (float)a, (float)b, (float*)y);
  if (dtype == NRS_F64)
    return launch_exp_affine<double>(h, n, (const double*)x, a, b, (double*)y);
  return nrs_fail(h, NRS_ERR_DTYPE, "exp needs f32 or f64");
}

extern "C" int nrs_ufunc(nrs_handle* h, int dtype, const nrs_ufunc_op* prog, int prog_len,
                         int ndim, const int64_t* shape, int n_inputs, const void* const* inputs,
                         const int64_t* in_strides, void* out, const int64_t* out_strides) {
  if (!h) return NRS_ERR_INVALID;
  h->last_error.clear();
  if (!prog || prog_len < 1 || prog_len > NRS_UFUNC_MAX_OPS)
    return nrs_fail(h, NRS_ERR_INVALID, "program length must be 1..32");
  if (ndim < 0 || ndim > NRS_UFUNC_MAX_DIMS || (ndim && !shape))
    return nrs_fail(h, NRS_ERR_INVALID, "bad ndim/shape");
  if (n_inputs < 0 || n_inputs > NRS_UFUNC_MAX_INPUTS || (n_inputs && (!inputs || (ndim && !in_strides))))
    return nrs_fail(h, NRS_ERR_INVALID, "bad inputs");
  const size_t es = nrs_dtype_size(dtype);
  if (!es) return nrs_fail(h, NRS_ERR_DTYPE, "unknown dtype");
  const bool is_int = (dtype == NRS_I32 || dtype == NRS_I64);
  // Validate the program: stack discipline, input indices, dtype support.
  Prog p{};
  p.len = prog_len;
  int depth = 0, max_depth = 0;
  for (int i = 0; i < prog_len; ++i) {
    const int c = prog[i].code;
    p.code[i] = c;
    p.arg[i] = prog[i].arg;
    p.scalar[i] = prog[i].scalar;
    if (c == NRS_OP_EXP) p.has_exp = 1;
    if (c == NRS_OP_INPUT) {
      if (prog[i].arg < 0 || prog[i].arg >= n_inputs)
        return nrs_fail(h, NRS_ERR_INVALID, "program reads a missing input");
      ++depth;
    } else if (c == NRS_OP_SCALAR) {
      ++depth;
    } else if (c >= NRS_OP_NEG && c <= NRS_OP_LN) {
      if (depth < 1) return nrs_fail(h, NRS_ERR_INVALID, "stack underflow");
      if (is_int && c >= NRS_OP_SQRT) return nrs_fail(h, NRS_ERR_DTYPE, "sqrt/exp/ln need f32/f64");
    } else if (is_binary(c)) {
      if (depth < 2) return nrs_fail(h, NRS_ERR_INVALID, "stack underflow");
      --depth;
    } else {
      return nrs_fail(h, NRS_ERR_INVALID, "unknown op code");
    }
    if (depth > kStack) return nrs_fail(h, NRS_ERR_INVALID, "stack deeper than 8");
    if (depth > max_depth) max_depth = depth;
  }
  if (depth != 1) return nrs_fail(h, NRS_ERR_INVALID, "program must leave exactly one value");
  int64_t n = 1;
  for (int d = 0; d < ndim; ++d) {
    if (shape[d] < 0) return nrs_fail(h, NRS_ERR_SHAPE, "negative dimension");
    n *= shape[d];
  }
  if (n == 0) return NRS_OK;
  if (!out) return nrs_fail(h, NRS_ERR_INVALID, "null output");
  Geometry g{};
  g.ndim = ndim;
  g.n_inputs = n_inputs;
  int64_t contig = 1;
  for (int d = ndim - 1; d >= 0; --d) {
    g.shape[d] = shape[d];
    g.out_stride[d] = out_strides ? out_strides[d] : contig;
    if (g.out_stride[d] < 0) return nrs_fail(h, NRS_ERR_STRIDE, "negative stride");
    contig *= shape[d];
  }
  bool all_contig = (out_strides == nullptr);
  for (int k = 0; k < n_inputs; ++k) {
    if (!inputs[k]) return nrs_fail(h, NRS_ERR_INVALID, "null input");
    g.in[k] = inputs[k];
    int64_t c = 1;
    for (int d = ndim - 1; d >= 0; --d) {
      int64_t s = in_strides[(size_t)k * ndim + d];
      if (s < 0) return nrs_fail(h, NRS_ERR_STRIDE, "negative stride");
      g.in_stride[k][d] = s;
      if (shape[d] != 1 && s != c) all_contig = false;
      c *= shape[d];
    }
  }
  int st = nrs_cuda_check(h, cudaSetDevice(h->device), "cudaSetDevice");
  if (st) return st;
  // The fused affine-exp program on contiguous data takes the vectorised path.
  if (all_contig && n_inputs == 1 && prog_len == 6 && prog[0].code == NRS_OP_INPUT &&
      prog[1].code == NRS_OP_SCALAR && prog[2].code == NRS_OP_MUL &&
      prog[3].code == NRS_OP_SCALAR && prog[4].code == NRS_OP_ADD && prog[5].code == NRS_OP_EXP &&
      (dtype == NRS_F32 || dtype == NRS_F64)) {
    // (x * a) rounds the same as (a * x): IEEE multiplication is commutative.
    return nrs_exp_affine(h, dtype, n, inputs[0], prog[1].scalar, prog[3].scalar, out);
  }
  // Same-shape contiguous operands, all 16-byte aligned: flat vector path.
  // Otherwise rows of 16-byte vectors when the last dimension is unit-stride
  // (or broadcast) everywhere and every row starts 16-byte aligned.
  Access flat = Access::kStrided;
  uintptr_t align = reinterpret_cast<uintptr_t>(out);
  for (int k = 0; k < n_inputs; ++k) align |= reinterpret_cast<uintptr_t>(inputs[k]);
  if (all_contig && (align & 15) == 0) {
    flat = Access::kFlat;
  } else if (ndim >= 1 && (align & 15) == 0 && g.shape[ndim - 1] >= 64 &&
             (g.shape[ndim - 1] * (int64_t)es) % 16 == 0 && g.out_stride[ndim - 1] == 1) {
    bool ok = true;
    for (int d = 0; d < ndim - 1; ++d)
      if (g.shape[d] > 1 && (g.out_stride[d] * (int64_t)es) % 16 != 0) ok = false;
    for (int k = 0; k < n_inputs && ok; ++k) {
      const int64_t ls = g.in_stride[k][ndim - 1];
      if (ls > 1) ok = false;
      for (int d = 0; d < ndim - 1 && ok; ++d)
        if (ls == 1 && g.shape[d] > 1 && (g.in_stride[k][d] * (int64_t)es) % 16 != 0) ok = false;
    }
    if (ok) flat = Access::kRowsVec;
  }
  switch (dtype) {
    case NRS_F32: return launch_program<float>(h, p, max_depth, g, n, flat, out);
    case NRS_F64: return launch_program<double>(h, p, max_depth, g, n, flat, out);
    case NRS_I64: return launch_program<int64_t>(h, p, max_depth, g, n, flat, out);
    default: return launch_program<int32_t>(h, p, max_depth, g, n, flat, out);
  }
}
