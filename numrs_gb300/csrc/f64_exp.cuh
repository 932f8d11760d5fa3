// exp of doubles in fixed-point integer arithmetic.
//
// GB300's FP64 pipe retires about 1.7 operations per clock per SM, so a
// polynomial exp in FP64 arithmetic runs at 29 G elements/s (0.47 TB/s of
// reads and writes), while the integer pipes have 32 (multiply) and 64 (add,
// shift) lanes. This is the table method of P. T. P. Tang ("Table-driven
// implementation of the exponential function in IEEE floating-point
// arithmetic", ACM TOMS 15, 1989) carried out on 64-bit fractions:
//   y = x log2(e) = k + j / 256 + z / 256,   0 <= z < 1,
//   exp(x) = 2^k 2^(j/256) (1 + p),   1 + p = e^(z ln2 / 256),
// with y from a 64 x 96 bit product, 2^(j/256) from a table of 64-bit
// fractions and p from five terms of the series. Every step truncates:
// the dropped sixth term is below 2^-60.7 and all errors together below 2^-56
// of the result, so that it is within 0.63 ulp (the FP64 form it replaces is
// specified to 1 ulp).
// Arguments below 32 in magnitude take y from a 64 x 64 bit product with 57
// fraction bits (about 60 integer operations in all); the others, to the ends
// of the normal range, from a 64 x 96 bit product with 64 fraction bits.
// Host and device code, so that CPU tests check what the kernels run.
#pragma once
#include "f64_round.cuh"

constexpr int kNrsExpTable = 256;

NRS_HD uint32_t nrs_mulhi32(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
// The high 64 bits of a * b, less up to 2 (the low x low product is left out).
NRS_HD uint64_t nrs_mulhi64_down(uint64_t a, uint64_t b) {
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  return (uint64_t)ah * bh + ((uint64_t)nrs_mulhi32(ah, bl) + nrs_mulhi32(al, bh));
}

// 2^(j / 256) in units of 2^-63, the product of the square roots 2^(1/2),
// 2^(1/4), ... that j's bits select (rounded down; below by less than 8 units).
NRS_HD uint64_t nrs_exp_entry(int j) {
  const uint64_t root[8] = {0x8058d7d2d5e5f6b0ull, 0x80b1ed4fd999ab6cull, 0x8164d1f3bc030773ull,
                            0x82cd8698ac2ba1d7ull, 0x85aac367cc487b14ull, 0x8b95c1e3ea8bd6e6ull,
                            0x9837f0518db8a96full, 0xb504f333f9de6484ull};  // 2^(2^b / 256)
  uint64_t t = 1ull << 63;
  for (int b = 0; b < 8; ++b)
    if ((j >> b) & 1) t = (uint64_t)(((unsigned __int128)t * root[b]) >> 63);
  return t;
}

// 2^k 2^(j/256) (1 + p) for z = zh:zl 2^-64, -1022 <= k <= 1023; t = the
// table's entry j. p 2^72 from c_i = (ln2 / 256)^i / i!: the third to fifth
// terms in 32-bit fractions of 2^-60, the first two in 64-bit fractions of
// 2^-72.
NRS_HD double nrs_exp_finish(int k, uint64_t t, uint32_t zh, uint32_t zl) {
  const uint64_t z = (uint64_t)zh << 32 | zl;
  const uint32_t q3 = nrs_mulhi32(nrs_mulhi32(0x00000576u, zh) + 0x00276556u, zh) + 0xe35846b8u;
  const uint64_t q2 = (((uint64_t)q3 * zh) >> 20) + 0x003d7f7bff058b1dull;
  const uint64_t q1 = nrs_mulhi64_down(q2, z) + 0xb17217f7d1cf79abull;
  const uint64_t p = nrs_mulhi64_down(q1, z);
  const uint64_t r = t + (nrs_mulhi64_down(t, p) >> 8);  // [2^63, 2^64)
  // 53 bits, the leading one adding 1 to the exponent field
  return nrs_f64_from_bits(((uint64_t)(uint32_t)(k + 1022) << 52) + (r >> 11) + ((r >> 10) & 1));
}

// exp(x) for |x| < 32; otherwise sets `far` and the value is meaningless.
NRS_HD double nrs_exp_near(double x, const uint64_t* table, bool& far) {
  uint64_t bits;
  memcpy(&bits, &x, sizeof bits);
  const uint32_t hi = (uint32_t)(bits >> 32);
  const uint32_t s = 1028u - ((hi >> 20) & 0x7FFu);  // 1 or more when near
  // |x| = m 2^(5 - s - 63) (the implicit one is wrong for zeros and
  // subnormals, whose y is 0 either way); y 2^57 = m log2(e) >> s, log2(e) in
  // units of 2^-63
  const uint64_t m = bits << 11 | 1ull << 63;
  uint64_t y = nrs_mulhi64_down(m, 0xb8aa3b295c17f0bbull);
  y = s < 64 ? y >> (s & 63) : 0;
  y = (int32_t)hi < 0 ? 0 - y : y;
  far = (int32_t)s <= 0;
  const uint32_t y1 = (uint32_t)(y >> 32), y0 = (uint32_t)y;
  return nrs_exp_finish((int32_t)y1 >> 25, table[(y1 >> 17) & 255u], nrs_shl_funnel(y0, y1, 15), y0 << 15);
}

// exp(x) for results that are normal; otherwise (overflow, a subnormal or zero
// result, Inf, NaN) sets `special` and the value is meaningless. `table`:
// kNrsExpTable entries of nrs_exp_entry.
NRS_HD double nrs_exp_fixed(double x, const uint64_t* table, bool& special) {
  uint64_t bits;
  memcpy(&bits, &x, sizeof bits);
  const uint32_t hi = (uint32_t)(bits >> 32), lo = (uint32_t)bits;
  const uint32_t be = (hi >> 20) & 0x7FFu;
  // |x| = mh:ml 2^(be - 1023 - 63) (the implicit one is wrong for zeros and
  // subnormals, whose y is 0 either way)
  const uint32_t mh = 0x80000000u | nrs_shl_funnel(lo, hi, 11), ml = lo << 11;
  // log2(e) = l2:l1:l0 2^-95; w4:w3:w2 = the product's words, 2^-94
  constexpr uint32_t l2 = 0xb8aa3b29u, l1 = 0x5c17f0bbu, l0 = 0xbe87fed0u;
  const uint64_t t1 = (uint64_t)mh * l1 + ((uint64_t)nrs_mulhi32(mh, l0) + nrs_mulhi32(ml, l1));
  const uint64_t t2 = (uint64_t)ml * l2 + (uint32_t)t1;
  const uint64_t top = (uint64_t)mh * l2 + (t1 >> 32) + (t2 >> 32);
  // y 2^64 = w >> (1053 - be); |x| < 2^10 keeps that shift at 21 or more
  const uint32_t s = 1053u - be;
  uint32_t x2 = (uint32_t)(top >> 32), x1 = (uint32_t)top, x0 = (uint32_t)t2;
  if (s >= 32) {
    const bool a = s >= 64, c = s >= 96;
    x0 = c ? 0u : a ? x2 : x1;
    x1 = a ? 0u : x2;
    x2 = 0;
  }
  const int n = (int)(s & 31);
  uint32_t f0 = nrs_shr_funnel(x0, x1, n), f1 = nrs_shr_funnel(x1, x2, n);
  int k = (int)(x2 >> n);
  if ((int32_t)hi < 0) {  // floor(-y)
    const uint64_t f = 0 - ((uint64_t)f1 << 32 | f0);
    k = ~k + (f == 0);
    f1 = (uint32_t)(f >> 32);
    f0 = (uint32_t)f;
  }
  special = (be > 1032u) | ((uint32_t)(k + 1022) > 2045u);
  return nrs_exp_finish(k, table[f1 >> 24], nrs_shl_funnel(f0, f1, 8), f0 << 8);
}
