"""Integer forms of floating-point steps, compiled for the host: the slice
GEMM's three-word rounding of an element's exact total (ozaki_round96),
bit-identical to the 128-bit exact path wherever it does not defer; the
slicing of f32 operands without a conversion (ozaki_decode), the same digits
as the widened value's; and the squared deviation of f64 variances
(nrs_square), the same bits as the product."""
import ctypes
import os
import random
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "numrs_gb300", "csrc")

HARNESS = r"""
#include "f64_round.cuh"
// Compares both formats for one element; returns the number of mismatches,
// *deferred counts the cases left to the exact path.
extern "C" int nrs_test_round96(int32_t R, uint64_t lo, int nd, int e, int* deferred) {
  bool neg, sp;
  uint64_t mhi, mlo;
  int bad = 0;
  ozaki_exact_total(R, lo, 0, 8, nd + 1, neg, mhi, mlo);
  const uint64_t F = nd ? lo << (64 - 8 * nd) : 0;
  uint64_t r = ozaki_round96<NrsF64Fmt>(R, (uint32_t)(F >> 32), (uint32_t)F, e + 8 * nd, sp);
  *deferred += sp;
  bad += !sp && r != int128_to_float_bits<NrsF64Fmt>(neg, mhi, mlo, e);
  r = ozaki_round96<NrsF32Fmt>(R, (uint32_t)(F >> 32), (uint32_t)F, e / 8 + 8 * nd, sp);
  bad += !sp && (uint32_t)r != (uint32_t)int128_to_float_bits<NrsF32Fmt>(neg, mhi, mlo, e / 8);
  return bad;
}
extern "C" int nrs_test_square(double x, int* special) {
  uint64_t u, w;
  memcpy(&u, &x, 8);
  bool sp;
  const uint64_t r = nrs_square(u, sp);
  *special = sp;
  const double d = x * x;
  memcpy(&w, &d, 8);
  return !sp && r != w;
}
extern "C" int nrs_test_f32_digits(float x, int e, int S) {
  const OzakiZ64 a = ozaki_z64(x, e, 8, S, ozaki_offset64(S, 8)), b = ozaki_z64((double)x, e, 8, S, ozaki_offset64(S, 8));
  int bad = 0;
  for (int t = 0; t < S; ++t) bad += ozaki_digit64<8>(a, t) != ozaki_digit64<8>(b, t);
  return bad;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("round96")
    src = d / "h.cpp"
    src.write_text(HARNESS)
    so = d / "h.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(src), "-o", str(so)], check=True)
    dll = ctypes.CDLL(str(so))
    dll.nrs_test_round96.argtypes = [ctypes.c_int32, ctypes.c_uint64, ctypes.c_int, ctypes.c_int,
                                     ctypes.POINTER(ctypes.c_int)]
    dll.nrs_test_f32_digits.argtypes = [ctypes.c_float, ctypes.c_int, ctypes.c_int]
    dll.nrs_test_square.argtypes = [ctypes.c_double, ctypes.POINTER(ctypes.c_int)]
    return dll


def test_round96_equals_exact_path(lib):
    r = random.Random(4)
    deferred = ctypes.c_int(0)
    n = 60000
    for _ in range(n):
        nd = r.randrange(9)
        lo = r.getrandbits(8 * nd) if nd else 0
        if r.random() < 0.3:  # ties and long zero tails
            lo &= (~0 << r.randrange(64)) & ((1 << 64) - 1)
        R = r.getrandbits(31) >> r.randrange(31)
        R = -R if r.random() < 0.5 else R
        if r.random() < 0.2:
            R = r.choice([0, -1, 1, -(1 << 31), (1 << 31) - 1])
        e = r.choice([r.randrange(-60, 60), r.randrange(-1300, 1200)])
        assert lib.nrs_test_round96(R, lo, nd, e, ctypes.byref(deferred)) == 0, (R, lo, nd, e)
    assert deferred.value < n // 4  # (it has to carry the ordinary case)


def test_f32_digits_equal_the_widened_value(lib):
    r = random.Random(6)
    for _ in range(20000):
        x = ctypes.c_float(r.uniform(-1, 1) * 2.0 ** r.randrange(-150, 100)).value
        e = max(-148, __import__("math").frexp(x)[1] + r.randrange(0, 12)) if x else 3
        assert lib.nrs_test_f32_digits(x, e, r.randrange(1, 9)) == 0, (x, e)


def test_square_equals_the_product(lib):
    r = random.Random(8)
    sp = ctypes.c_int(0)
    for _ in range(60000):
        m = r.getrandbits(53) | (1 << 52)
        if r.random() < 0.3:
            m = (m >> r.randrange(52) << r.randrange(52)) or 1
        x = float(m) * 2.0 ** r.randrange(-600, 400) * r.choice([-1, 1])
        assert lib.nrs_test_square(x, ctypes.byref(sp)) == 0, x
    for x, want in ((0.0, 1), (-0.0, 1), (float("inf"), 1), (float("nan"), 1), (1e200, 1), (1e-170, 1), (5e-324, 1),
                    (1.0, 0), (-1.5, 0), (1.3e154, 0), (1.6e-154, 0), (1.9999999999999998, 0)):
        assert lib.nrs_test_square(x, ctypes.byref(sp)) == 0 and sp.value == want, x
