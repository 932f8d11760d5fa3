"""Slice pairs that the slice GEMM does not multiply count in its choice of a
slice count. Operands that show them: one large entry in every row of A and
in every column of B, at k that they do not share, and small entries, alike
for every k, at all others. The small entries' digits are then the same for
every k, and what the pairs with s + t >= S leave out adds up.

Bounds, relative to (|A||B|)_ij in units u of the element type (2^-53,
2^-24): 1 (f32: 1/4) for the operands' rounding and tau for the pairs left
out, tau = 7 where the call chooses the slices by itself and 0.24 K + 4 where
the caller asks for them (measured to a percent or two: 8 and K / 4 + 4); 1 for
the product's rounding and, with K in up to 16 ranges, 15 for their sum in
f64.
"""
import ctypes
import math
import os
import random
import shutil
import subprocess
from fractions import Fraction as F

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "numrs_gb300", "csrc")
HARNESS = r"""
#include "f64_round.cuh"
extern "C" int nrs_test_holds(int S, int b, int target, float spread, float drop) {
  return ozaki_count_holds(S, b, target, spread, drop);
}
extern "C" float nrs_test_units(int target, double k, int asked) {
  return asked ? ozaki_drop_units_asked(target, k) : ozaki_drop_units(target);
}
extern "C" void nrs_test_digits(double x, int e, int S, int* d) {
  const OzakiZ64 z = ozaki_z64(x, e, 8, S, ozaki_offset64(S, 8));
  for (int t = 0; t < S; ++t) d[t] = ozaki_digit64<8>(z, t);
}
"""
# (K, entry of A, entry of B, f32): errors of 230 to 6500 u where only the spread decides the count
CASES = [(4096, 3e-6, 3e-6, False), (512, 1e-5, 1e-5, False), (512, 1.871e-5, 4.049e-6, False),
         (2048, 2.346025939914398e-05, 2.346025939914398e-05, True),
         (2048, 2.659886195033323e-05, 2.659886195033323e-05, True)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("dropped")
    (d / "h.cpp").write_text(HARNESS)
    so = d / "h.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "h.cpp"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.nrs_test_holds.argtypes = [ctypes.c_int] * 3 + [ctypes.c_float] * 2
    lib.nrs_test_units.argtypes = [ctypes.c_int, ctypes.c_double, ctypes.c_int]
    lib.nrs_test_units.restype = ctypes.c_float
    lib.nrs_test_digits.argtypes = [ctypes.c_double, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int)]
    return lib


def _digits(x, S):
    """8-bit signed digits of the scaled operand x (a Fraction below 1), any S."""
    y = math.floor(x * 2 ** (8 * S - 1) + F(1, 2))
    d = []
    for _ in range(S - 1):
        r = (y + 128) % 256 - 128
        d.append(r)
        y = (y - r) // 256
    return [y] + d[::-1]


def _kept(a, b, S):
    """The slices' product of one k."""
    da, db = _digits(a, S), _digits(b, S)
    return sum(F(da[s] * db[t], 1 << (14 + 8 * (s + t))) for s in range(S) for t in range(S - s))


def test_pairs_left_out_stay_within_their_bound(lib):
    r = random.Random(1)
    for i in range(3000):
        S = r.randint(1, 8)
        x, y = (r.uniform(-1, 1) * 2.0 ** -r.choice([0, 3, 9, 17, 30, 60]) for _ in range(2))
        if i % 3 == 0:  # digits of the largest magnitude
            x, y = (float(F(128, 255)) * 2.0 ** -r.choice([0, 8, 16, 24]) * r.choice([-1, 1]) for _ in range(2))
        d = (ctypes.c_int * 16)()
        lib.nrs_test_digits(x, 0, S, d)
        a, b = F(x), F(y)
        assert list(d[:S]) == _digits(a, S)
        # |a'| and |b'| for the rounding (the top digit may exceed |a'| by its own half unit, 2^-8)
        assert abs(_kept(a, b, S) - a * b) <= (abs(a) + F(1, 256) + abs(b) + S - 1) / 2 ** (8 * S)


@pytest.mark.parametrize("K,c1,c2,f32", CASES)
@pytest.mark.parametrize("asked", [False, True])
def test_count_rule(lib, K, c1, c2, f32, asked):
    target = 26 if f32 else 53
    c1, c2 = (float(np.float32(c)) if f32 else c for c in (c1, c2))
    n = K - 2
    D = n * c1 * c2 / 4  # (the large entries are 1: exponent 1)
    spread = (1 + n * (c1 + c2) / 2) / D
    tau = lib.nrs_test_units(target, K, int(asked))
    drop = K / D / tau
    count = [next(s for s in range(1, 16) if lib.nrs_test_holds(s, 8, target, spread, v)) for v in (0.0, drop)]
    err = [abs(float(n * (_kept(F(c1) / 2, F(c2) / 2, s) - F(c1) * F(c2) / 4)) / D) * 2.0 ** target for s in count]
    assert err[0] > 1 + tau      # the spread alone: too few slices
    assert err[1] <= 1 + tau


def _operands(K, c1, c2, dt, m, n, draw=None):
    import torch
    a, b = np.full(K, c1), np.full(K, c2)
    if draw is not None:
        a = b = np.random.default_rng(draw).uniform(0.5, 1.0, K) * c1
    a, b = (v.astype(np.float32 if dt == torch.float32 else np.float64) for v in (a.copy(), b.copy()))
    a[:2], b[:2] = (1, 0), (0, 1)
    exact = sum(F(float(x)) * F(float(y)) for x, y in zip(a, b))
    A = torch.from_numpy(a).cuda().expand(m, K).contiguous()
    B = torch.from_numpy(b).cuda()[:, None].expand(K, n).contiguous()
    return A, B, exact


def _units(c, exact, u):
    v = set(np.unique(c.cpu().numpy()).tolist())
    return max(abs(float((F(x) - exact) / exact)) for x in v) / u


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES + [(2048, 5.5e-6, None, False)])
def test_products_of_alike_small_entries(K, case):
    import torch
    k, c1, c2, f32 = case
    dt, u = (torch.float32, 2.0 ** -24) if f32 else (torch.float64, 2.0 ** -53)
    m = 1536 if f32 else 512
    A, B, exact = _operands(k, c1, c2, dt, m, m, draw=5 if c2 is None else None)
    assert _units(K.matmul(A, B), exact, u) <= (8 + 0.25 + 1.01 if f32 else 1 + 8 + 16)
    asked = k / 4 + 4 + 2
    if f32:
        c = torch.zeros((130, 140), dtype=dt, device="cuda")
        plan = K.Plan([(A[:130].contiguous(), B[:, :140].contiguous(), c, False)], f32_mode=1)
        plan.run()
        assert plan.f32_info()[0] == 1
        assert _units(c, exact, u) <= asked
    else:
        c, info = K.gemm_ozaki(A[:130].contiguous(), B[:, :140].contiguous())
        assert info["slices"] > 0
        assert _units(c, exact, u) <= asked
        assert _units(c, exact, u) * u <= info["est_rel_error"]
        c = torch.zeros((130, 140), dtype=dt, device="cuda")
        on, _ = K.gemm_ozaki_grouped([(A[:130].contiguous(), B[:, :140].contiguous(), c, False)])
        assert all(on) and _units(c, exact, u) <= asked
