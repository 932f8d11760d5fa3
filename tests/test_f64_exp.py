"""The fixed-point f64 exp (numrs_gb300/csrc/f64_exp.cuh), compiled for the
host, against 40-digit decimal arithmetic over the whole range and near 0;
arguments it must leave to the general function. GPU: every access path of
the ufunc kernels against numpy's exp, and programs that the launcher
rewrites (a squared difference, power-of-two scalars) against the same
operations one by one, bit for bit."""
import ctypes
import decimal
import math
import os
import random
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "numrs_gb300", "csrc")

HARNESS = r"""
#include "f64_exp.cuh"
// as the kernels: the near form where it applies, else the whole-range form
extern "C" double nrs_test_exp(double x, int* special) {
  static uint64_t table[kNrsExpTable];
  if (!table[0]) for (int j = 0; j < kNrsExpTable; ++j) table[j] = nrs_exp_entry(j);
  bool far, sp;
  const double near = nrs_exp_near(x, table, far), r = nrs_exp_fixed(x, table, sp);
  *special = sp;
  return far ? r : near;
}
extern "C" int nrs_test_exp_near(double x) {
  uint64_t table[kNrsExpTable] = {};
  bool far;
  nrs_exp_near(x, table, far);
  return !far;
}
"""


@pytest.fixture(scope="module")
def fixed(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("f64exp")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "h.cpp"), "-o",
                    str(d / "h.so")], check=True)
    dll = ctypes.CDLL(str(d / "h.so"))
    dll.nrs_test_exp.restype = ctypes.c_double
    dll.nrs_test_exp.argtypes = [ctypes.c_double, ctypes.POINTER(ctypes.c_int)]

    def f(x):
        sp = ctypes.c_int(0)
        return dll.nrs_test_exp(x, ctypes.byref(sp)), sp.value
    f.near = dll.nrs_test_exp_near
    f.near.argtypes = [ctypes.c_double]
    return f


def test_near_form_covers_32(fixed):
    for x in (0.0, -0.0, 5e-324, 1e-300, 1.0, -31.9, math.nextafter(32.0, 0.0), -math.nextafter(32.0, 0.0)):
        assert fixed.near(x), x
    for x in (32.0, -32.0, 1e300, float("inf"), float("nan")):
        assert not fixed.near(x), x


def test_error_below_063_ulp(fixed):
    decimal.getcontext().prec = 40
    r = random.Random(2)
    for i in range(6000):
        x = [r.uniform(-708, 709.7), r.uniform(-3, 3), r.uniform(-1, 1) * 2.0 ** -r.randrange(70),
             r.randrange(-700, 700) + r.choice([-1, 0, 1]) * 2.0 ** -r.randrange(60)][i % 4]
        got, sp = fixed(x)
        assert not sp, x
        want = decimal.Decimal(x).exp()
        ulp = decimal.Decimal(math.ulp(float(want)))
        assert abs(decimal.Decimal(got) - want) <= decimal.Decimal("0.63") * ulp, x


def test_defers_and_exact_values(fixed):
    for x in (float("inf"), float("-inf"), float("nan"), 709.8, 1e300, -708.5, -745.2, -1e300, 1024.0, -1024.0):
        assert fixed(x)[1] == 1, x
    for x in (0.0, -0.0, 5e-324, -5e-324, 1e-300, 1e-20, -1e-20):
        assert fixed(x) == (1.0, 0), x


def _values():
    r = np.random.default_rng(3)
    x = np.concatenate([r.uniform(-745, 710, 4000), r.normal(0, 1, 4000), r.uniform(-1, 1, 1000) * 1e-17,
                        [0.0, -0.0, np.inf, -np.inf, np.nan, 709.8, -708.5, -745.2, -746.0, 5e-324, 1e300, -1e300]])
    return x


@pytest.mark.gpu
def test_gpu_every_access_path(K):
    import torch
    x = _values()
    want = np.exp(x)
    dev = torch.from_numpy(x).cuda()
    flat = K.exp(dev)
    got = flat.cpu().numpy()
    fin = np.isfinite(want)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    np.testing.assert_array_equal(got[~fin & ~np.isnan(want)], want[~fin & ~np.isnan(want)])
    # 0.63 ulp here, below 1 ulp in numpy's: at most 1 ulp apart (2 where a
    # subnormal result comes from CUDA's exp)
    ulps = np.abs(got[fin] - want[fin]) / np.spacing(np.maximum(want[fin], 5e-324))
    assert ulps.max() <= 2 and ulps[want[fin] > 1e-300].max() <= 1
    n = x.size // 3 * 3
    base = torch.zeros(2 * n + 1, dtype=torch.float64, device="cuda")
    views = []
    strided = base[:2 * n:2]          # scalar row walk
    strided.copy_(dev[:n])
    views.append(strided)
    off = base.clone()[1:n + 1]       # unaligned
    off.copy_(dev[:n])
    views.append(off)
    views.append(dev[:n].view(3, n // 3).t().contiguous().t())  # decode / rows
    ref = flat[:n]
    for v in views:
        assert torch.equal(K.exp(v).reshape(-1).view(torch.int64), ref.view(torch.int64))
    one = K.exp_affine(dev[:n].contiguous(), 1.0, 0.0)
    assert torch.equal(one.view(torch.int64), ref.view(torch.int64))
    for m in (1, 2, 3, 7, 512, 513, 4097):
        assert torch.equal(K.exp(dev[:m].clone()).view(torch.int64), flat[:m].view(torch.int64))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("shape", [(1, 64), (37, 130), (513, 1000), (5, 3, 7)])
def test_gpu_rewritten_programs_keep_every_bit(K, dtype, shape):
    import torch
    dt = getattr(torch, dtype)
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(shape, dtype=dt, device="cuda", generator=g)
    x.view(-1)[:6] = torch.tensor([0.0, -0.0, float("inf"), float("nan"), 1e-320, 1e-38], dtype=dt)
    mu = torch.randn(shape[-1], dtype=dt, device="cuda", generator=g)
    leaf = K.Expr.leaf

    def const(s):
        return torch.tensor([s], dtype=torch.float64).to(dt).cuda()  # (f32: out of range is Inf, as the cast is)
    d = K.subtract(x, mu)
    dd = K.multiply(d, d)
    e = leaf(x) - leaf(mu)
    bits = torch.int64 if dt == torch.float64 else torch.int32

    def same(a, b):
        assert torch.equal(a.contiguous().view(bits), b.contiguous().view(bits))
    same((e * e).eval(), dd)
    same((e * e * -0.5).eval(), K.multiply(dd, const(-0.5)))
    same((0.25 * (e * e)).eval(), K.multiply(const(0.25), dd))
    same((e * 2.0 ** -1040).eval(), K.multiply(d, const(2.0 ** -1040)))
    same((e * 2.0 ** 1000 * 2.0 ** 40).eval(), K.multiply(K.multiply(d, const(2.0 ** 1000)), const(2.0 ** 40)))
    same((e * 3.0).eval(), K.multiply(d, const(3.0)))
    same(((e * e) - (e * e)).eval(), K.subtract(dd, dd))
    same(((e + 1.0) / (e + 2.0)).eval(), K.divide(K.add(d, const(1.0)), K.add(d, const(2.0))))
    same((e * e * -0.5).exp().eval(), K.exp(K.multiply(dd, const(-0.5))))
