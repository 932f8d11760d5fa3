"""Short flat reductions (one launch, a warp per chunk) give the bits of the
two-launch path: at the chunk tiers (one chunk below 10000 for sums, 40000
for variances, 8192 otherwise), unaligned views, NaNs, signed zeros and
extremes, against the oracle's order-exact cases and nrs_reduce_flat_noalloc,
which keeps the two-launch kernels."""
import ctypes as C

import numpy as np
import pytest
import torch

from numrs_gb300 import _lib as L
from tests.conftest import bits, to_np

pytestmark = pytest.mark.gpu

SIZES = [1, 7, 255, 256, 257, 1000, 8191, 8192, 8193, 9999, 10000, 16385, 39999, 40000, 65535, 65536, 65537, 131072,
         131073, 200000]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n", SIZES)
def test_bits_equal_the_two_launch_kernels(K, dtype, n):
    lib = L.load()
    code = L.F32 if dtype == torch.float32 else L.F64
    g = torch.Generator(device="cuda").manual_seed(n)
    base = torch.randn(n + 1, dtype=dtype, device="cuda", generator=g)
    nans = base.clone()
    nans[n // 2] = float("nan")
    zeros = -base.abs()
    zeros[::3], zeros[1::3] = 0.0, -0.0
    for buf in (base, nans, zeros, -zeros):
        for x in (buf[:n], buf[1:]):
            for op in (L.SUM, L.MEAN, L.MAX, L.MIN):
                want = torch.empty(1, dtype=dtype, device="cuda")
                assert lib.nrs_reduce_flat_noalloc(C.c_void_p(torch.cuda.current_stream().cuda_stream), code, op, n,
                                                   C.c_void_p(x.data_ptr()), C.c_void_p(want.data_ptr())) == L.OK
                got = K.reduce(x, op)
                assert np.array_equal(bits(to_np(got)), bits(to_np(want))), (op, n)


@pytest.mark.parametrize("n", SIZES)
def test_variance_product_and_integers(K, ora, n):
    r = np.random.default_rng(n)
    x = r.standard_normal(n) * 2 + 3
    d = torch.from_numpy(x).cuda()
    for name in ("var", "std"):
        if n > 1:
            got = float(getattr(K, name)(d, ddof=1))
            want = getattr(np, name)(x.astype(np.longdouble), ddof=1)
            # two passes of sums of n non-negative terms: n 2^-53, far below 1e-12 here
            assert abs(got - want) <= 1e-12 * want
    p = 1.0 + 1e-4 * r.standard_normal(n)
    got, want = float(K.prod(torch.from_numpy(p).cuda())), float(np.prod(p.astype(np.longdouble)))
    assert abs(got - want) <= n * 2.0 ** -52 * want
    for dt in (np.int64, np.int32):
        i = r.integers(-1000, 1000, n).astype(dt)
        di = torch.from_numpy(i).cuda()
        assert int(K.sum(di)) == int(i.sum()) and int(K.max(di)) == i.max() and int(K.min(di)) == i.min()
    i = r.integers(-1000, 1000, n).astype(np.int64)
    assert float(K.mean(torch.from_numpy(i).cuda())) == float(i.sum()) / n
