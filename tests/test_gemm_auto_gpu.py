"""f64 matmul through the call's own choice of kernel: products large enough
for the tensor cores run as slice GEMMs whose slice count is decided on the
device, the rest (and operands that the slices cannot carry) on the FP64
kernel.

Error bar against the double-double product, max |C - C_dd| / (|A||B|)_ij:
the slices keep 2^-53 of it, each of up to 16 K ranges is rounded once and
their sum rounds 15 times, so (1 + 16) 2^-53 < 2e-15.
"""
import numpy as np
import pytest
import torch

from numrs_gb300 import _lib as L
from tests.conftest import to_np

pytestmark = pytest.mark.gpu

BAR = 2e-15


def _operands(m, k, n, phi, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def one(r, c):
        u = torch.rand((r, c), dtype=torch.float64, device="cuda", generator=g) - 0.5
        return u * torch.exp(phi * torch.randn((r, c), dtype=torch.float64, device="cuda", generator=g))
    return one(m, k), one(k, n)


def _err(ora, c, a, b):
    Cdd, ab = ora.gemm_dd(to_np(a.contiguous()), to_np(b.contiguous()))
    return float(np.max(np.abs(to_np(c) - Cdd) / ab))


# one and several K ranges, tile edges in m and n, K padding, K past the 8-bit digits' exact range, more than 9 slices
# (the last: a product that is faster on the FP64 kernel and has its bits)
@pytest.mark.parametrize("mkn,phi,slices", [((384, 384, 384), 0.0, True), ((513, 449, 385), 1.0, True),
                                            ((129, 2047, 257), 0.0, True), ((1025, 129, 640), 4.0, True),
                                            ((64, 10249, 200), 0.0, True), ((3000, 500, 10), 1.0, False)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True)])
def test_auto_error_bar(K, ora, mkn, phi, slices, ta, tb):
    m, k, n = mkn
    a, b = _operands(m, k, n, phi, 11)
    av = a.t().contiguous().t() if ta else a
    bv = b.t().contiguous().t() if tb else b
    c = K.matmul(av, bv)
    assert _err(ora, c, a, b) <= BAR
    assert torch.equal(c, K.matmul(av, bv, variant=L.GEMM_DMMA)) != slices  # (the two round differently)
    out = torch.full((m, n), 3.0, dtype=torch.float64, device="cuda")
    K.matmul_to(av, bv, out)  # the product is rounded before it meets `out`
    assert torch.equal(out, c + 3.0)


def test_auto_unaligned_rows(K, ora):
    """Rows that start 8 bytes off a 16-byte boundary, and a C with a pitch."""
    a0, b0 = _operands(400, 401, 403, 0.0, 5)
    a, b = a0[:, 1:], b0[1:, 3:]
    c = torch.zeros((400, 403), dtype=torch.float64, device="cuda")[:, 1:401]
    K.matmul_to(a, b, c)
    assert _err(ora, c, a, b) <= BAR


def test_auto_leaves_operands_it_cannot_carry(K):
    """Inf / NaN, sums that overflow and spreads beyond the slice limit give
    the FP64 kernel's bits; an exact product (I * A) stays exact."""
    a, b = _operands(512, 512, 512, 0.0, 7)
    bad = a.clone()
    bad[3, 5], bad[7, 1] = float("inf"), float("nan")
    for x, y in ((bad, b), (a * 1e200, b * 1e110), (a, bad.t().contiguous())):
        c, d = K.matmul(x, y), K.matmul(x, y, variant=L.GEMM_DMMA)
        assert torch.equal(torch.nan_to_num(c, nan=7.0), torch.nan_to_num(d, nan=7.0))
        assert torch.equal(c.isnan(), d.isnan())
    wide = a.clone()
    wide[:, ::2] *= 1e-200
    mate = b.clone()
    mate[1::2] *= 1e-200
    assert torch.equal(K.matmul(wide, mate), K.matmul(wide, mate, variant=L.GEMM_DMMA))
    eye = torch.eye(512, dtype=torch.float64, device="cuda")
    assert torch.equal(K.matmul(eye, eye), eye)
    assert torch.equal(K.matmul(torch.zeros_like(a), b), torch.zeros_like(a))


def test_auto_streams_and_capture(K):
    """Calls on two streams have their own scratch; under capture the FP64
    kernel runs and replays see new inputs."""
    a, b = _operands(640, 700, 600, 0.0, 9)
    want = K.matmul(a, b)
    s = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    got = []
    for i in range(6):
        with torch.cuda.stream(s[i % 2]):
            got.append(K.matmul(a, b))
    torch.cuda.synchronize()
    assert all(torch.equal(g, want) for g in got)
    x, y = a.clone(), b.clone()
    c = torch.empty_like(want)
    K.gemm_2d(640, 700, 600, x, y, c, variant=L.GEMM_DMMA)  # (its split scratch is in place before the capture)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        K.gemm_2d(640, 700, 600, x, y, c)
    x.mul_(2.0)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(c, K.matmul(x, y, variant=L.GEMM_DMMA))


def test_auto_bits_do_not_depend_on_the_sm_budget(K):
    a, b = _operands(512, 1500, 700, 1.0, 3)
    want = K.matmul(a, b)
    for sms in (100, 37):
        with K.sm_budget(sms):
            assert torch.equal(K.matmul(a, b), want)
