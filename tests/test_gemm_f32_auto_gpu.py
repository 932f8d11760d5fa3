"""f32 matmul through the call's own choice of kernel: 64 x 64 tiles with K
split over a cluster, 128 x 128 tiles, or slice products on the tensor cores;
and the tiles' vector loads.

Error bars against the double-double product, max |C - C_dd| / (|A||B|)_ij:
an FMA chain over K rounds at most K times (K 2^-24, the test sizes stay below
1e-5 in practice, the library's f32 bar); slice products keep 2^-26 and round
once to f32 (2^-24), at most 2^-23 together.
"""
import numpy as np
import pytest
import torch

from numrs_gb300 import _lib as L
from tests.conftest import to_np

pytestmark = pytest.mark.gpu


def _pair(m, k, n, seed=1):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.rand((m, k), device="cuda", generator=g) * 2 - 1, torch.rand((k, n), device="cuda", generator=g) * 2 - 1)


def _err(ora, c, a, b):
    Cdd, ab = ora.gemm_dd(to_np(a.contiguous()).astype(np.float64), to_np(b.contiguous()).astype(np.float64))
    return float(np.max(np.abs(to_np(c).astype(np.float64) - Cdd) / ab))


# one CTA, every split of the cluster, ragged tile edges, short and odd K, rows shorter than a vector
@pytest.mark.parametrize("mkn", [(1, 1, 1), (3, 2, 5), (64, 64, 64), (65, 127, 63), (130, 128, 70), (200, 515, 129),
                                 (300, 1000, 257), (64, 4096, 64), (1, 3000, 1), (700, 33, 900)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_small_products(K, ora, mkn, ta, tb):
    m, k, n = mkn
    a, b = _pair(m, k, n)
    av = a.t().contiguous().t() if ta else a
    bv = b.t().contiguous().t() if tb else b
    c = K.matmul(av, bv)
    assert _err(ora, c, a, b) <= 1e-5
    out = torch.full((m, n), 2.0, device="cuda")
    K.matmul_to(av, bv, out)
    assert torch.equal(out, c + 2.0)
    # (operands one element off a 16-byte boundary: scalar loads, same bits)
    pad = torch.zeros(m * k + n * k + 2, device="cuda")
    a2 = pad[1:1 + m * k].view(k, m).t() if ta else pad[1:1 + m * k].view(m, k)
    b2 = pad[1 + m * k:1 + m * k + n * k].view(n, k).t() if tb else pad[1 + m * k:1 + m * k + n * k].view(k, n)
    a2.copy_(a)
    b2.copy_(b)
    assert torch.equal(K.matmul(a2, b2), c)
    for v in (L.GEMM_SIMT, L.GEMM_SIMT_SMALL):
        x = K.matmul(av, bv, variant=v)
        assert torch.equal(K.matmul(a2, b2, variant=v), x)
        assert _err(ora, x, a, b) <= 1e-5


@pytest.mark.parametrize("mkn", [(1537, 1999, 1801), (2048, 1024, 2100), (1200, 10500, 1100)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, True)])
def test_large_products_on_slices(K, mkn, ta, tb):
    m, k, n = mkn
    a, b = _pair(m, k, n, 3)
    av = a.t().contiguous().t() if ta else a
    bv = b.t().contiguous().t() if tb else b
    c = K.matmul(av, bv)
    # (f64 products: their own error is 2^-53 K, far below the bar)
    ref, ab = torch.matmul(a.double(), b.double()), torch.matmul(a.double().abs(), b.double().abs())
    assert float(((c.double() - ref).abs() / ab).max()) <= 2.0 ** -23
    out = torch.full((m, n), 2.0, device="cuda")
    K.matmul_to(av, bv, out)
    assert torch.equal(out, c + 2.0)
    ints = torch.randint(-8, 9, (m, k), device="cuda").float()
    mate = torch.randint(-8, 9, (k, n), device="cuda").float()
    assert torch.equal(K.matmul(ints, mate).double(), ints.double() @ mate.double())


def test_large_products_that_slices_cannot_carry(K):
    """Inf / NaN, sums that overflow f32 and operands of subnormals (which the
    spread estimate counts as zeros) give the FP32 kernel's bits."""
    a, b = _pair(2048, 2048, 2048, 5)
    bad = a.clone()
    bad[5, 7], bad[9, 1] = float("inf"), float("nan")
    for x, y in ((bad, b), (a * 1e30, b * 1e30), (a * 1e-42, b)):
        c, d = K.matmul(x, y), K.matmul(x, y, variant=L.GEMM_SIMT)
        assert torch.equal(c.isnan(), d.isnan())
        assert torch.equal(torch.nan_to_num(c, nan=7.0), torch.nan_to_num(d, nan=7.0))


def test_capture_and_sm_budget(K):
    a, b = _pair(500, 900, 300, 7)
    big = _pair(2048, 2048, 2048, 8)
    want, wide = K.matmul(a, b), K.matmul(*big)
    with K.sm_budget(37):
        assert torch.equal(K.matmul(a, b), want) and torch.equal(K.matmul(*big), wide)
    c, d = torch.empty_like(want), torch.empty_like(wide)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        K.gemm_2d(500, 900, 300, a, b, c)
        K.gemm_2d(2048, 2048, 2048, big[0], big[1], d)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(c, want)
    assert torch.equal(d, K.matmul(*big, variant=L.GEMM_SIMT))  # (captured: the FP32 kernel)
