"""N-D matmul as one batched launch, and integer products on tiles: panels
against the oracle's Array::matmul (integers exact; f64 1e-14 and f32 1e-5 of
(|A||B|)_ij, the library's bars) at tile edges, with broadcast axes, transposed
and strided panels, more panels than a grid dimension holds, and panels large
enough for the single product's kernels."""
import numpy as np
import pytest
import torch

from numrs_gb300 import _lib as L
from tests.conftest import to_np

pytestmark = pytest.mark.gpu

DT = {"f64": torch.float64, "f32": torch.float32, "i64": torch.int64, "i32": torch.int32}


def _make(shape, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if dtype[0] == "i":
        return torch.randint(-1000, 1000, shape, dtype=DT[dtype], device="cuda", generator=g)
    return torch.rand(shape, dtype=DT[dtype], device="cuda", generator=g) * 2 - 1


def _check(c, a, b):
    """Against plain products of the panels (f64: their own rounding is within the bar)."""
    assert c.is_contiguous() and c.dtype == a.dtype
    if not c.dtype.is_floating_point:
        want = np.matmul(to_np(a).astype(np.int64), to_np(b).astype(np.int64))
        np.testing.assert_array_equal(to_np(c), want.astype(to_np(c).dtype))
        return
    ref = torch.matmul(a.double(), b.double())
    ab = torch.matmul(a.double().abs(), b.double().abs())
    assert c.shape == ref.shape
    bar = 1e-14 if c.dtype == torch.float64 else 1e-5
    assert float(((c.double() - ref).abs() - bar * ab).max()) <= 0


@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("mkn", [(1, 1, 1), (31, 33, 32), (32, 16, 33), (64, 64, 64), (65, 17, 63), (96, 80, 112),
                                 (7, 300, 5)])
@pytest.mark.parametrize("batches", [((3,), (3,)), ((2, 1), (1, 5)), ((4,), (2, 4)), ((1,), (6,)), ((), (3, 2))])
def test_panels(K, dtype, mkn, batches):
    m, k, n = mkn
    a, b = _make((*batches[0], m, k), dtype, 1), _make((*batches[1], k, n), dtype, 2)
    c = K.matmul(a, b)
    _check(c, a, b)
    at, bt = a.mT.contiguous().mT, b.mT.contiguous().mT  # column-contiguous panels
    assert torch.equal(K.matmul(at, b), c) and torch.equal(K.matmul(a, bt), c) and torch.equal(K.matmul(at, bt), c)
    wide = torch.zeros((*a.shape[:-1], 2 * k), dtype=a.dtype, device="cuda")
    wide[..., ::2] = a
    assert torch.equal(K.matmul(wide[..., ::2], b), c)  # neither contiguous: copied


def test_empty_and_degenerate(K):
    for dtype in DT:
        assert K.matmul(_make((2, 3, 0), dtype, 1), _make((2, 0, 4), dtype, 2)).eq(0).all()
        assert K.matmul(_make((0, 3, 2), dtype, 1), _make((0, 2, 4), dtype, 2)).shape == (0, 3, 4)
        assert K.matmul(_make((5, 0, 2), dtype, 1), _make((2, 4), dtype, 2)).shape == (5, 0, 4)


@pytest.mark.parametrize("dtype", ["f64", "f32", "i64"])
def test_more_panels_than_a_grid_dimension(K, dtype):
    a, b = _make((70001, 3, 2), dtype, 1), _make((2, 4), dtype, 2)
    _check(K.matmul(a, b), a, b)


@pytest.mark.parametrize("dtype,shape", [("f64", (3, 500, 450, 520)), ("f32", (2, 1700, 300, 1600)),
                                         ("i64", (2, 1700, 20, 1600))])
def test_panels_that_fill_the_gpu_are_single_products(K, dtype, shape):
    batch, m, k, n = shape
    a, b = _make((batch, m, k), dtype, 1), _make((batch, k, n), dtype, 2)
    c = K.matmul(a, b)
    _check(c, a, b)
    for i in range(batch):
        assert torch.equal(c[i], K.matmul(a[i], b[i]))


@pytest.mark.parametrize("dtype", ["i64", "i32"])
@pytest.mark.parametrize("mkn", [(31, 5, 33), (32, 32, 32), (64, 65, 63), (129, 100, 257), (300, 1000, 65)])
def test_integer_products_on_tiles(K, dtype, mkn):
    m, k, n = mkn
    a, b = _make((m, k), dtype, 3), _make((k, n), dtype, 4)
    big = 2 ** (62 if dtype == "i64" else 30)
    a[0, 0], b[0, 0] = big, big  # wraps
    want = K.matmul(a, b, variant=L.GEMM_GENERIC)
    for x in (a, a.t().contiguous().t()):
        for y in (b, b.t().contiguous().t()):
            assert torch.equal(K.matmul(x, y), want)
            out = torch.ones_like(want)
            K.matmul_to(x, y, out)
            assert torch.equal(out, want + 1)
    for v in (L.GEMM_SIMT, L.GEMM_DMMA):
        with pytest.raises(Exception):
            K.matmul(a, b, variant=v)


def test_errors(K):
    lib, h = L.load(), K.handle()
    one = L.i64_array([1])
    x = _make((4, 4), "f64", 1)
    p = x.data_ptr()
    assert lib.nrs_gemm_batched(None, L.F64, 0, None, 1, 1, 1, p, None, 1, p, None, 1, p, 0) == L.ERR_INVALID
    assert lib.nrs_gemm_batched(h, L.F64, 9, one, 1, 1, 1, p, one, 1, p, one, 1, p, 0) == L.ERR_INVALID
    assert lib.nrs_gemm_batched(h, L.F64, 1, one, 2, 2, 2, p, one, 1, p, one, 2, p, 0) == L.ERR_SHAPE
    assert lib.nrs_gemm_batched(h, L.F64, 1, one, 2, 2, 2, p, L.i64_array([-1]), 2, p, one, 2, p, 0) == L.ERR_STRIDE
    assert lib.nrs_gemm_batched(h, L.F64, 1, one, 2, 2, 2, None, one, 2, p, one, 2, p, 0) == L.ERR_INVALID
    assert lib.nrs_gemm_batched(h, 77, 1, one, 2, 2, 2, p, one, 2, p, one, 2, p, 0) == L.ERR_DTYPE
