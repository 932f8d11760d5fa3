"""Batches of few panels with long sums: K in ranges over clusters of CTAs."""
import pytest
import torch

from tests.test_gemm_batched_gpu import DT, _check, _make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("batch,m,k,n", [(2, 64, 4096, 64), (1, 5, 200, 7), (3, 33, 130, 65), (2, 64, 127, 64),
                                         (2, 130, 1000, 40), (18, 32, 1025, 31), (19, 32, 1025, 31), (75, 32, 160, 32),
                                         (76, 32, 160, 32), (2, 1, 5000, 1)])
def test_few_panels_with_long_sums(K, dtype, batch, m, k, n):
    """K in ranges over clusters: every number of ranges, ragged last ranges and
    tiles, and the batches on both sides of a full GPU."""
    a, b = _make((batch, m, k), dtype, 5), _make((batch, k, n), dtype, 6)
    c = K.matmul(a, b)
    _check(c, a, b)
    assert torch.equal(K.matmul(a.mT.contiguous().mT, b.mT.contiguous().mT), c)


def _us(f, reps=7):
    best = float("inf")
    for _ in range(reps + 2):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        for _ in range(5):
            f()
        e.record()
        e.synchronize()
        best = min(best, s.elapsed_time(e) * 200.0)
    return best


@pytest.mark.parametrize("dtype", ["f64", "f32", "i64"])
def test_two_panels_take_about_two_products(K, dtype):
    a, b = _make((2, 64, 4096), dtype, 5), _make((2, 4096, 64), dtype, 6)
    both = _us(lambda: K.matmul(a, b))
    assert both <= 2.0 * _us(lambda: (K.matmul(a[0], b[0]), K.matmul(a[1], b[1])))
