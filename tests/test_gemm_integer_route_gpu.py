"""i64 products whose padding to tiles costs more than the tiles save run one
thread per element, with the same wrapped sums."""
import pytest
import torch

from numrs_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _us(f):
    best = float("inf")
    for _ in range(15):  # (small calls are the host's time: many of them, and the best)
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        for _ in range(25):
            f()
        e.record()
        e.synchronize()
        best = min(best, s.elapsed_time(e) * 40.0)
    return best


@pytest.mark.parametrize("m,k,n", [(1 << 20, 64, 16), (4096, 1, 4096), (512, 512, 512), (20000, 100, 100), (64, 3000, 64),
                                   (33, 33, 33)])
def test_no_slower_than_one_thread_per_element(K, m, k, n):
    g = torch.Generator(device="cuda").manual_seed(1)
    a, b = (torch.randint(-(1 << 40), 1 << 40, s, device="cuda", generator=g) for s in ((m, k), (k, n)))
    want = K.matmul(a, b, variant=L.GEMM_GENERIC)
    assert torch.equal(K.matmul(a, b), want)
    at = a.t().contiguous().t()
    assert torch.equal(K.matmul(at, b), want)
    assert _us(lambda: K.matmul(a, b)) <= 1.3 * _us(lambda: K.matmul(a, b, variant=L.GEMM_GENERIC))
