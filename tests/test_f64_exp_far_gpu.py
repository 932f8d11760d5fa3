"""f64 exp where results underflow, overflow or are not numbers: the values at
both ends of every class of argument, in vectors that mix them with ordinary
ones, and no slower than the ordinary ones' worst (FP64 arithmetic)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _near(x):
    return [np.nextafter(x, -np.inf), x, np.nextafter(x, np.inf)]


EDGES = np.array(sum((_near(x) for x in (-32.0, 32.0, -708.3964185322641, -708.5, -745.1332191019411, -745.2, -746.0,
                                         709.782712893384, 709.8, 710.0, -1e300, 1e300)), [])
                 + [np.inf, -np.inf, np.nan, -np.nan, 0.0, -0.0])


@pytest.mark.parametrize("width", [1, 2, 3, 4, 7, 8, 16])
def test_every_class_in_every_place(K, width):
    r = np.random.default_rng(width)
    x = np.tile(r.normal(0, 1, width), EDGES.size)
    x[r.integers(0, width, EDGES.size) + np.arange(EDGES.size) * width] = EDGES
    with np.errstate(over="ignore", under="ignore"):
        want = np.exp(x)
    for got in (K.exp(torch.from_numpy(x).cuda()), K.exp_affine(torch.from_numpy(x).cuda(), 1.0, 0.0)):
        got = got.cpu().numpy()
        np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
        np.testing.assert_array_equal(np.isinf(got), np.isinf(want))
        np.testing.assert_array_equal((got == 0)[x <= -746], True)
        fin = np.isfinite(want)
        # 1 ulp for normal results, 2 for subnormal ones (CUDA's exp)
        ulps = np.abs(got[fin] - want[fin]) / np.spacing(np.maximum(want[fin], 5e-324))
        assert ulps.max() <= 2 and ulps[want[fin] > 1e-300].max() <= 1


@pytest.mark.parametrize("kind", ["-inf", "inf", "below", "mixed"])
def test_certain_results_are_not_slower_than_others(K, kind):
    n = 1 << 24
    g = torch.Generator(device="cuda").manual_seed(2)
    far = torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * 1400 - 700  # none certain, most beyond 32
    x = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    if kind == "below":
        x = x * 100 - 2000
    else:
        x[torch.rand(n, device="cuda", generator=g) < (0.5 if kind == "mixed" else 2)] = float(kind) if kind != "mixed" else -np.inf

    def us(v):
        best = float("inf")
        for _ in range(7):
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            s.record()
            K.exp(v)
            e.record()
            e.synchronize()
            best = min(best, s.elapsed_time(e) * 1e3)
        return best
    assert us(x) <= 1.5 * us(far)
