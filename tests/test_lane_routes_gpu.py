"""Axis reductions of views that TMA cannot address, on both sides of the
lines between the element-copy ring and one thread per lane: the same bits as
the fold in plain numpy order, and the ring's shorter tiles (more than three
blocks per SM)."""
import numpy as np
import pytest
import torch

from tests.conftest import bits, to_np

pytestmark = pytest.mark.gpu


def _x(shape, dt, seed=3):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if dt.is_floating_point:
        return torch.randn(shape, dtype=dt, device="cuda", generator=g)
    return torch.randint(-(1 << 20), 1 << 20, shape, dtype=dt, device="cuda", generator=g)


def _folds(x):
    """Left-to-right folds along axis 1, one numpy operation per position."""
    v = np.asarray(x)
    with np.errstate(over="ignore"):
        run = np.zeros(v.shape[0], v.dtype)
        best, at = v[:, 0].copy(), np.zeros(v.shape[0], np.int64)
        prefix = np.empty_like(v)
        for j in range(v.shape[1]):
            run = run + v[:, j]
            prefix[:, j] = v[:, j] if j == 0 else prefix[:, j - 1] + v[:, j]
            at = np.where(v[:, j] > best, j, at)
            best = np.maximum(best, v[:, j])
        n = v.dtype.type(v.shape[1])
        ssd = None
        if v.dtype.kind == "f":
            mean = run / n
            ssd = np.zeros(v.shape[0], v.dtype)
            for j in range(v.shape[1]):
                d = v[:, j] - mean
                ssd = ssd + d * d
    return run, best, at, prefix, ssd


F32, F64, I64 = torch.float32, torch.float64, torch.int64


@pytest.mark.parametrize("dt,shape", [
    (F64, (14592, 257)), (F64, (14593, 257)), (F64, (15001, 65)), (F64, (19999, 289)), (F64, (20001, 257)),
    (F64, (55999, 257)), (F64, (56001, 257)), (F64, (29185, 257)), (F32, (15001, 321)), (F32, (14593, 65)),
    (F32, (56001, 287)), (F32, (56001, 289)), (I64, (15001, 257)), (I64, (56001, 287)), (I64, (56001, 289))])
@pytest.mark.parametrize("columns", [False, True])
def test_folds_of_many_lanes(K, dt, shape, columns):
    x = _x(shape, dt)
    run, best, at, prefix, ssd = _folds(to_np(x))
    if columns:
        x = x.t().contiguous()
    ax = 0 if columns else 1
    turn = (lambda p: p.T) if columns else (lambda p: p)

    def same(got, want):
        assert np.array_equal(bits(to_np(got)), bits(np.ascontiguousarray(want)))
    same(K.sum(x, ax), run)
    same(K.max(x, ax), best)
    assert np.array_equal(to_np(K.argmax(x, ax)), at)
    same(K.cumsum(x, ax), turn(prefix))
    same(K.ufunc_reduce("add", x, ax), prefix[:, -1])
    same(K.ufunc_reduce("maximum", x, ax), best)
    if ssd is not None:
        same(K.var(x, ax), ssd / ssd.dtype.type(shape[1]))


@pytest.mark.parametrize("n,k", [(16383, 300), (16385, 300), (16385, 1023), (16385, 1025)])
def test_f32_variances_of_columns(K, n, k):
    x = _x((n, k), F32)
    ssd = _folds(to_np(x))[4]
    assert np.array_equal(bits(to_np(K.var(x.t().contiguous(), 0))), bits(ssd / np.float32(k)))
