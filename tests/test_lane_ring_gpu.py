"""Lane folds of views that TMA cannot address (odd pitches, odd bases,
strided lanes and axes, few lanes): the element-copy ring against the CPU
oracle, bit for bit, at the edges of its tiles (64 / 128 positions of 8- / 4-
byte types, 32 lanes, blocks of 16) and against the TMA pipelines on the same
values."""
import numpy as np
import pytest
import torch

from numrs_gb300 import _lib as L
from oracle import oracle as O
from tests.conftest import bits, to_np

pytestmark = pytest.mark.gpu

OPS = {"sum": O.SUM, "mean": O.MEAN, "max": O.MAX, "min": O.MIN, "prod": O.PROD}
UOPS = {"add": L.OP_ADD, "subtract": L.OP_SUB, "multiply": L.OP_MUL, "maximum": L.OP_MAX, "minimum": L.OP_MIN}
# (rows, cols): axis 1 runs along contiguous lanes, axis 0 across them
SHAPES = [(1, 64), (1, 1001), (31, 65), (32, 127), (33, 129), (70, 255), (64, 257), (95, 513), (257, 33), (1025, 31),
          (300, 1), (513, 67)]


def _values(dtype, shape, seed, special):
    r = np.random.default_rng(seed)
    if dtype in (np.int32, np.int64):
        return r.integers(-1000, 1000, shape).astype(dtype)
    x = (r.standard_normal(shape) * 0.3 + 1.0).astype(dtype)
    if special:
        x[r.random(shape) < 0.02] = 0.0
        x[r.random(shape) < 0.02] = -0.0
        x[r.random(shape) < 0.003] = np.nan
        x[r.random(shape) < 0.003] = -np.inf
    return x


def _same(got, want):
    got, want = np.ascontiguousarray(got).ravel(), np.ascontiguousarray(want).ravel()
    assert got.shape == want.shape and got.dtype == want.dtype
    if want.dtype.kind == "f":  # (NaN payloads are free)
        nan = np.isnan(want)
        np.testing.assert_array_equal(np.isnan(got), nan)
        got, want = bits(got)[~nan], bits(want)[~nan]
    np.testing.assert_array_equal(got, want)


def _views(x):
    """The array as given, transposed, one element off its base and with every other column."""
    d = torch.from_numpy(x).cuda()
    yield x, d
    yield x.T, d.t()
    pad = torch.zeros(x.size + 1, dtype=d.dtype, device="cuda")[1:].view(x.shape)
    pad.copy_(d)
    yield x, pad
    wide = torch.zeros((x.shape[0], 2 * x.shape[1]), dtype=d.dtype, device="cuda")[:, ::2]
    wide.copy_(d)
    yield x, wide


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int64, np.int32])
@pytest.mark.parametrize("shape", SHAPES)
def test_folds_and_args(K, ora, dtype, shape):
    for special in (False, True):
        x = _values(dtype, shape, 3, special)
        for xv, d in _views(x):
            # (the oracle has no i32: the low 32 bits of its i64 results)
            ov = xv.astype(np.int64) if dtype == np.int32 else xv
            for axis in (0, 1):
                for op, code in OPS.items():
                    if dtype == np.int32 and op == "mean":
                        continue
                    want = ora.axis(code, ov, axis)
                    _same(to_np(getattr(K, op)(d, axis=axis)), want.astype(np.int32) if dtype == np.int32 else want)
                for want_max, fn in ((True, K.argmax), (False, K.argmin)):
                    np.testing.assert_array_equal(to_np(fn(d, axis=axis)).ravel(),
                                                  np.asarray(ora.axis_arg(ov, axis, want_max)).ravel())
                if np.dtype(dtype).kind == "f" and xv.shape[axis] > 1 and not special:
                    _same(to_np(K.var(d, axis=axis, ddof=1)), ora.axis_var(xv, axis, ddof=1))
                    _same(to_np(K.std(d, axis=axis)), ora.axis_var(xv, axis, std=True))


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int64])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("op", list(UOPS))
def test_running_and_seeded_folds(K, ora, dtype, shape, op):
    x = _values(dtype, shape, 5, op in ("maximum", "minimum"))
    for xv, d in _views(x):
        for axis in (0, 1):
            _same(to_np(K.ufunc_accumulate(op, d, axis)), ora.accumulate(UOPS[op], xv, axis))
            _same(to_np(K.ufunc_reduce(op, d, axis)), ora.ufunc_reduce(UOPS[op], xv, axis))
            init = 3 if np.dtype(dtype).kind == "i" else 0.75
            _same(to_np(K.ufunc_reduce(op, d, axis, initial=init)), ora.ufunc_reduce(UOPS[op], xv, axis, init))


def test_three_dimensional_views(K, ora):
    x = _values(np.float64, (5, 67, 129), 7, False)
    d = torch.from_numpy(x).cuda()
    for perm in ((0, 1, 2), (2, 0, 1), (1, 2, 0)):
        xv, dv = x.transpose(perm), d.permute(perm)
        for axis in range(3):
            _same(to_np(K.sum(dv, axis=axis)), ora.axis(O.SUM, xv, axis))
            _same(to_np(K.cumsum(dv, axis)), ora.accumulate(L.OP_ADD, xv, axis))
            _same(to_np(K.std(dv, axis=axis)), ora.axis_var(xv, axis, std=True))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_large_unaligned_equals_aligned(K, dtype):
    """The same values with an odd pitch (ring) and a padded one (TMA)."""
    g = torch.Generator(device="cuda").manual_seed(9)
    rows, cols = 1203, 4099
    wide = torch.randn((rows, cols + 5), dtype=dtype, device="cuda", generator=g)
    tight = wide[:, :cols].contiguous()  # pitch of 4099 elements
    for axis in (0, 1):
        for fn in (K.sum, K.max, K.std, K.argmax, K.cumsum):
            a, b = fn(tight, axis), fn(wide[:, :cols], axis)
            assert torch.equal(a, b), (fn.__name__, axis)
