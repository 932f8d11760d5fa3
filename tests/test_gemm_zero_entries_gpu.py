"""Operands with zero rows, columns and blocks through matmul's own choice of
kernel: a sum whose every product has a zero factor is exact at any slice
count, so they run as slice products like dense ones. Nonzero entries too
small for the estimate still leave the slices.

Error bar: test_dropped_pairs.py's, 10 units of the element type and 15 more
for the sum of up to 16 K ranges.
"""
import numpy as np
import pytest
import torch

from numrs_gb300 import _lib as L
from tests.conftest import to_np

pytestmark = pytest.mark.gpu


def _sparse(kind, m, k, n, dt):
    g = torch.Generator(device="cuda").manual_seed(21)
    a, b = (torch.rand(s, dtype=dt, device="cuda", generator=g) * 2 - 1 for s in ((m, k), (k, n)))
    if kind == "row":
        a[m // 3] = 0
    elif kind == "column":
        b[:, n - 1] = 0
    elif kind == "columns":
        b[:, torch.rand(n, device="cuda", generator=g) < 0.3] = 0
    elif kind == "blocks":
        a *= torch.arange(m, device="cuda")[:, None] * 4 // m == torch.arange(k, device="cuda") * 4 // k
        b *= torch.arange(k, device="cuda")[:, None] * 4 // k == torch.arange(n, device="cuda") * 4 // n
    elif kind == "one-hot":
        a = torch.nn.functional.one_hot(torch.arange(m, device="cuda") * 7 % k, k).to(dt)
    return a, b


def _err(ora, c, a, b):
    Cdd, ab = ora.gemm_dd(to_np(a.double()), to_np(b.double()))
    d = np.abs(to_np(c).astype(np.float64) - Cdd)
    assert np.all(d[ab == 0] == 0)
    return float(np.max(d[ab > 0] / ab[ab > 0]))


@pytest.mark.parametrize("kind", ["row", "column", "columns", "blocks", "one-hot"])
@pytest.mark.parametrize("dt,mkn", [(torch.float64, (400, 390, 410)), (torch.float64, (513, 900, 385)),
                                    (torch.float32, (1500, 1400, 1700))])
def test_zero_entries_run_on_the_slices(K, ora, kind, dt, mkn):
    a, b = _sparse(kind, *mkn, dt)
    c = K.matmul(a, b)
    plain = K.matmul(a, b, variant=L.GEMM_DMMA if dt == torch.float64 else L.GEMM_SIMT)
    if kind == "one-hot":  # (one product per entry: nothing is rounded but the operand, whose bits all fit)
        assert torch.equal(c, plain)
    else:
        assert not torch.equal(c, plain)  # (the two round differently)
        u = 2.0 ** -53 if dt == torch.float64 else 2.0 ** -24
        assert _err(ora, c, a, b) <= 25 * u


@pytest.mark.parametrize("dt,small", [(torch.float64, 1e-310), (torch.float64, 1e-60), (torch.float32, 1e-40)])
def test_tiny_entries_beside_zeros_leave_the_slices(K, dt, small):
    """Row 5's products are all too small for |A'||B'|: it is no zero row."""
    m = 512 if dt == torch.float64 else 1536
    a, b = _sparse("columns", m, m, m, dt)
    a[:, ::2] = 0
    b[1::2] *= small
    a[5] = 0
    a[5, 1::2] = small
    a[5, 0] = 1
    b[0] = 0
    assert torch.equal(K.matmul(a, b), K.matmul(a, b, variant=L.GEMM_DMMA if dt == torch.float64 else L.GEMM_SIMT))
