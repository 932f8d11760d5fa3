"""The slice GEMM's large-problem kernel (CTA pairs on 256 x 256 tiles).

Row and column exponents depend on a whole row of A and column of B only, and
every element's total is exact before its one rounding. So a block of C is,
bit for bit, the product of its rows and columns alone, which runs on the
128 x 128 tiles. Blocks lie at the problem's corners and across the tiles'
inner edges.
"""
import pytest
import torch

from numrs_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _operand(r, c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand((r, c), dtype=torch.float64, device="cuda", generator=g) - 0.5
    return u * torch.exp(2.0 * torch.randn((r, c), dtype=torch.float64, device="cuda", generator=g))


def _blocks(extent):
    return [slice(0, 70), slice(100, 300), slice(extent - 70, extent)]


# one and several K chunks, ragged K, K below one 64-wide block; digits in one word, in two, beyond eight; the digit
# widths 8 and 7
@pytest.mark.parametrize("k,slices", [(1, 1), (63, 2), (64, 5), (200, 7), (257, 9), (1025, 7), (2049, 8), (130, 12),
                                      (1100, 15), (12300, 12), (11000, 12)])
@pytest.mark.parametrize("m,n", [(1793, 2055), (1919, 2201)])
def test_pair_blocks_have_the_small_tiles_bits(K, m, n, k, slices):
    a, b = _operand(m, k, 1), _operand(k, n, 2)
    c, info = K.gemm_ozaki(a, b, slices=slices)
    assert info["slices"] == slices
    for rows in _blocks(m):
        for cols in _blocks(n):
            small, i2 = K.gemm_ozaki(a[rows].contiguous(), b[:, cols].contiguous(), slices=slices)
            assert i2["slice_bits"] == info["slice_bits"]
            assert torch.equal(c[rows, cols], small)


def test_pair_accumulates_into_a_pitched_view(K):
    a, b = _operand(1800, 300, 3), _operand(300, 2060, 4)
    c, _ = K.gemm_ozaki(a, b, slices=7)
    out = torch.full((1800, 2101), 2.0, dtype=torch.float64, device="cuda")
    K.gemm_ozaki(a, b, slices=7, out=out[:, 1:2061], accumulate=True)
    assert torch.equal(out[:, 1:2061], 2.0 + c)
    assert bool((out[:, 0] == 2.0).all()) and bool((out[:, 2061:] == 2.0).all())


# several K ranges on pairs (the slabs are added in order): the error bar of 16 ranges
@pytest.mark.parametrize("m,k,n", [(1536, 1536, 1536), (1000, 8192, 1000), (1999, 1537, 3001)])
def test_pair_with_k_ranges(K, m, k, n):
    a, b = _operand(m, k, 5), _operand(k, n, 6)
    c = K.matmul(a, b)
    ref, _ = K.gemm_ozaki(a, b, slices=12)  # 2^-96 of the scaled operands: its own rounding of C only
    bar = 2e-15 * (a.abs() @ b.abs())
    assert bool(((c - ref).abs() <= bar).all())


def test_pair_launch_returns_at_once_for_operands_it_cannot_carry(K):
    a, b = _operand(2048, 700, 7), _operand(700, 2100, 8)
    a[5, 9], b[3, 77] = float("inf"), float("nan")
    c, d = K.matmul(a, b), K.matmul(a, b, variant=L.GEMM_DMMA)
    assert torch.equal(c.isnan(), d.isnan())
    assert torch.equal(torch.nan_to_num(c, nan=7.0), torch.nan_to_num(d, nan=7.0))
    a[5, 9], b[3, 77] = 1.0, 1.0  # and the next call on the stream is served
    assert bool(((K.matmul(a, b) - a @ b).abs() <= 1e-12 * (a.abs() @ b.abs())).all())
