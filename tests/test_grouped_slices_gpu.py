"""Grouped slicing (a block takes 8 rows of a problem, a warp two of them, and
finds their exponents itself) at the edges of its blocks: every product equals
the single call's bits, whose exponents come from other kernels. Rows of zeros,
of subnormals, and one element that sets a row's exponent alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])
def test_grouped_rows_and_columns_at_block_edges(K, shift):
    g = torch.Generator(device="cuda").manual_seed(4)

    def one(r, c):  # rows (columns) of different pitches; shift: 8 bytes off a 16-byte boundary
        x = torch.rand((r, c + 3), dtype=torch.float64, device="cuda", generator=g) - 0.5
        return x[:, shift:shift + c]
    problems = []
    for m, k, n in [(1, 1, 1), (4, 31, 33), (5, 33, 31), (7, 64, 40), (8, 65, 257), (9, 257, 9), (12, 300, 64), (17, 129, 130)]:
        a, b = one(m, k), one(k, n)
        a[0, k // 2] = 3e5
        a[m - 1] *= 5e-324 if m == 7 else 1.0
        a[m // 2] *= 0.0 if m == 9 else 1.0
        b[k - 1, n - 1] = -7e4
        problems.append((a, b, torch.zeros((m, n), dtype=torch.float64, device="cuda"), False))
    flags, info = K.gemm_ozaki_grouped(problems, slices=7)
    assert all(flags)
    for a, b, c, _ in problems:
        ref, i1 = K.gemm_ozaki(a, b, slices=7)
        assert i1["slice_bits"] == info["slice_bits"]
        assert torch.equal(c, ref)
