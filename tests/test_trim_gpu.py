"""The scratch that large products leave with a handle can be given back."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_trim_returns_the_scratch(K):
    g = torch.Generator(device="cuda").manual_seed(1)
    a, b = (torch.rand((3000, 3000), dtype=torch.float64, device="cuda", generator=g) - 0.5 for _ in range(2))
    want = K.matmul(a, b)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    K.trim()
    # 12 planes of two bytes per element of either operand, at the least
    assert torch.cuda.mem_get_info()[0] - before >= 12 * 2 * 2 * 9_000_000
    assert torch.equal(K.matmul(a, b), want)
    K.trim()
    K.trim()


def test_f32_scratch_holds_eight_planes(K):
    g = torch.Generator(device="cuda").manual_seed(2)
    a, b = (torch.rand((4096, 4096), device="cuda", generator=g) - 0.5 for _ in range(2))
    K.trim()
    K.matmul(a, b)  # (its result and torch's own cache are in place before the measurement)
    K.trim()
    before = torch.cuda.mem_get_info()[0]
    K.matmul(a, b)
    torch.cuda.synchronize()
    held = before - torch.cuda.mem_get_info()[0]
    planes = 2 * 2 * 4096 * 4096
    # 8 planes; digit slots (80 MB) and the pool's granularity beside them
    assert 8 * planes <= held <= 8 * planes + 150_000_000
