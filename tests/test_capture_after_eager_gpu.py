"""A call that has run once outside a stream capture can be captured: what it
needs of the handle's workspace, which cannot grow during a capture, is there.
Each test has a handle of its own, so that no other call has made the room.
"""
import ctypes as C

import pytest
import torch

from numrs_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.fixture
def call(K):
    lib, h = L.load(), C.c_void_p()
    L.check(lib.nrs_create(0, C.byref(h)))

    def f(name, *args):
        lib.nrs_set_stream(h, C.c_void_p(torch.cuda.current_stream().cuda_stream))
        L.check(getattr(lib, name)(h, *args), h)
    yield f
    torch.cuda.synchronize()
    lib.nrs_destroy(h)


def _p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("n", [512, 1000, 1024])
def test_f64_product(K, call, n):
    g = torch.Generator(device="cuda").manual_seed(n)
    a, b = (torch.rand((n, n), dtype=torch.float64, device="cuda", generator=g) - 0.5 for _ in range(2))
    c = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()

    def product():
        call("nrs_gemm", L.F64, n, n, n, _p(a), n, _p(b), n, _p(c), n, 0, L.GEMM_AUTO)
    product()
    torch.cuda.synchronize()
    assert not torch.equal(c, K.matmul(a, b, variant=L.GEMM_DMMA))  # (the slices ran)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        product()
    a.mul_(-3.0)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(c, K.matmul(a, b, variant=L.GEMM_DMMA))


def test_flat_reduction_after_a_short_one(K, call):
    """(300,000 elements: 37 chunk partials; 1000 run in one launch without any)"""
    x = torch.randn(300_000, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()

    def total(n):
        call("nrs_reduce", L.F64, L.SUM, 1, L.i64_array([n]), L.i64_array([1]), L.AXIS_NONE, 0, _p(x), _p(out))
    total(1000)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        total(300_000)
    x.mul_(2.0)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, K.sum(x))


def test_a_larger_call_leaves_a_captured_workspace_alone(K, call):
    """The graph's launches hold the workspace's address; the variances of
    200,000 rows need a larger one (1.6 MB of means)."""
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(300_000, dtype=torch.float64, device="cuda", generator=g)
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    rows = torch.randn((200_000, 40), dtype=torch.float64, device="cuda", generator=g)
    var = torch.zeros(200_000, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()

    def total():
        call("nrs_reduce", L.F64, L.SUM, 1, L.i64_array([300_000]), L.i64_array([1]), L.AXIS_NONE, 0, _p(x), _p(out))
    total()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        total()
    call("nrs_reduce", L.F64, L.VAR, 2, L.i64_array([200_000, 40]), L.i64_array([40, 1]), 1, 0, _p(rows), _p(var))
    others = [torch.full((1 << 18,), -1, dtype=torch.int64, device="cuda") for _ in range(8)]
    x.mul_(2.0)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, K.sum(x)) and torch.equal(var, K.var(rows, 1))
    assert all(int(t.min()) == -1 and int(t.max()) == -1 for t in others)
