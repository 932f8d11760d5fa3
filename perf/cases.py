"""The performance cases of this framework.

Each case is one call (or one short chain of calls) of numrs_gb300.kernels on
device arrays, as a numrs2 user's program makes it: matrix products, grouped
GEMMs, reductions, elementwise expressions and running folds, from a thousand
elements to 2 GiB arrays. Sizes and value distributions are those of this
repository's benchmark configurations and tests (16384 x 16384 f32 N(0,1) and
i64 in [-2^20, 2^20); 512^3 and 8192^3 f64 products; a group of 4096 uneven
GEMMs; U(-1,1) and U(-0.5,0.5) * exp(phi * N(0,1)) matrix entries) and ragged
sizes between them. Every case is a plain dict; "kind" says which family it
belongs to.
"""
import numpy as np
import torch

from numrs_gb300 import _lib as L
from numrs_gb300 import kernels as K

DTYPES = {"f32": torch.float32, "f64": torch.float64, "i32": torch.int32, "i64": torch.int64}
SIZEOF = {"f32": 4, "f64": 8, "i32": 4, "i64": 8}


def listed():
    return [
        # The smallest call: the sum of a short vector, all host work and launch latency.
        {"name": "sum_f64_1000", "kind": "reduce", "op": "sum", "dtype": "f64", "rows": 1, "cols": 1000, "axis": -9,
         "view": "row"},
        # The benchmark's plain f64 product (the reference's own published size).
        {"name": "matmul_f64_512", "kind": "matmul", "dtype": "f64", "m": 512, "k": 512, "n": 512, "ta": False,
         "tb": False, "phi": 0.0},
        # A least-squares / covariance product A^T B at sizes no tile divides.
        {"name": "matmul_f64_tn_ragged", "kind": "matmul", "dtype": "f64", "m": 1999, "k": 3001, "n": 1537, "ta": True,
         "tb": False, "phi": 1.0},
        # A large single-precision product.
        {"name": "matmul_f32_4096", "kind": "matmul", "dtype": "f32", "m": 4096, "k": 4096, "n": 4096, "ta": False,
         "tb": False, "phi": 0.0},
        # An ordinary small f32 product at odd sizes, the second operand a transposed view.
        {"name": "matmul_f32_nt_small", "kind": "matmul", "dtype": "f32", "m": 300, "k": 1000, "n": 257, "ta": False,
         "tb": True, "phi": 0.0},
        # N-D Array::matmul: a stack of small f64 panels.
        {"name": "matmul_f64_batched", "kind": "batched", "dtype": "f64", "batch": 32, "m": 96, "k": 80, "n": 112,
         "shared_b": False},
        # The largest product: the split-precision f64 GEMM, slice count from the operands' spread.
        {"name": "gemm_ozaki_8192", "kind": "ozaki", "m": 8192, "k": 8192, "n": 8192, "phi": 1.0},
        # The benchmark's grouped batch, replayed from its plan's graph: 4096 uneven GEMMs (half f32, half f64, the
        # f64 half on the tensor cores) and 4096 row reductions.
        {"name": "group_4096", "kind": "group", "count": 4096, "shape_seed": 7, "f64_tc": True, "f32_tc": False},
        # The benchmark's axis reductions: column means of a 1 GiB f32 array.
        {"name": "mean_axis0_f32_16384", "kind": "reduce", "op": "mean", "dtype": "f32", "rows": 16384, "cols": 16384,
         "axis": 0, "view": "row"},
        # Row standard deviations of an f64 table at odd sizes (two passes over the lanes).
        {"name": "std_axis1_f64_ragged", "kind": "reduce", "op": "std", "dtype": "f64", "rows": 9973, "cols": 12001,
         "axis": 1, "view": "row"},
        # A fused f64 expression, exp((x - mu)^2 * -s) with a broadcast row of means.
        {"name": "gauss_f64_8192", "kind": "ufunc", "expr": "gauss", "dtype": "f64", "rows": 8192, "cols": 8192},
        # The flattened running sum of a 1 GiB f32 array.
        {"name": "cumsum_flat_f32_16384", "kind": "scan", "op": "add", "dtype": "f32", "rows": 16384, "cols": 16384,
         "axis": -9},
    ]


def _log_int(rng, lo, hi):
    v = int(round(2.0 ** rng.uniform(np.log2(lo), np.log2(hi))))
    return min(hi, max(lo, v))


def _capped(rng, ranges, cap):
    """Sizes log-uniform in their ranges whose product is at most `cap`."""
    while True:
        v = [_log_int(rng, lo, hi) for lo, hi in ranges]
        if float(np.prod([float(x) for x in v])) <= cap:
            return v


def draw(rng):
    kind = rng.choice(["matmul", "matmul", "matmul", "batched", "ozaki", "group", "reduce", "reduce", "reduce",
                       "ufunc", "ufunc", "scan", "scan"])
    if kind == "matmul":
        dtype = rng.choice(["f64", "f64", "f64", "f32", "f32", "i64"])
        cap = {"f64": 1.2e10, "f32": 7e10, "i64": 1e9}[dtype]
        top = {"f64": 4096, "f32": 8192, "i64": 2048}[dtype]
        m, k, n = _capped(rng, [(16, top), (16, top), (1, top)], cap)
        return {"kind": kind, "dtype": dtype, "m": m, "k": k, "n": n, "ta": rng.random() < 0.3,
                "tb": rng.random() < 0.3, "phi": 0.0 if dtype == "i64" else rng.choice([0.0, 0.0, 1.0])}
    if kind == "batched":
        b, m, k, n = _capped(rng, [(2, 128), (4, 256), (4, 256), (4, 256)], 3e8)
        return {"kind": kind, "dtype": rng.choice(["f64", "f32"]), "batch": b, "m": m, "k": k, "n": n,
                "shared_b": rng.random() < 0.3}
    if kind == "ozaki":
        m, k, n = _capped(rng, [(256, 8192), (256, 8192), (256, 8192)], 2.5e11)
        return {"kind": kind, "m": m, "k": k, "n": n, "phi": rng.choice([0.0, 1.0, 4.0])}
    if kind == "group":
        return {"kind": kind, "count": _log_int(rng, 64, 4096), "shape_seed": rng.randrange(1 << 20),
                "f64_tc": rng.random() < 0.8, "f32_tc": rng.random() < 0.4}
    dtype = rng.choice(["f32", "f64", "i64"])
    rows, cols = _capped(rng, [(1, 20000), (32, 20000)], 2 ** 28 * 4 / SIZEOF[dtype])
    if kind == "reduce":
        ops = ["sum", "mean", "max", "min", "argmax"] + ([] if dtype == "i64" else ["std", "var", "prod"])
        return {"kind": kind, "op": rng.choice(ops), "dtype": dtype, "rows": rows, "cols": cols,
                "axis": rng.choice([-9, 0, 1]), "view": rng.choice(["row", "row", "transposed"])}
    if kind == "ufunc":
        dtype = rng.choice(["f32", "f64"])
        rows, cols = _capped(rng, [(1, 16384), (32, 16384)], 2 ** 26 if dtype == "f64" else 2 ** 28)
        return {"kind": kind, "expr": rng.choice(["gauss", "exp_affine", "axpy", "ratio"]), "dtype": dtype,
                "rows": rows, "cols": cols}
    return {"kind": kind, "op": rng.choice(["add", "add", "maximum"]), "dtype": dtype, "rows": rows, "cols": cols,
            "axis": rng.choice([-9, 0, 1])}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _entries(g, shape, dtype, phi):
    """Matrix entries: U(-1, 1), or U(-0.5, 0.5) * exp(phi * N(0, 1)), or integers in [-1000, 1000)."""
    dt = DTYPES[dtype]
    if dtype in ("i32", "i64"):
        return torch.randint(-1000, 1000, shape, dtype=dt, device="cuda", generator=g)
    if phi == 0.0:
        return torch.rand(shape, dtype=dt, device="cuda", generator=g) * 2 - 1
    u = torch.rand(shape, dtype=dt, device="cuda", generator=g) - 0.5
    return u * torch.exp(phi * torch.randn(shape, dtype=dt, device="cuda", generator=g))


def _table(g, rows, cols, dtype):
    """Data tables: N(0, 1), or integers uniform in [-2^20, 2^20)."""
    if dtype in ("i32", "i64"):
        return torch.randint(-(1 << 20), 1 << 20, (rows, cols), dtype=DTYPES[dtype], device="cuda", generator=g)
    return torch.randn((rows, cols), dtype=DTYPES[dtype], device="cuda", generator=g)


def _group_shapes(case):
    r = np.random.default_rng(case["shape_seed"])

    def lu(lo, hi):
        return np.exp(r.uniform(np.log(lo), np.log(hi), case["count"])).astype(np.int64)
    return lu(16, 512), lu(16, 512), lu(16, 512), lu(64, 65536)


def _packed(sizes):
    """Start of each array in one buffer (256-byte multiples for every element size), and the buffer's length."""
    starts = np.concatenate([[0], np.cumsum((np.asarray(sizes, dtype=np.int64) + 63) // 64 * 64)])
    return starts[:-1], int(starts[-1])


def _group_inputs(case, seed):
    """Per element type: (A, B, C buffer, C views); and the rows to reduce."""
    g = _gen(seed)
    M, N, Kd, lens = _group_shapes(case)
    parts = {}
    for dtype, first in (("f32", 0), ("f64", 1)):
        idx = range(first, case["count"], 2)
        sa, na = _packed([M[i] * Kd[i] for i in idx])
        sb, nb = _packed([Kd[i] * N[i] for i in idx])
        sc, nc = _packed([M[i] * N[i] for i in idx])
        a, b = _entries(g, (na,), dtype, 0.0), _entries(g, (nb,), dtype, 0.0)
        c = torch.zeros(nc, dtype=DTYPES[dtype], device="cuda")

        def views(buf, starts, R, C):
            return [buf[s:s + R[i] * C[i]].view(int(R[i]), int(C[i])) for s, i in zip(starts.tolist(), idx)]
        parts[dtype] = (views(a, sa, M, Kd), views(b, sb, Kd, N), c, views(c, sc, M, N))
    sx, nx = _packed(lens)
    x = torch.randn(nx, dtype=torch.float32, device="cuda", generator=g)
    return parts, [x[s:s + int(n)] for s, n in zip(sx.tolist(), lens)]


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind in ("matmul", "ozaki"):
        m, k, n, dtype = case["m"], case["k"], case["n"], case.get("dtype", "f64")
        a = _entries(g, (k, m) if case.get("ta") else (m, k), dtype, case["phi"])
        b = _entries(g, (n, k) if case.get("tb") else (k, n), dtype, case["phi"])
        return {"case": case, "a": a.t() if case.get("ta") else a, "b": b.t() if case.get("tb") else b}
    if kind == "batched":
        a = _entries(g, (case["batch"], case["m"], case["k"]), case["dtype"], 0.0)
        b = _entries(g, (case["k"], case["n"]) if case["shared_b"] else (case["batch"], case["k"], case["n"]),
                     case["dtype"], 0.0)
        return {"case": case, "a": a, "b": b}
    if kind == "group":
        parts, rows = _group_inputs(case, seed)
        gemms = []
        for a32, a64 in zip(zip(*[parts["f32"][i] for i in (0, 1, 3)]), zip(*[parts["f64"][i] for i in (0, 1, 3)])):
            gemms += [(*a32, False), (*a64, False)]
        sums = torch.zeros(len(rows), dtype=torch.float32, device="cuda")
        reds = [(x, L.SUM, sums[i:i + 1]) for i, x in enumerate(rows)]
        plan = K.Plan(gemms, reds, f64_mode=L.PLAN_F64_OZAKI if case["f64_tc"] else L.PLAN_F64_DMMA,
                      f32_mode=L.PLAN_F32_OZAKI if case["f32_tc"] else L.PLAN_F32_FMA)
        return {"case": case, "plan": plan, "c32": parts["f32"][2], "c64": parts["f64"][2], "sums": sums}
    x = _table(g, case["rows"], case["cols"], case["dtype"])
    state = {"case": case, "x": x}
    if kind == "reduce":
        if case["axis"] == -9 and case["rows"] == 1:
            state["x"] = x.view(-1)
        elif case["view"] == "transposed":
            state["x"] = x.t()
        if case["op"] == "prod":  # values whose products stay finite
            x.mul_(1e-4).add_(1.0)
    elif kind == "ufunc":
        if case["expr"] == "gauss":
            state["mu"] = torch.randn(case["cols"], dtype=x.dtype, device="cuda", generator=g)
        elif case["expr"] in ("axpy", "ratio"):
            state["y"] = _table(g, case["rows"], case["cols"], case["dtype"])
            if case["expr"] == "ratio":
                state["y"].abs_().add_(0.5)
            else:
                state["z"] = _table(g, case["rows"], case["cols"], case["dtype"])
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("matmul", "batched"):
        return K.matmul(state["a"], state["b"])
    if kind == "ozaki":
        return K.gemm_ozaki(state["a"], state["b"])[0]
    if kind == "group":
        state["plan"].run()
        return [state["c32"], state["c64"], state["sums"]]
    x, axis = state["x"], None if case.get("axis", -9) == -9 else case["axis"]
    if kind == "reduce":
        return getattr(K, case["op"])(x, axis)
    if kind == "scan":
        return K.ufunc_accumulate(case["op"], x, axis)
    leaf = K.Expr.leaf
    if case["expr"] == "gauss":
        d = leaf(x) - leaf(state["mu"])
        return (d * d * -0.5).exp().eval()
    if case["expr"] == "exp_affine":
        return K.exp_affine(x, 0.5, -0.25)
    if case["expr"] == "axpy":
        return (leaf(x) * leaf(state["y"]) + leaf(state["z"])).eval()
    return K.divide(x, state["y"])


def work(case):
    kind = case["kind"]
    if kind in ("matmul", "ozaki", "batched"):
        m, k, n, b, s = case["m"], case["k"], case["n"], case.get("batch", 1), SIZEOF[case.get("dtype", "f64")]
        kn = k * n * (1 if case.get("shared_b") else b)
        return {"bytes": s * (b * m * k + kn + b * m * n), "flops": 2 * b * m * k * n}
    if kind == "group":
        M, N, Kd, lens = (v.astype(np.float64) for v in _group_shapes(case))
        elems = M * Kd + Kd * N + M * N
        return {"bytes": float(4 * elems[0::2].sum() + 8 * elems[1::2].sum() + 4 * lens.sum() + 4 * case["count"]),
                "flops": float((2 * M * N * Kd).sum() + lens.sum())}
    s, n = SIZEOF[case["dtype"]], case["rows"] * case["cols"]
    if kind == "reduce":
        passes = 2 if case["op"] in ("std", "var") else 1
        axis = case["axis"] if case["view"] == "row" or case["axis"] < 0 else 1 - case["axis"]
        out = 1 if axis < 0 else case["cols"] if axis == 0 else case["rows"]
        out_size = 8 if case["op"] == "argmax" or (case["op"] == "mean" and case["dtype"] == "i64") else s
        return {"bytes": s * n + out_size * out, "flops": n * (3 if passes == 2 else 1)}
    if kind == "scan":
        return {"bytes": 2 * s * n, "flops": n}
    inputs = {"gauss": 1, "exp_affine": 1, "axpy": 3, "ratio": 2}[case["expr"]]
    ops = {"gauss": 4, "exp_affine": 3, "axpy": 2, "ratio": 1}[case["expr"]]
    return {"bytes": s * (n * (inputs + 1) + (case["cols"] if case["expr"] == "gauss" else 0)), "flops": ops * n}


# ---------------------------------------------------------------------------
# The same results in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "group":
        parts, rows = _group_inputs(case, seed)
        outs = []
        for dtype in ("f32", "f64"):
            a, b, c, views = parts[dtype]
            wide = torch.zeros(c.numel(), dtype=torch.float64, device="cuda")
            for x, y, v in zip(a, b, views):
                at = v.storage_offset()
                wide[at:at + v.numel()] = (x.double() @ y.double()).reshape(-1)
            outs.append(wide)
        return outs + [torch.stack([x.double().sum() for x in rows])]
    if case.get("dtype") == "i64":
        return None
    if kind in ("matmul", "ozaki", "batched"):
        s = _plain(case, seed)
        return torch.matmul(s["a"].double(), s["b"].double())
    s = _plain(case, seed)
    x, axis = s["x"].double(), None if case.get("axis", -9) == -9 else case["axis"]
    if kind == "reduce":
        if case["op"] == "argmax":
            return None
        if axis is None:
            x, axis = x.reshape(-1), 0
        if case["op"] in ("max", "min"):
            r = getattr(torch, "a" + case["op"])(x, axis)
        elif case["op"] in ("std", "var"):
            r = getattr(torch, case["op"])(x, axis, correction=0)
        else:
            r = getattr(torch, case["op"])(x, axis)
        return r.reshape(1) if r.dim() == 0 else r
    if kind == "scan":
        if axis is None:
            x, axis = x.reshape(-1), 0
        return torch.cumsum(x, axis) if case["op"] == "add" else torch.cummax(x, axis).values
    if case["expr"] == "gauss":
        return torch.exp((x - s["mu"].double()) ** 2 * -0.5)
    if case["expr"] == "exp_affine":
        return torch.exp(0.5 * x - 0.25)
    if case["expr"] == "axpy":
        return x * s["y"].double() + s["z"].double()
    return x / s["y"].double()


def _plain(case, seed):
    """The arrays that prepare() makes (it calls nothing of the framework for these kinds)."""
    return prepare(case, seed)
