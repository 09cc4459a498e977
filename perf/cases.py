"""The work that users of gbblas have it do, as measurable cases over its public entry points.

Sizes and distributions are those of the library's own benchmark workloads and tests: the
reference's 16 x 32 x 14 call, 256^3, the 1024..16384 sweep with its tall-skinny shape, the
8192^3 emulated-FP64 product, 4096 uneven grouped problems, small strided batches, the
4096 x 2048 x 4096 adjoint and shortest-path (semiring) products.

A case's "kind" names the entry point:
  gemm      gbblas.gemm_(C, A, B, alpha, beta, mode=...)  (mode "native" with alpha = 1 and
            beta = 0 goes through gbblas.jmul_, the same product)
  grouped   gbblas.grouped.GroupedGemm(...).run()
  batched   gbblas.gemm_strided_batched_
  autograd  gbblas.gemm_autograd, forward and backward
  semiring  gbblas.gemm_semiring_
"la", "lb", "lc" are the layouts of A, B and C: "col" (the library's own) or "row".
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jblas.jl_gb300"))
import gbblas  # noqa: E402

DTYPES = {"f64": torch.float64, "f32": torch.float32, "i32": torch.int32}


def _gemm(name, dtype, mode, m, n, k, alpha=1.0, beta=0.0, la="col", lb="col", lc="col"):
    return {"name": name, "kind": "gemm", "dtype": dtype, "mode": mode, "m": m, "n": n, "k": k, "alpha": alpha,
            "beta": beta, "la": la, "lb": lb, "lc": lc}


def listed():
    return [
        # jBLAS's own benchmark call, jmul!(D 16x14, A 16x32, X 32x14): one small static product,
        # where the call's latency is all there is.
        _gemm("jmul_f64_16x14x32", "f64", "native", 16, 14, 32),
        # The plain Float64 gemm! of ordinary matrices.
        _gemm("jmul_f64_256", "f64", "native", 256, 256, 256),
        # The Float32 gemm! sweep: a large square product with alpha and beta.
        _gemm("gemm_f32_4096", "f32", "native", 4096, 4096, 4096, 1.5, 0.5),
        # The sweep's tall-skinny shape (a large matrix times a block of vectors).
        _gemm("gemm_f32_tall", "f32", "native", 16384, 64, 16384, 1.5, 0.5),
        # The headline: FP64-accurate product on the tensor cores at the benchmark's size.
        _gemm("crt_f64_8192", "f64", "ozaki_crt", 8192, 8192, 8192),
        # The same for an ordinary, ragged problem with a transposed operand, alpha and beta.
        _gemm("crt_f64_ragged", "f64", "ozaki_crt", 1531, 1999, 1021, 1.5, 0.5, "row", "col", "col"),
        # Float32 on the tensor cores with Float32-level error, ragged, C row-major as torch has it.
        _gemm("bf16x6_f32_ragged", "f32", "bf16x6", 3001, 2503, 2047, 1.0, 0.0, "row", "row", "row"),
        # Thousands of uneven products at once, both element types.
        {"name": "grouped_f32", "kind": "grouped", "dtype": "f32", "count": 4096, "lo": 8, "hi": 512, "sizes": 7},
        {"name": "grouped_f64", "kind": "grouped", "dtype": "f64", "count": 4096, "lo": 8, "hi": 512, "sizes": 7},
        # Many small products of one shape (jBLAS's fastmul! on static matrices).
        {"name": "batched_f64", "kind": "batched", "dtype": "f64", "count": 8192, "m": 33, "n": 17, "k": 65,
         "alpha": 1.0, "beta": 0.0},
        # A training step through the differentiable product: forward, dA and dB.
        {"name": "autograd_f32", "kind": "autograd", "dtype": "f32", "m": 4096, "n": 4096, "k": 2048},
        # One squaring step of all-pairs shortest paths.
        {"name": "semiring_f32_min_plus", "kind": "semiring", "dtype": "f32", "op": "min_plus", "m": 2048, "n": 2048,
         "k": 2048, "accumulate": False, "la": "col", "lb": "col"},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _mnk(rng, lo, hi, most):
    """Three sizes in [lo, hi], log-uniform, one time in three multiples of 32, of at most `most` products."""
    while True:
        s = [_log(rng, lo, hi) for _ in range(3)]
        if rng.random() < 0.33:
            s = [max(lo, x // 32 * 32) for x in s]
        if s[0] * s[1] * s[2] <= most:
            return s


def draw(rng):
    kind = rng.choice(["f64", "f32", "f32", "tall", "crt", "crt", "tc32", "grouped", "batched", "autograd",
                       "semiring", "semiring"])
    lay = lambda: rng.choice(["col", "col", "row"])   # noqa: E731
    ab = rng.choice([(1.0, 0.0), (1.0, 0.0), (1.5, 0.5), (-1.0, 1.0)])
    case = None
    if kind == "f64":
        case = _gemm("", "f64", "native", *_mnk(rng, 8, 2048, 4 * 10 ** 9), *ab, lay(), lay(), lay())
    elif kind == "f32":
        case = _gemm("", "f32", "native", *_mnk(rng, 8, 8192, 2 * 10 ** 11), *ab, lay(), lay(), lay())
    elif kind == "tall":
        m, n, k = _log(rng, 2048, 16384), _log(rng, 8, 128), _log(rng, 2048, 16384)
        if rng.random() < 0.5:
            m, n = n, m
        case = _gemm("", "f32", "native", m, n, k, *ab, lay(), lay(), lay())
    elif kind == "crt":
        case = _gemm("", "f64", "ozaki_crt", *_mnk(rng, 384, 8192, 3 * 10 ** 11), *ab, lay(), lay(), lay())
    elif kind == "tc32":
        case = _gemm("", "f32", rng.choice(["bf16x3", "bf16x6"]), *_mnk(rng, 384, 8192, 3 * 10 ** 11), *ab, lay(),
                     lay(), lay())
    if case is not None:
        del case["name"]
        return case
    if kind == "grouped":
        return {"kind": "grouped", "dtype": rng.choice(["f32", "f64"]), "count": _log(rng, 128, 4096), "lo": 8,
                "hi": _log(rng, 48, 512), "sizes": rng.randrange(1, 1 << 20)}
    if kind == "batched":
        m, n, k = (_log(rng, 4, 96) for _ in range(3))
        return {"kind": "batched", "dtype": rng.choice(["f32", "f64"]), "count": _log(rng, 64, 16384), "m": m, "n": n,
                "k": k, "alpha": ab[0], "beta": ab[1]}
    if kind == "autograd":
        m, n, k = _mnk(rng, 256, 4096, 2 ** 35)
        return {"kind": "autograd", "dtype": "f32", "m": m, "n": n, "k": k}
    dtype = rng.choice(["f32", "f64", "i32"])
    m, n, k = _mnk(rng, 64, 4096, 2 * 10 ** 9 if dtype == "f64" else 6 * 10 ** 10)
    return {"kind": "semiring", "dtype": dtype,
            "op": rng.choice(["min_plus", "min_plus", "max_plus", "max_min", "min_max", "max_times"]), "m": m, "n": n,
            "k": k, "accumulate": rng.random() < 0.5, "la": lay(), "lb": lay()}


# ---------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _empty(r, c, dt, layout):
    """An r x c matrix of the layout."""
    return torch.empty((r, c), dtype=dt, device="cuda") if layout == "row" else \
        torch.empty((c, r), dtype=dt, device="cuda").t()


def _uniform(g, r, c, dt, layout="col"):
    X = _empty(r, c, dt, layout)
    (X if layout == "row" else X.t()).uniform_(-1.0, 1.0, generator=g)
    return X


def _ozaki(g, r, c, per, layout):
    """sign U[1, 2) 2^(e_line + e_elem): rows of A (columns of B) of widely different magnitude."""
    X = _uniform(g, r, c, torch.float64, layout)
    X.copy_(torch.where(X < 0, X - 1.0, X + 1.0))
    line = torch.randint(-30, 31, (r, 1) if per == "row" else (1, c), generator=g, device="cuda")
    elem = torch.randint(-8, 9, (r, c), generator=g, device="cuda", dtype=torch.int32)
    X.copy_(torch.ldexp(X, elem + line.to(torch.int32)))
    return X


def _weights(g, r, c, dt, op, layout):
    """Edge weights of a graph with about half of its edges missing."""
    U = torch.empty((r, c), dtype=torch.float64, device="cuda").uniform_(0.0, 1.0, generator=g)
    there = torch.rand((r, c), generator=g, device="cuda") < 0.5
    inf = float("inf")
    if dt == torch.int32:
        U = torch.floor(U * 30000.0)
        inf = float(1 << 29)
    missing = {"min_plus": inf, "max_plus": -inf, "max_min": 0.0, "min_max": inf, "max_times": 0.0}[op]
    X = _empty(r, c, dt, layout)
    X.copy_(torch.where(there, U, torch.full_like(U, missing)).to(dt))
    return X


def _sizes(case):
    g = np.random.default_rng([case["sizes"], case["count"]])
    return [tuple(int(x) for x in r) for r in
            np.rint(np.exp(g.uniform(np.log(case["lo"]), np.log(case["hi"]), size=(case["count"], 3)))).astype(np.int64)]


def _matrices(flat, shapes):
    """Column-major matrices of the shapes, one after another in `flat`."""
    out, at = [], 0
    for r, c in shapes:
        out.append(torch.as_strided(flat, (r, c), (1, r), at))
        at += r * c
    return out


def _inputs(case, seed):
    g, dt = _gen(seed), DTYPES[case["dtype"]]
    kind = case["kind"]
    if kind == "grouped":
        sizes = _sizes(case)
        flat = lambda shapes: torch.empty(sum(r * c for r, c in shapes), dtype=dt, device="cuda")   # noqa: E731
        sa, sb = [(m, k) for m, _, k in sizes], [(k, n) for _, n, k in sizes]
        fa, fb = flat(sa).uniform_(-1.0, 1.0, generator=g), flat(sb).uniform_(-1.0, 1.0, generator=g)
        return {"A": _matrices(fa, sa), "B": _matrices(fb, sb)}
    m, n, k = case["m"], case["n"], case["k"]
    if kind == "batched":
        make = lambda r, c: torch.empty((case["count"], c, r), dtype=dt, device="cuda").uniform_(   # noqa: E731
            -1.0, 1.0, generator=g).transpose(1, 2)
        return {"A": make(m, k), "B": make(k, n), "C": make(m, n)}
    if kind == "autograd":
        normal = lambda r, c: torch.randn((c, r), dtype=dt, device="cuda", generator=g).t()   # noqa: E731
        return {"A": normal(m, k), "B": normal(k, n), "W": normal(m, n)}
    if kind == "semiring":
        return {"A": _weights(g, m, k, dt, case["op"], case["la"]), "B": _weights(g, k, n, dt, case["op"], case["lb"]),
                "C": _weights(g, m, n, dt, case["op"], "col")}
    if case["mode"] == "ozaki_crt":
        A, B = _ozaki(g, m, k, "row", case["la"]), _ozaki(g, k, n, "col", case["lb"])
    else:
        A, B = _uniform(g, m, k, dt, case["la"]), _uniform(g, k, n, dt, case["lb"])
    return {"A": A, "B": B, "C": _uniform(g, m, n, dt, case["lc"])}


def prepare(case, seed):
    state = dict(case, **_inputs(case, seed))
    if case["kind"] == "grouped":
        sizes, dt = _sizes(case), DTYPES[case["dtype"]]
        flat = torch.empty(sum(m * n for m, n, _ in sizes), dtype=dt, device="cuda")
        state["C"] = flat
        state["plan"] = gbblas.grouped.GroupedGemm(state["A"], state["B"], _matrices(flat, [(m, n) for m, n, _ in sizes]))
    elif case["kind"] == "autograd":
        state["A"].requires_grad_()
        state["B"].requires_grad_()
    return state


# ---------------------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "gemm":
        if s["mode"] == "native" and s["alpha"] == 1.0 and s["beta"] == 0.0:
            return gbblas.jmul_(s["C"], s["A"], s["B"])
        return gbblas.gemm_(s["C"], s["A"], s["B"], s["alpha"], s["beta"], mode=s["mode"])
    if kind == "grouped":
        s["plan"].run()
        return s["C"]
    if kind == "batched":
        return gbblas.gemm_strided_batched_(s["C"], s["A"], s["B"], s["alpha"], s["beta"])
    if kind == "autograd":
        C = gbblas.gemm_autograd(s["A"], s["B"])
        dA, dB = torch.autograd.grad(C, (s["A"], s["B"]), s["W"])
        return {"C": C.detach(), "dA": dA, "dB": dB}
    return gbblas.gemm_semiring_(s["C"], s["A"], s["B"], s["op"], accumulate=s["accumulate"])


# ---------------------------------------------------------------------------- work and exact values
def work(case):
    size = {"f64": 8, "f32": 4, "i32": 4}[case["dtype"]]
    if case["kind"] == "grouped":
        sizes = _sizes(case)
        return {"bytes": size * sum(m * k + k * n + m * n for m, n, k in sizes),
                "flops": 2 * sum(m * n * k for m, n, k in sizes)}
    m, n, k = case["m"], case["n"], case["k"]
    if case["kind"] == "autograd":   # A, B and the incoming gradient read; C, dA and dB written
        return {"bytes": size * (2 * m * k + 2 * k * n + 2 * m * n), "flops": 6 * m * n * k}
    reads_c = case["accumulate"] if case["kind"] == "semiring" else case["beta"] != 0.0
    count = case["count"] if case["kind"] == "batched" else 1
    return {"bytes": count * size * (m * k + k * n + (2 if reads_c else 1) * m * n), "flops": count * 2 * m * n * k}


def exact(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "grouped":
        return torch.cat([(a.double() @ b.double()).t().reshape(-1) for a, b in zip(x["A"], x["B"])])
    A, B = x["A"].double(), x["B"].double()
    if kind == "autograd":
        W = x["W"].double()
        return {"C": A @ B, "dA": W @ B.t(), "dB": A.t() @ W}
    if kind in ("gemm", "batched"):
        C = A @ B
        C *= case["alpha"]
        return C if case["beta"] == 0.0 else C + case["beta"] * x["C"].double()
    op = case["op"]
    plus = torch.minimum if op in ("min_plus", "min_max") else torch.maximum
    times = {"min_plus": torch.add, "max_plus": torch.add, "max_min": torch.minimum, "min_max": torch.maximum,
             "max_times": torch.mul}[op]
    C = x["C"].double() if case["accumulate"] else None
    for k in range(A.shape[1]):
        P = times(A[:, k:k + 1], B[k:k + 1, :])
        C = P if C is None else plus(C, P)
    return C.to(torch.int32) if case["dtype"] == "i32" else C
