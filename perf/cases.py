"""Measured workloads of the library, each one pass through the public entry points of gbpoly.Context.

A case is a dict of plain values: "op" names the entry point (or the chain of
entry points a benchmark program issues), the rest are its sizes, precision
form and layout.  Inputs are seeded random matrices resident on the device, as
the benchmarks' seeded initialisations (uniform[-1, 1], normal(0, 1)) make
them.  Where a call updates its output in place (beta * C + ...), beta is
0.5, the grouped workload's value, so that any number of passes stays finite.
"""
from __future__ import annotations

import math
import sys
import weakref
from pathlib import Path

import torch

sys.path.insert(0, str(Path.cwd() / "sycl-bench_gb300"))
import gbpoly  # noqa: E402
from gbpoly import Op, Precision  # noqa: E402

ALPHA, BETA = 1.5, 0.5


def listed() -> list[dict]:
    return [
        # A small ragged product: one call's latency (launches, host path).
        {"name": "gemm_small_bf16x3", "op": "gemm", "prec": "BF16X3", "M": 200, "N": 136, "K": 328, "ta": False,
         "tb": False, "pad": 0},
        # The suite's default: gemm --size=1024, plain FP32, the drop-in form.
        {"name": "gemm_fp32_1024", "op": "gemm", "prec": "FP32", "M": 1024, "N": 1024, "K": 1024, "ta": False,
         "tb": False, "pad": 0},
        # Plain FP32 at odd sizes: packed rows start off 16-byte boundaries.
        {"name": "gemm_fp32_odd", "op": "gemm", "prec": "FP32", "M": 1501, "N": 1023, "K": 2047, "ta": False,
         "tb": False, "pad": 0},
        # The largest: the headline benchmark, gemm at N = 8192 in the split-BF16 form.
        {"name": "gemm_bf16x3_8192", "op": "gemm", "prec": "BF16X3", "M": 8192, "N": 8192, "K": 8192, "ta": False,
         "tb": False, "pad": 0},
        # The matched-error form on both operands transposed as stored, rectangular, padded rows.
        {"name": "gemm_fp16x3_tt", "op": "gemm", "prec": "FP16X3", "M": 4096, "N": 3000, "K": 2560, "ta": True,
         "tb": True, "pad": 8},
        # A symmetric update at the family's size.
        {"name": "syrk_bf16x3_4096", "op": "syrk", "prec": "BF16X3", "N": 4096, "K": 4096, "pad": 0},
        # The FP32 rank-2k update (two products in one accumulator).
        {"name": "syr2k_fp32_1536", "op": "syr2k", "prec": "FP32", "N": 1536, "K": 1536, "pad": 0},
        # 3mm's three stages as one captured graph: E and F one grouped launch, then G.
        {"name": "3mm_bf16x3_2048", "op": "3mm", "prec": "BF16X3", "N": 2048},
        # Correlation of a data set: means, deviations, the contraction; rows one element wider
        # than the matrix, as the benchmark stores them.
        {"name": "correlation_fp16x3", "op": "correlation", "prec": "FP16X3", "rows": 3000, "cols": 2000},
        # atax at the suite's size, the matrix read from HBM.
        {"name": "atax_4096", "op": "atax", "rows": 4096, "cols": 4096, "pad": 0},
        # Independent products of uneven shapes in one grouped plan.
        {"name": "grouped_bf16x3_64", "op": "grouped", "prec": "BF16X3", "count": 64, "lo": 64, "hi": 2048},
        # The double variant every benchmark also runs, at the suite's size.
        {"name": "gemm_f64_1024", "op": "gemm_f64", "M": 1024, "N": 1024, "K": 1024, "ta": False, "tb": False},
    ]


# Most floating-point operations of a drawn product, per form: about the time
# of the largest listed case at the form's rate.
MOST = {"FP32": 9e10, "BF16X3": 1.0e12, "FP16X3": 0.9e12, "TF32X3": 5e11, "BF16X6": 5e11, "TF32": 8e11, "FP8": 1.0e12}


def _log_int(rng, lo: int, hi: int) -> int:
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))


def draw(rng) -> dict:
    op = rng.choice(["gemm", "gemm", "gemm", "gemm", "syrk", "syr2k", "3mm", "correlation", "atax", "bicg", "mvt",
                     "gesummv", "grouped", "gemm_f64"])
    prec = rng.choice(["FP32", "FP32", "BF16X3", "BF16X3", "FP16X3", "FP16X3", "TF32X3", "BF16X6", "TF32", "FP8"])
    pad = rng.choice([0, 0, 1, 4, 8])
    if op in ("gemm", "gemm_f64"):
        most = 2e9 if op == "gemm_f64" else MOST[prec]
        while True:
            M, N, K = (_log_int(rng, 64, 1500 if op == "gemm_f64" else 8192) for _ in range(3))
            if 2.0 * M * N * K <= most:
                break
        case = {"op": op, "M": M, "N": N, "K": K, "ta": rng.random() < 0.4, "tb": rng.random() < 0.4}
        return case if op == "gemm_f64" else {**case, "prec": prec, "pad": pad}
    if op in ("syrk", "syr2k"):
        while True:
            N, K = _log_int(rng, 64, 6144), _log_int(rng, 64, 6144)
            if (4.0 if op == "syr2k" else 2.0) * N * N * K <= MOST[prec]:
                break
        return {"op": op, "prec": prec, "N": N, "K": K, "pad": pad}
    if op == "3mm":
        return {"op": op, "prec": rng.choice(["BF16X3", "FP16X3", "TF32X3", "BF16X6"]), "N": _log_int(rng, 128, 3072)}
    if op == "correlation":
        prec = rng.choice(["FP32", "BF16X3", "FP16X3", "TF32X3"])
        hi = 2048 if prec == "FP32" else 4096
        return {"op": op, "prec": prec, "rows": _log_int(rng, 256, hi), "cols": _log_int(rng, 128, hi)}
    if op == "grouped":
        return {"op": op, "prec": rng.choice(["BF16X3", "BF16X3", "FP16X3", "BF16X6", "TF32X3"]),
                "count": rng.randint(8, 64), "lo": 64, "hi": _log_int(rng, 256, 2048)}
    # matrix-vector products: up to the suite's 16384 columns
    while True:
        rows, cols = _log_int(rng, 256, 16384), _log_int(rng, 256, 16384)
        if rows * cols <= 1.4e8:
            break
    return {"op": op, "rows": rows, "cols": cols, "pad": pad}


# ------------------------------------------------------------------- inputs
class _Gen:
    """Seeded matrices on the device."""

    def __init__(self, seed: int):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def uniform(self, rows: int, cols: int, pad: int = 0, dtype=torch.float32) -> torch.Tensor:
        """rows x cols of uniform[-1, 1], leading dimension cols + pad (the padding's values are not used)."""
        x = torch.rand((rows, cols + pad), generator=self.g, device="cuda", dtype=dtype)
        return x.mul_(2).sub_(1)

    def normal(self, rows: int, cols: int, pad: int = 0) -> torch.Tensor:
        return torch.randn((rows, cols + pad), generator=self.g, device="cuda")


def _shapes(case: dict) -> list[tuple[int, int, int]]:
    """The group's problem shapes, M, N, K log-uniform: the same for every seed (a case is one workload)."""
    g = torch.Generator()
    g.manual_seed(2024 + case["count"])
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    u = torch.rand((case["count"], 3), generator=g, dtype=torch.float64)
    return [tuple(int(math.exp(lo + (hi - lo) * float(v))) for v in row) for row in u]


def _inputs(case: dict, seed: int) -> dict:
    g, op = _Gen(seed), case["op"]
    if op in ("gemm", "gemm_f64"):
        M, N, K, pad = case["M"], case["N"], case["K"], case.get("pad", 0)
        dt = torch.float64 if op == "gemm_f64" else torch.float32
        return {"A": g.uniform(*((K, M) if case["ta"] else (M, K)), pad, dt),
                "B": g.uniform(*((N, K) if case["tb"] else (K, N)), pad, dt), "C": g.uniform(M, N, pad, dt)}
    if op in ("syrk", "syr2k"):
        N, K, pad = case["N"], case["K"], case["pad"]
        d = {"A": g.normal(N, K, pad), "C": g.normal(N, N, pad)}
        if op == "syr2k":
            d["B"] = g.normal(N, K, pad)
        return d
    if op == "3mm":
        return {k: g.normal(case["N"], case["N"]) for k in "ABCD"}
    if op == "correlation":
        # columns with means and spreads of their own; rows cols + 1 apart
        X = g.normal(case["rows"], case["cols"], 1)
        spread, mean = g.uniform(1, case["cols"] + 1).abs_().add_(0.5), g.uniform(1, case["cols"] + 1).add_(2)
        return {"X": X.mul_(spread).add_(mean)}
    if op == "grouped":
        # per-problem scales log-uniform in [1e-3, 1e3]
        out = []
        for M, N, K in _shapes(case):
            s = 10.0 ** float(torch.rand((), generator=g.g, device="cuda") * 6 - 3)
            out.append((g.uniform(M, K).mul_(s), g.uniform(K, N).mul_(s), g.uniform(M, N).mul_(s)))
        return {"problems": out}
    rows, cols, pad = case["rows"], case["cols"], case["pad"]
    d = {"A": g.uniform(rows, cols, pad)}
    if op == "gesummv":
        d["B"] = g.uniform(rows, cols, pad)
    for k, n in {"atax": (("x", cols), ("tmp", rows), ("y", cols)), "bicg": (("r", rows), ("p", cols), ("s", cols), ("q", rows)),
                 "mvt": (("y1", cols), ("y2", cols), ("x1", rows), ("x2", rows)),
                 "gesummv": (("x", cols), ("tmp", rows), ("y", rows))}[op]:
        d[k] = g.uniform(1, n).reshape(-1)
    return d


# ------------------------------------------------------------------- passes
_ctx = None


def _context() -> gbpoly.Context:
    """The process's one context, as the benchmark programs keep one queue."""
    global _ctx
    if _ctx is None:
        _ctx = gbpoly.Context(0)
    return _ctx


class State:
    """A case's buffers and what a program keeps for it (a grouped plan, a captured graph)."""

    def __init__(self, case: dict, seed: int):
        self.case, self.ctx = case, _context()
        self.prec = Precision[case["prec"]] if "prec" in case else None
        self.t = _inputs(case, seed)
        self.p = {k: v.data_ptr() for k, v in self.t.items() if isinstance(v, torch.Tensor)}
        self.ld = {k: v.stride(0) for k, v in self.t.items() if isinstance(v, torch.Tensor)}
        self.plan = self.graph = None
        if case["op"] == "correlation":
            n, ld = case["cols"], case["cols"] + 1
            self.t.update(mean=torch.empty(n, device="cuda"), sd=torch.empty(n, device="cuda"),
                          S=torch.empty((n, ld), device="cuda"))
            self.p.update({k: self.t[k].data_ptr() for k in ("mean", "sd", "S")})
            self.ld["S"] = ld
        elif case["op"] == "grouped":
            self.plan = self.ctx.grouped_plan(self.prec, self.ctx.descs([
                {"M": C.shape[0], "N": C.shape[1], "K": A.shape[1], "alpha": 1.0, "beta": BETA, "A": A.data_ptr(),
                 "lda": A.stride(0), "B": B.data_ptr(), "ldb": B.stride(0), "C": C.data_ptr(), "ldc": C.stride(0)}
                for A, B, C in self.t["problems"]]))
        elif case["op"] == "3mm":
            self._capture_3mm()
        weakref.finalize(self, _release, self.ctx, self.plan, self.graph)

    def _capture_3mm(self) -> None:
        n, ctx, t = self.case["N"], self.ctx, self.t
        t.update({k: torch.empty((n, n), device="cuda") for k in "EFG"})
        self.p.update({k: t[k].data_ptr() for k in "EFG"})
        p = self.p
        self.plan = ctx.grouped_plan(self.prec, ctx.descs([
            {"M": n, "N": n, "K": n, "alpha": 1.0, "beta": 0.0, "A": p[a], "lda": n, "B": p[b], "ldb": n, "C": p[c],
             "ldc": n} for a, b, c in ("ABE", "CDF")]))
        ctx.workspace_reserve(ctx.workspace_query(self.prec, n, n, n))

        def stages():
            ctx.grouped_run(self.plan)
            ctx.gemm(self.prec, n, n, n, 1.0, p["E"], n, p["F"], n, 0.0, p["G"], n)
        torch.cuda.synchronize()
        stages()  # once outside the capture: kernels are set up
        ctx.graph_begin()
        stages()
        self.graph = ctx.graph_end()
        ctx.synchronize()


def _release(ctx, plan, graph) -> None:
    if graph is not None:
        ctx.graph_destroy(graph)
    if plan is not None:
        ctx.grouped_destroy(plan)


def prepare(case: dict, seed: int) -> State:
    return State(case, seed)


def run(st: State):
    c, ctx, t, p, ld, op = st.case, st.ctx, st.t, st.p, st.ld, st.case["op"]
    if op == "gemm":
        ctx.gemm(st.prec, c["M"], c["N"], c["K"], ALPHA, p["A"], ld["A"], p["B"], ld["B"], BETA, p["C"], ld["C"],
                 Op.T if c["ta"] else Op.N, Op.T if c["tb"] else Op.N)
        return t["C"]
    if op == "gemm_f64":
        ctx.gemm_f64(c["M"], c["N"], c["K"], ALPHA, p["A"], ld["A"], p["B"], ld["B"], BETA, p["C"], ld["C"],
                     Op.T if c["ta"] else Op.N, Op.T if c["tb"] else Op.N)
        return t["C"]
    if op == "syrk":
        ctx.syrk(st.prec, c["N"], c["K"], ALPHA, p["A"], ld["A"], BETA, p["C"], ld["C"])
        return t["C"]
    if op == "syr2k":
        ctx.syr2k(st.prec, c["N"], c["K"], ALPHA, p["A"], ld["A"], p["B"], ld["B"], BETA, p["C"], ld["C"])
        return t["C"]
    if op == "3mm":
        ctx.graph_launch(st.graph)
        return {k: t[k] for k in "EFG"}
    if op == "correlation":
        rows, n = c["rows"], c["cols"]
        ctx.column_mean(rows, n, p["X"], ld["X"], float(rows), p["mean"])
        ctx.column_stddev(rows, n, p["X"], ld["X"], p["mean"], float(rows), 0.005, p["sd"])
        ctx.covariance(st.prec, rows, n, p["X"], ld["X"], p["mean"], p["sd"], math.sqrt(rows), p["S"], ld["S"])
        ctx.set_diagonal(n, 1.0, p["S"], ld["S"])
        return {"mean": t["mean"], "sd": t["sd"], "S": t["S"][:, :n]}
    if op == "grouped":
        ctx.grouped_run(st.plan)
        return [C for _, _, C in t["problems"]]
    rows, cols = c["rows"], c["cols"]
    if op == "atax":
        ctx.atax(rows, cols, p["A"], ld["A"], p["x"], p["tmp"], p["y"])
        return {"tmp": t["tmp"], "y": t["y"]}
    if op == "bicg":
        ctx.gemv_pair(rows, cols, p["A"], ld["A"],
                      [(Op.T, 1.0, BETA, p["r"], p["s"]), (Op.N, 1.0, BETA, p["p"], p["q"])])
        return {"s": t["s"], "q": t["q"]}
    if op == "mvt":
        ctx.gemv_pair(rows, cols, p["A"], ld["A"],
                      [(Op.N, 1.0, BETA, p["y1"], p["x1"]), (Op.N, 1.0, BETA, p["y2"], p["x2"])])
        return {"x1": t["x1"], "x2": t["x2"]}
    ctx.gesummv(rows, cols, ALPHA, p["A"], ld["A"], p["B"], ld["B"], p["x"], BETA, p["tmp"], p["y"])
    return {"tmp": t["tmp"], "y": t["y"]}


# ----------------------------------------------------------- work and values
def work(case: dict) -> dict:
    op = case["op"]
    if op in ("gemm", "gemm_f64"):
        M, N, K, e = case["M"], case["N"], case["K"], 8 if op == "gemm_f64" else 4
        return {"bytes": e * (M * K + K * N + 2 * M * N), "flops": 2 * M * N * K}
    if op in ("syrk", "syr2k"):  # a symmetric product: the unique half of its outputs
        N, K, two = case["N"], case["K"], 2 if op == "syr2k" else 1
        return {"bytes": 4 * (two * N * K + 2 * N * N), "flops": two * N * (N + 1) * K}
    if op == "3mm":
        return {"bytes": 4 * 7 * case["N"] ** 2, "flops": 6 * case["N"] ** 3}
    if op == "correlation":
        r, n = case["rows"], case["cols"]
        return {"bytes": 4 * (r * n + n * n + 2 * n), "flops": n * (n + 1) * r + 6 * r * n}
    if op == "grouped":
        s = _shapes(case)
        return {"bytes": sum(4 * (M * K + K * N + 2 * M * N) for M, N, K in s), "flops": sum(2 * M * N * K for M, N, K in s)}
    r, n = case["rows"], case["cols"]
    mats = 2 if op == "gesummv" else 1
    return {"bytes": 4 * mats * r * n + 16 * (r + n), "flops": 2 * r * n * 2}


def exact(case: dict, seed: int):
    d, op = _inputs(case, seed), case["op"]
    f = {k: v.double() for k, v in d.items() if isinstance(v, torch.Tensor)}
    if op in ("gemm", "gemm_f64"):
        M, N, K = case["M"], case["N"], case["K"]
        A = f["A"][:, :M].T if case["ta"] else f["A"][:, :K]
        B = f["B"][:, :K].T if case["tb"] else f["B"][:, :N]
        f["C"][:, :N] = ALPHA * (A @ B) + BETA * f["C"][:, :N]
        return f["C"]
    if op in ("syrk", "syr2k"):
        N, K = case["N"], case["K"]
        A = f["A"][:, :K]
        P = A @ A.T if op == "syrk" else A @ f["B"][:, :K].T
        f["C"][:, :N] = ALPHA * (P if op == "syrk" else P + P.T) + BETA * f["C"][:, :N]
        return f["C"]
    if op == "3mm":
        E, F = f["A"] @ f["B"], f["C"] @ f["D"]
        return {"E": E, "F": F, "G": E @ F}
    if op == "correlation":
        rows, n = case["rows"], case["cols"]
        X = f["X"][:, :n]
        mean = X.sum(0) / rows
        sd = ((X - mean).square().sum(0) / rows).sqrt()
        Y = (X - mean) / math.sqrt(rows) / sd
        S = Y.T @ Y
        S.fill_diagonal_(1.0)
        return {"mean": mean, "sd": sd, "S": S}
    if op == "grouped":
        return [A.double() @ B.double() + BETA * C.double() for A, B, C in d["problems"]]
    A = f["A"][:, :case["cols"]]
    if op == "atax":
        tmp = f["tmp"] + A @ f["x"]
        return {"tmp": tmp, "y": f["y"] + A.T @ tmp}
    if op == "bicg":
        return {"s": BETA * f["s"] + A.T @ f["r"], "q": BETA * f["q"] + A @ f["p"]}
    if op == "mvt":
        return {"x1": BETA * f["x1"] + A @ f["y1"], "x2": BETA * f["x2"] + A @ f["y2"]}
    tmp = f["tmp"] + A @ f["x"]
    return {"tmp": tmp, "y": ALPHA * tmp + BETA * (f["y"] + f["B"][:, :case["cols"]] @ f["x"])}
