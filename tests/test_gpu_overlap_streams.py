"""Kernels that become resident under their predecessors, beside work the library
did not queue: two contexts at once, a caller's stream, and kernels of another
library between two calls of one stream.  Every result has the bits of the same
calls with a synchronisation after each."""
import ctypes as ct

import numpy as np
import pytest

import gbpoly
from gbpoly import Op, Precision

pytestmark = pytest.mark.gpu

FORMS = [Precision.FP32, Precision.BF16X3, Precision.FP16X3, Precision.FP8]


def calls(ctx, p, n, between=lambda: None):
    for prec in FORMS:
        ctx.gemm(prec, n, n, n, 0.02, p["A"], n, p["B"], n, 0.5, p["C"], n)
        between()
        ctx.syrk(prec, n, n, 0.02, p["C"], n, 0.5, p["B"], n)
        between()
        ctx.column_mean(n, n, p["B"], n, float(n), p["m"])
        between()
        ctx.column_stddev(n, n, p["B"], n, p["m"], float(n), 0.005, p["s"])
        between()
        ctx.atax(n, n, p["C"], n, p["m"], p["s"], p["v"])
        between()
        ctx.gemv_pair(n, n, p["C"], n, [(Op.T, 0.1, 0.5, p["s"], p["m"]), (Op.N, 0.1, 0.5, p["v"], p["w"])])
        between()


def inputs(n, seed):
    rng = np.random.default_rng(seed)
    d = {k: rng.standard_normal((n, n)).astype(np.float32) for k in "ABC"}
    return {**d, **{k: rng.standard_normal(n).astype(np.float32) for k in "msvw"}}


def same(got, want):
    for k in want:
        np.testing.assert_array_equal(got[k].view(np.uint32), want[k].view(np.uint32), err_msg=k)


def test_two_contexts_at_once():
    sizes = (1024, 260)
    with gbpoly.Context(0) as c0, gbpoly.Context(0) as c1:
        jobs = []
        for ctx, n in zip((c0, c1), sizes):
            init = inputs(n, n)
            jobs.append((ctx, n, init, {k: ctx.upload(v) for k, v in init.items()}))

        def run(order):
            for ctx, n, init, p in jobs:
                for k, v in init.items():
                    ctx.h2d(p[k], v)
                ctx.synchronize()
            order()
            out = []
            for ctx, n, init, p in jobs:
                ctx.synchronize()
                out.append({k: ctx.download(p[k], v.shape) for k, v in init.items()})
            return out

        def one_by_one():
            for ctx, n, _, p in jobs:
                calls(ctx, p, n, ctx.synchronize)

        def together():
            (a, na, _, pa), (b, nb, _, pb) = jobs
            a.stream_hold(200000)
            calls(a, pa, na)
            b.stream_hold(200000)
            calls(b, pb, nb)
            a.stream_release()
            b.stream_release()

        want = run(one_by_one)
        for _ in range(3):
            for g, w in zip(run(together), want):
                same(g, w)


def test_a_callers_stream_with_foreign_kernels():
    torch = pytest.importorskip("torch")
    n = 644
    init = inputs(n, 7)
    stream = torch.cuda.Stream()
    with gbpoly.Context(0) as ctx:
        assert ctx.lib.gbpoly_set_stream(ctx.handle, ct.c_void_p(stream.cuda_stream)) == 0
        t = {k: torch.empty(v.shape, device="cuda") for k, v in init.items()}

        def run(sync):
            for k, v in init.items():
                t[k].copy_(torch.from_numpy(v))
            torch.cuda.synchronize()

            def between():  # kernels of another library that read and write what the calls do
                t["B"].mul_(0.5).add_(t["C"], alpha=0.25)
                t["m"].add_(1.0)
                t["A"].copy_(t["B"])
                if sync:
                    torch.cuda.synchronize()

            with torch.cuda.stream(stream):
                calls(ctx, {k: v.data_ptr() for k, v in t.items()}, n, between)
            ctx.synchronize()
            torch.cuda.synchronize()
            return {k: v.cpu().numpy() for k, v in t.items()}

        want = run(True)
        assert all(np.isfinite(v).all() for v in want.values())
        for _ in range(3):
            same(run(False), want)
        ctx.lib.gbpoly_set_stream(ctx.handle, None)
