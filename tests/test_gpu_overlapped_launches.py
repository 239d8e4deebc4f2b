"""Calls queued back to back, each reading what the one before wrote, give the
bits of the same calls with a synchronisation after each: kernels become
resident under their predecessors but wait for them before any access.  The
same chain captured into a graph, too."""
import numpy as np
import pytest

import gbpoly
from gbpoly import Op, Precision

pytestmark = pytest.mark.gpu


def chain(ctx, p, n, sync):
    """Products, statistics and matrix-vector passes that reuse workspace, scratch and operands."""
    done = ctx.synchronize if sync else (lambda: None)
    for prec in (Precision.BF16X3, Precision.FP32, Precision.FP16X3, Precision.FP8, Precision.TF32X3):
        ctx.gemm(prec, n, n, n, 0.01, p["A"], n, p["B"], n, 0.5, p["C"], n)
        done()
        ctx.gemm(prec, n, n, n, 0.01, p["C"], n, p["C"], n, 0.5, p["B"], n, op_a=Op.T, op_b=Op.N)
        done()
        ctx.syr2k(prec, n, n, 0.001, p["B"], n, p["C"], n, 0.25, p["A"], n)
        done()
    ctx.column_mean(n, n, p["A"], n, float(n), p["m"])
    done()
    ctx.column_stddev(n, n, p["A"], n, p["m"], float(n), 0.005, p["s"])
    done()
    ctx.covariance(Precision.BF16X6, n, n, p["A"], n, p["m"], p["s"], 2.0, p["C"], n)
    done()
    ctx.set_diagonal(n, 1.0, p["C"], n)
    done()
    ctx.atax(n, n, p["C"], n, p["m"], p["s"], p["v"])
    done()
    ctx.gemv_pair(n, n, p["C"], n, [(Op.T, 0.1, 0.5, p["s"], p["m"]), (Op.N, 0.1, 0.5, p["v"], p["w"])])
    done()
    ctx.gesummv(n, n, 0.1, p["A"], n, p["C"], n, p["w"], 0.5, p["v"], p["s"])
    done()


@pytest.mark.parametrize("n", [132, 1024])
def test_queued_chain_is_bitwise_the_synchronised_one(n):
    rng = np.random.default_rng(n)
    init = {k: rng.standard_normal((n, n)).astype(np.float32) for k in "ABC"}
    init.update({k: rng.standard_normal(n).astype(np.float32) for k in "msvw"})
    with gbpoly.Context(0) as ctx:
        p = {k: ctx.upload(v) for k, v in init.items()}

        def run(how):
            for k, v in init.items():
                ctx.h2d(p[k], v)
            ctx.synchronize()
            how()
            ctx.synchronize()
            return {k: ctx.download(p[k], v.shape) for k, v in init.items()}

        want = run(lambda: chain(ctx, p, n, True))
        assert all(np.isfinite(v).all() for v in want.values())
        for _ in range(3):
            got = run(lambda: chain(ctx, p, n, False))
            for k in init:
                np.testing.assert_array_equal(got[k].view(np.uint32), want[k].view(np.uint32), err_msg=k)
        ctx.graph_begin()
        try:
            chain(ctx, p, n, False)
        finally:
            g = ctx.graph_end()
        got = run(lambda: ctx.graph_launch(g))
        for k in init:
            np.testing.assert_array_equal(got[k].view(np.uint32), want[k].view(np.uint32), err_msg=k)
        ctx.graph_destroy(g)
