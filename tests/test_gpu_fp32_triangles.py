"""Plain FP32 symmetric contractions that run as two launches over the triangle.

Inputs are whole numbers in [-4, 4] and K <= 700, so every partial sum is a
whole number below 2^24 and exact in FP32 in any order: equality, not a bound.
Sizes whose triangle of 128 x 128 tiles takes two launches (91 to 253 tiles, the
line between them in the middle of a row of tiles) and, 896, one that does not;
n on and off tile edges.
"""
import numpy as np
import pytest

from gbpoly import Op, Precision

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", ["syrk", "syr2k", "xtx"])
@pytest.mark.parametrize("n,k", [(896, 100), (1537, 700), (2304, 512), (2560, 600), (2700, 330)])
def test_triangles_are_exact_on_whole_numbers(ctx, op, n, k):
    rng = np.random.default_rng(n + k)
    A = rng.integers(-4, 5, (n, k)).astype(np.float32)
    B = rng.integers(-4, 5, (n, k)).astype(np.float32)
    C = rng.integers(-4, 5, (n, n)).astype(np.float32)  # not symmetric
    X = np.ascontiguousarray(A.T)
    dA, dB, dC, dX = ctx.upload(A), ctx.upload(B), ctx.upload(C), ctx.upload(X)
    a, b = A.astype(np.float64), B.astype(np.float64)
    if op == "syrk":
        ctx.syrk(Precision.FP32, n, k, 1.0, dA, k, 1.0, dC, n)
        want = a @ a.T + C
    elif op == "syr2k":
        ctx.syr2k(Precision.FP32, n, k, 1.0, dA, k, dB, k, 1.0, dC, n)
        want = a @ b.T + b @ a.T + C
    else:
        ctx.gemm(Precision.FP32, n, n, k, 1.0, dX, n, dX, n, 1.0, dC, n, op_a=Op.T)
        want = a @ a.T + C
    ctx.synchronize()
    np.testing.assert_array_equal(ctx.download(dC, C.shape), want.astype(np.float32))
    for x in (dA, dB, dC, dX):
        ctx.free(x)
