"""Plain FP32 products of 2^31 - 1 rows or columns, the largest of the 128 x 128
kernel's coordinates, on operands on 16-byte boundaries (8.6 GB each for the long
operand and C; whole numbers, exact)."""
import numpy as np
import pytest

from gbpoly import Op, Precision

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", ["rows", "columns"])
def test_largest_dimension(ctx, side):
    n = 2 ** 31 - 1
    one = np.full(4, 3.0, np.float32)
    dLong, dC, dOne = ctx.alloc((n + 1) * 4), ctx.alloc(n * 4), ctx.upload(one)
    ctx.memset(dLong, 0, (n + 1) * 4)
    ctx.memset(dC, 0, n * 4)
    at = [0, 1, 127, 128, 2 ** 30 + 77, n - 129, n - 128, n - 127, n - 2, n - 1]
    for i, p in enumerate(at):
        ctx.h2d(dLong.ptr + 4 * p, np.full(1, i + 1, np.float32))
    ctx.synchronize()
    if side == "rows":  # C (n x 1) = A^T (n x 1) B (1 x 1), A stored 1 x n
        ctx.gemm(Precision.FP32, n, 1, 1, 2.0, dLong, n + 1, dOne, 4, 0.0, dC, 1, op_a=Op.T)
    else:               # C (1 x n) = A (1 x 1) B (1 x n)
        ctx.gemm(Precision.FP32, 1, n, 1, 2.0, dOne, 4, dLong, n + 1, 0.0, dC, n)
    ctx.synchronize()
    for i, p in enumerate(at):
        assert ctx.download(dC.ptr + 4 * p, (1,))[0] == 6.0 * (i + 1), p
    assert ctx.download(dC.ptr + 4 * 1000, (1,))[0] == 0.0
    for x in (dLong, dC, dOne):
        ctx.free(x)
