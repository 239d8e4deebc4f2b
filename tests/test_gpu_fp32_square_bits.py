"""Plain FP32 X X^T and X^T X at sizes of one to several rounds of tiles: the
triangle of tiles gives, bit for bit, the full square of the same call with a
copy of the matrix as its right operand, from the device and from host buffers.
Random inputs and a C that is not symmetric."""
import numpy as np
import pytest

from gbpoly import Op, Precision

pytestmark = pytest.mark.gpu
P = Precision.FP32


@pytest.mark.parametrize("ops", [(Op.N, Op.T), (Op.T, Op.N)], ids=["xxt", "xtx"])
@pytest.mark.parametrize("n,k,pad", [(641, 700, 0), (770, 1500, 0), (900, 512, 0), (1024, 64, 0), (1100, 1001, 1),
                                     (1537, 1540, 0), (1800, 300, 0), (2304, 2304, 0), (2305, 512, 1), (2560, 130, 0),
                                     (3200, 640, 0), (900, 40, 1), (3000, 33, 1), (200, 72, 1), (650, 80, 1)])
def test_triangle_is_the_full_square(ctx, ops, n, k, pad):
    rng = np.random.default_rng(n + k)
    rows, cols = (n, k) if ops[0] == Op.N else (k, n)
    A = rng.uniform(-1, 1, (rows, cols + pad)).astype(np.float32)
    C = rng.uniform(-1, 1, (n, n)).astype(np.float32)
    dA, dA2, d1, d2 = ctx.upload(A), ctx.upload(A), ctx.upload(C), ctx.upload(C)
    ld = cols + pad
    ctx.gemm(P, n, n, k, 1.25, dA, ld, dA, ld, -0.5, d1, n, op_a=ops[0], op_b=ops[1])
    ctx.gemm(P, n, n, k, 1.25, dA, ld, dA2, ld, -0.5, d2, n, op_a=ops[0], op_b=ops[1])
    out = C.copy()
    ctx.gemm_host(P, n, n, k, 1.25, A, ld, A, ld, -0.5, out, n, op_a=ops[0], op_b=ops[1])
    ctx.synchronize()
    triangle, full = ctx.download(d1, C.shape), ctx.download(d2, C.shape)
    for b in (dA, dA2, d1, d2):
        ctx.free(b)
    np.testing.assert_array_equal(triangle.view(np.uint32), full.view(np.uint32))
    np.testing.assert_array_equal(out.view(np.uint32), full.view(np.uint32))
