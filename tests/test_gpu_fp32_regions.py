"""Plain FP32 contractions that run as two launches, by rows of C.

Inputs are whole numbers in [-4, 4] with K <= 3803, so every partial sum is a
whole number below 2^24 and exact in FP32 in any order: equality, not a bound.
The sizes have 26 to 600 tiles of 128 x 128 and a last round of tiles that is
partly empty; M and N ragged, operands in both orders, rows on and off 16-byte
boundaries.  Row panels of host matrices split where the whole call does:
random inputs, the same bits.
"""
import numpy as np
import pytest

from gbpoly import Op, Precision

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ops", [(Op.N, Op.N), (Op.T, Op.N), (Op.N, Op.T), (Op.T, Op.T)])
@pytest.mark.parametrize("M,N,K,pad", [(1007, 2632, 400, 0), (1501, 1023, 2047, 1), (227, 1644, 3803, 0),
                                       (3900, 200, 256, 4)])
def test_two_regions_are_exact_on_whole_numbers(ctx, M, N, K, pad, ops):
    rng = np.random.default_rng(M + N + K)
    ints = lambda r, c: rng.integers(-4, 5, (r, c)).astype(np.float32)  # noqa: E731
    A = ints(*((K, M + pad) if ops[0] == Op.T else (M, K + pad)))
    B = ints(*((N, K + pad) if ops[1] == Op.T else (K, N + pad)))
    C = ints(M, N + pad)
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(C)
    ctx.gemm(Precision.FP32, M, N, K, 1.0, dA, A.shape[1], dB, B.shape[1], 1.0, dC, N + pad, op_a=ops[0], op_b=ops[1])
    ctx.synchronize()
    a = A[:, :M].T if ops[0] == Op.T else A[:, :K]
    b = B[:, :K].T if ops[1] == Op.T else B[:, :N]
    want = C.copy()
    want[:, :N] += (a.astype(np.float64) @ b.astype(np.float64)).astype(np.float32)
    np.testing.assert_array_equal(ctx.download(dC, C.shape), want)
    for x in (dA, dB, dC):
        ctx.free(x)


@pytest.mark.parametrize("M,N,K", [(1408, 2124, 264), (2458, 1059, 1369), (2048, 2048, 128)])
def test_row_panels_give_the_bits_of_the_whole_call(ctx, M, N, K):
    rng = np.random.default_rng(M + 3 * N)
    A = rng.uniform(-1, 1, (M, K)).astype(np.float32)
    B = rng.uniform(-1, 1, (K, N)).astype(np.float32)
    C = rng.uniform(-1, 1, (M, N)).astype(np.float32)
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(C)
    ctx.gemm(Precision.FP32, M, N, K, 1.5, dA, K, dB, N, 0.5, dC, N)
    ctx.synchronize()
    out = C.copy()
    ctx.gemm_host(Precision.FP32, M, N, K, 1.5, A, K, B, N, 0.5, out, N)
    ctx.synchronize()
    np.testing.assert_array_equal(out, ctx.download(dC, C.shape))
    for x in (dA, dB, dC):
        ctx.free(x)


def test_one_stored_matrix_on_both_sides(ctx):
    # op(A) and op(B) of one matrix, more rows than columns: neither region is a symmetric product
    K = 300
    X = np.random.default_rng(3).integers(-4, 5, (2600, K)).astype(np.float32)
    dX = ctx.upload(X)
    for M, N in ((2600, 1024), (2600, 1300), (1500, 1024)):
        dC = ctx.alloc(M * N * 4)
        ctx.gemm(Precision.FP32, M, N, K, 1.0, dX, K, dX, K, 0.0, dC, N, op_b=Op.T)
        ctx.synchronize()
        np.testing.assert_array_equal(ctx.download(dC, (M, N)), X[:M] @ X[:N].T)
        ctx.free(dC)
    ctx.free(dX)
