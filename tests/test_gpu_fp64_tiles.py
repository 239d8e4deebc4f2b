"""FP64 tiled kernel at the edges of its 16 x 16 tiles and 16-deep k steps.

Tolerance: a sum of K products, scaled, plus beta * C, in double: at most
(K + 4) 2^-53 (|alpha| |A||B| + |beta| |C|) elementwise from the exact value,
and the float64 reference as much again."""
import numpy as np
import pytest

from gbpoly import Op

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op_a", [Op.N, Op.T])
@pytest.mark.parametrize("op_b", [Op.N, Op.T])
@pytest.mark.parametrize("mnk", [(1, 17, 1), (15, 16, 17), (16, 33, 16), (49, 31, 40)])
def test_tile_edges(ctx, op_a, op_b, mnk):
    M, N, K = mnk
    rng = np.random.default_rng(M + N + K)
    A = rng.standard_normal((M, K) if op_a == Op.N else (K, M))
    B = rng.standard_normal((K, N) if op_b == Op.N else (N, K))
    C = rng.standard_normal((M, N + 2))
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(C)
    ctx.gemm_f64(M, N, K, 1.5, dA, A.shape[1], dB, B.shape[1], -0.25, dC, N + 2, op_a=op_a, op_b=op_b)
    ctx.synchronize()
    got = ctx.download(dC, C.shape, np.float64)
    a, b = (A if op_a == Op.N else A.T), (B if op_b == Op.N else B.T)
    bound = 2 * (K + 4) * 2.0 ** -53 * (1.5 * (np.abs(a) @ np.abs(b)) + 0.25 * np.abs(C[:, :N]))
    assert (np.abs(got[:, :N] - (1.5 * a @ b - 0.25 * C[:, :N])) <= bound).all()
    np.testing.assert_array_equal(got[:, N:], C[:, N:])
    for x in (dA, dB, dC):
        ctx.free(x)


@pytest.mark.parametrize("n,k", [(1, 3), (16, 16), (17, 5), (100, 33)])
def test_mirrored_tiles(ctx, n, k):
    rng = np.random.default_rng(n + k)
    A, B, C = rng.standard_normal((n, k)), rng.standard_normal((n, k)), rng.standard_normal((n, n))
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(C)
    ctx.syr2k_f64(n, k, 2.0, dA, k, dB, k, 0.5, dC, n)
    ctx.synchronize()
    bound = 2 * (2 * k + 4) * 2.0 ** -53 * (2.0 * (np.abs(A) @ np.abs(B.T) + np.abs(B) @ np.abs(A.T)) + 0.5 * np.abs(C))
    assert (np.abs(ctx.download(dC, C.shape, np.float64) - (2.0 * (A @ B.T + B @ A.T) + 0.5 * C)) <= bound).all()
    for x in (dA, dB, dC):
        ctx.free(x)
