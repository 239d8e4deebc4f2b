"""FP32 syr2k: a diagonal tile is one product plus its own transpose.

Inputs are whole numbers in [-8, 8] and K <= 1000, so every partial sum is a
whole number below 2^24 and exact in FP32 in any order: the results must be
equal, not close.  Sizes: one row, one tile and its edges, several tiles with
a ragged last one, split over two and more CTAs and not split (few k tiles).
"""
import numpy as np
import pytest

from gbpoly import Precision

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(1, 1), (5, 70), (127, 33), (128, 1000), (129, 31), (257, 512), (700, 1000),
                                 (1300, 40), (1537, 96), (2050, 32)])
@pytest.mark.parametrize("beta", [0.0, 1.0])
def test_diagonal_tiles_are_exact_on_whole_numbers(ctx, n, k, beta):
    rng = np.random.default_rng(n * 7 + k)
    A = rng.integers(-8, 9, (n, k)).astype(np.float32)
    B = rng.integers(-8, 9, (n, k)).astype(np.float32)
    C = rng.integers(-8, 9, (n, n)).astype(np.float32)  # not symmetric
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(C)
    ctx.syr2k(Precision.FP32, n, k, 1.0, dA, k, dB, k, beta, dC, n)
    ctx.synchronize()
    S = A.astype(np.float64) @ B.T.astype(np.float64)
    np.testing.assert_array_equal(ctx.download(dC, C.shape), (S + S.T + beta * C).astype(np.float32))
    for x in (dA, dB, dC):
        ctx.free(x)
