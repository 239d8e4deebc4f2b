"""A C of one row may have any leading dimension, also one beyond what a tensor
map's strides hold (2^40 bytes): every form computes it.  Whole numbers below 5
in every factor, exact in every form but fp8, whose block scales are not powers
of two (three roundings of each of two scales and the sum: 8 2^-24)."""
import numpy as np
import pytest

from gbpoly import Precision

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", list(Precision), ids=lambda p: p.name.lower())
@pytest.mark.parametrize("ldc", [2 ** 38 - 4, 2 ** 38, 2 ** 44])
def test_one_row_any_stride(ctx, prec, ldc):
    N, K = 260, 64
    rng = np.random.default_rng(1)
    A = rng.choice([-4, -2, -1, 0, 1, 2, 4], (1, K)).astype(np.float32)
    B = rng.choice([-4, -2, -1, 0, 1, 2, 4], (K, N)).astype(np.float32)
    C = rng.integers(-4, 5, (1, N)).astype(np.float32)
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(C)
    ctx.gemm(prec, 1, N, K, 1.0, dA, K, dB, N, 2.0, dC, ldc)
    ctx.synchronize()
    got, want = ctx.download(dC, C.shape), A @ B + 2 * C
    if prec == Precision.FP8:
        assert (np.abs(got - want) <= 8 * 2.0 ** -24 * (np.abs(A) @ np.abs(B) + 2 * np.abs(C))).all()
    else:
        np.testing.assert_array_equal(got, want)
    for b in (dA, dB, dC):
        ctx.free(b)
