"""Plain FP32 contractions that run as two launches on a GB300, each with its own
split of K: the profile shows both, and the results are exact (whole numbers in
[-4, 4], every partial sum below 2^24)."""
import numpy as np
import pytest

from gbpoly import Op, Precision

pytestmark = pytest.mark.gpu
P = Precision.FP32


def launches(ctx, call):
    ctx.synchronize()
    ctx.profile(True)
    ctx.profile_read()
    call()
    ctx.synchronize()
    n = sum(c for c, _ in ctx.profile_read().values())
    ctx.profile(False)
    return n


@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("M,N,K", [(1007, 2632, 400), (1501, 1023, 2047), (1408, 2124, 264), (2458, 1059, 1369)])
def test_rows_of_tiles_in_two_launches(ctx, M, N, K, pad):
    if ctx.device_props()["sm_count"] != 152:
        pytest.skip("plans of a 152-SM device")
    rng = np.random.default_rng(M)
    A, B, C = (rng.integers(-4, 5, s).astype(np.float32) for s in ((M, K + pad), (K, N + pad), (M, N + pad)))
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(C)
    assert launches(ctx, lambda: ctx.gemm(P, M, N, K, 1.0, dA, K + pad, dB, N + pad, 1.0, dC, N + pad)) == 2
    want = C.copy()
    want[:, :N] += (A[:, :K].astype(np.float64) @ B[:, :N].astype(np.float64)).astype(np.float32)
    np.testing.assert_array_equal(ctx.download(dC, C.shape), want)
    for x in (dA, dB, dC):
        ctx.free(x)


@pytest.mark.parametrize("n,k", [(2304, 512), (2560, 600)])
def test_syr2k_in_two_launches(ctx, n, k):
    if ctx.device_props()["sm_count"] != 152:
        pytest.skip("plans of a 152-SM device")
    rng = np.random.default_rng(n)
    A, B, C = (rng.integers(-4, 5, s).astype(np.float32) for s in ((n, k), (n, k), (n, n)))
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(C)
    assert launches(ctx, lambda: ctx.syr2k(P, n, k, 1.0, dA, k, dB, k, 1.0, dC, n)) == 2
    p = A.astype(np.float64) @ B.astype(np.float64).T
    np.testing.assert_array_equal(ctx.download(dC, C.shape), (p + p.T + C).astype(np.float32))
    # a symmetric product is one launch (its split is the full square's)
    assert launches(ctx, lambda: ctx.gemm(P, n, n, k, 1.0, dA, k, dA, k, 0.0, dC, n, op_b=Op.T)) == 1
    for x in (dA, dB, dC):
        ctx.free(x)
