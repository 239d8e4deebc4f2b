"""Plain FP32 kernel: every way an operand tile is fetched (TMA, words of an
unaligned MN-major operand, words of a K-major one), K splits over a cluster,
and the mirrored triangle, at tile edges.

Tolerance: every output is a sum of K products in some order, scaled, plus
beta * C.  With u = 2^-24 its error is at most (K + 12) u (|alpha| |A||B| +
|beta| |C|) elementwise (one rounding per product-sum step, at most 8 for the
partial sums of a split and 4 in the epilogue), whatever the order, to first
order in u.
"""
import numpy as np
import pytest

from gbpoly import Op, Precision

pytestmark = pytest.mark.gpu


def stored(rng, rows, cols, ld, off):
    """A rows x cols matrix in a flat buffer: leading dimension ld, starting `off` floats in."""
    flat = rng.uniform(-1, 1, off + rows * ld).astype(np.float32)
    return flat, flat[off:].reshape(rows, ld)[:, :cols].astype(np.float64)


def check(got, a, b, c, alpha, beta):
    K = a.shape[1]
    ref = alpha * (a @ b) + beta * c
    bound = (K + 12) * 2.0 ** -24 * (abs(alpha) * (np.abs(a) @ np.abs(b)) + abs(beta) * np.abs(c))
    assert (np.abs(got.astype(np.float64) - ref) <= bound * (1 + 1e-5)).all()


@pytest.mark.parametrize("op_a", [Op.N, Op.T])
@pytest.mark.parametrize("op_b", [Op.N, Op.T])
@pytest.mark.parametrize("pad,off", [(0, 0), (1, 0), (4, 1)], ids=["packed", "ld+1", "offset"])
@pytest.mark.parametrize("mnk", [(1, 1, 1), (127, 129, 31), (128, 128, 32), (129, 257, 33), (130, 64, 611), (260, 300, 1029)])
def test_every_fetch_and_split(ctx, op_a, op_b, pad, off, mnk):
    M, N, K = mnk
    rng = np.random.default_rng(M + 7 * N + 13 * K + pad + off)
    ra, ca = (M, K) if op_a == Op.N else (K, M)
    rb, cb = (K, N) if op_b == Op.N else (N, K)
    fa, a = stored(rng, ra, ca, ca + pad, off)
    fb, b = stored(rng, rb, cb, cb + pad, off)
    fc, c = stored(rng, M, N, N + pad, off)
    dA, dB, dC = ctx.upload(fa), ctx.upload(fb), ctx.upload(fc)
    ctx.gemm(Precision.FP32, M, N, K, 1.5, dA.ptr + 4 * off, ca + pad, dB.ptr + 4 * off, cb + pad, -0.5,
             dC.ptr + 4 * off, N + pad, op_a=op_a, op_b=op_b)
    ctx.synchronize()
    out = ctx.download(dC, fc.shape)
    check(out[off:].reshape(M, N + pad)[:, :N], a if op_a == Op.N else a.T, b if op_b == Op.N else b.T, c, 1.5, -0.5)
    np.testing.assert_array_equal(out[off:].reshape(M, N + pad)[:, N:], fc[off:].reshape(M, N + pad)[:, N:])
    np.testing.assert_array_equal(out[:off], fc[:off])
    for x in (dA, dB, dC):
        ctx.free(x)


@pytest.mark.parametrize("pad", [0, 3])
@pytest.mark.parametrize("n,k", [(129, 40), (700, 333), (900, 70)])
def test_mirrored_splits(ctx, n, k, pad):
    # syr2k: lower triangle of tiles, split or not, each below the diagonal also stored transposed
    rng = np.random.default_rng(n + k + pad)
    fa, a = stored(rng, n, k, k + pad, 0)
    fb, b = stored(rng, n, k, k + pad, 0)
    fc, c = stored(rng, n, n, n + pad, 0)
    dA, dB, dC = ctx.upload(fa), ctx.upload(fb), ctx.upload(fc)
    ctx.syr2k(Precision.FP32, n, k, 2.0, dA, k + pad, dB, k + pad, 0.75, dC, n + pad)
    ctx.synchronize()
    got = ctx.download(dC, fc.shape).reshape(n, n + pad)[:, :n]
    check(got, np.hstack([a, b]), np.vstack([b.T, a.T]), c, 2.0, 0.75)
    for x in (dA, dB, dC):
        ctx.free(x)
