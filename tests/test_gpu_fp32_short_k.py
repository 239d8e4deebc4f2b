"""Plain FP32 with short K and with rows off 16-byte boundaries: the 64 x 64
kernel, the lines between it and the 128 x 128 one, and the 128 x 128 kernel's
way of writing C whose rows are off those boundaries.

Inputs are whole numbers in [-4, 4] with K <= 200, so every partial sum is a
whole number below 2^24 and exact in FP32 in any order: equality, not a bound.
"""
import numpy as np
import pytest

from gbpoly import Op, Precision

pytestmark = pytest.mark.gpu
P = Precision.FP32


def ints(seed, r, c):
    return np.random.default_rng(seed).integers(-4, 5, (r, c)).astype(np.float32)


def kernels(ctx, call):
    """The FP32 kernels that `call` launches."""
    ctx.synchronize()
    ctx.profile(True)
    ctx.profile_read()
    call()
    ctx.synchronize()
    names = ctx.profile_read()
    ctx.profile(False)
    return {k: v[0] for k, v in names.items()}


def check(ctx, M, N, K, ops=(Op.N, Op.N), pads=(1, 1, 1), same=False, beta=1.0, dual=False):
    """One product against whole numbers; returns the kernels it ran."""
    ra, ca = (K, M) if ops[0] == Op.T else (M, K)
    rb, cb = (N, K) if ops[1] == Op.T else (K, N)
    A = ints(M + K, ra, ca + pads[0])
    B = A if same else ints(N + 2 * K, rb, cb + pads[1])
    C = ints(M + N, M, N + pads[2])
    dA = ctx.upload(A)
    dB = dA if same else ctx.upload(B)
    dC = ctx.upload(C)
    if dual:
        ran = kernels(ctx, lambda: ctx.syr2k(P, N, K, 1.0, dA, A.shape[1], dB, B.shape[1], beta, dC, C.shape[1]))
    else:
        ran = kernels(ctx, lambda: ctx.gemm(P, M, N, K, 1.0, dA, A.shape[1], dB, B.shape[1], beta, dC, C.shape[1],
                                            op_a=ops[0], op_b=ops[1]))
    a = (A[:, :ca].T if ops[0] == Op.T else A[:, :ca]).astype(np.float64)
    b = (B[:, :cb].T if ops[1] == Op.T else B[:, :cb]).astype(np.float64)
    want = C.copy()
    prod = a @ b
    want[:, :N] = prod + (prod.T if dual else 0) + beta * C[:, :N]
    np.testing.assert_array_equal(ctx.download(dC, C.shape), want)
    for x in {dA, dB, dC}:
        ctx.free(x)
    return ran


OPS = [(Op.N, Op.N), (Op.T, Op.N), (Op.N, Op.T), (Op.T, Op.T)]


@pytest.mark.parametrize("ops", OPS)
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (64, 64, 16), (65, 63, 17), (200, 301, 32), (130, 70, 33), (500, 130, 48),
                                   (129, 257, 64), (70, 500, 65), (333, 222, 80), (130, 131, 81), (1500, 1700, 16),
                                   (2500, 1500, 31)])
def test_short_k_off_boundaries(ctx, ops, M, N, K):
    ran = check(ctx, M, N, K, ops, pads=(1 - K % 2 if ops[0] == Op.N else 1 - M % 2, 1, 1), beta=-0.5)
    assert ("sgemm_tiled" in ran) == (K <= 80 and not (K > 16 and M == 2500))


@pytest.mark.parametrize("K", [1, 32, 48, 64, 80, 96])
@pytest.mark.parametrize("n", [1, 64, 130, 333])
def test_short_k_symmetric(ctx, n, K):
    pad = 1 - K % 2 if K % 4 else 1
    for ops in ((Op.N, Op.T), (Op.T, Op.N)):
        check(ctx, n, n, K, ops, pads=(pad if ops[0] == Op.N else 1 - n % 2,) * 3, same=True, beta=0.5)
    ran = check(ctx, n, n, K, (Op.N, Op.T), pads=(pad, pad, 3), dual=True)
    assert ("sgemm_tiled" in ran) == (K <= 64)


def test_empty_k(ctx):
    C = ints(1, 70, 131)
    dA, dC = ctx.alloc(64), ctx.upload(C)
    ctx.gemm(P, 70, 130, 0, 2.0, dA, 1, dA, 130, 0.5, dC, 131)
    ctx.synchronize()
    C[:, :130] *= 0.5
    np.testing.assert_array_equal(ctx.download(dC, C.shape), C)
    for x in (dA, dC):
        ctx.free(x)


# operands on boundaries, C off them: one and several rounds of tiles, tiles cut in
# both directions, the mirrored tiles of symmetric products, C read and not read
@pytest.mark.parametrize("beta", [0.0, 1.0])
@pytest.mark.parametrize("M,N,K,kind", [(130, 257, 40, ""), (1537, 1283, 36, ""), (2600, 1289, 64, ""), (257, 257, 36, "same"),
                                        (2049, 2049, 40, "same"), (2305, 2305, 36, "dual"), (129, 129, 200, "dual")])
def test_c_off_boundaries(ctx, beta, M, N, K, kind):
    ran = check(ctx, M, N, K, (Op.N, Op.T), pads=(0, 0, 4 - N % 4 + 1), same=kind == "same", dual=kind == "dual", beta=beta)
    assert "sgemm_tiled" not in ran


def test_both_kernels_give_the_same_bits(ctx):
    # an unsplit product (K = 32 is one round of the 128 x 128 kernel's loop) on the same values, on and off boundaries
    M, N, K = 300, 260, 32
    rng = np.random.default_rng(5)
    A, B, C = (rng.uniform(-1, 1, s).astype(np.float32) for s in ((M, K), (K, N), (M, N)))
    outs = []
    for pad in (0, 1):
        dA = ctx.upload(np.pad(A, ((0, 0), (0, pad))))
        dB, dC = ctx.upload(B), ctx.upload(C)
        ran = kernels(ctx, lambda: ctx.gemm(P, M, N, K, 1.5, dA, K + pad, dB, N, -0.5, dC, N))
        assert ("sgemm_tiled" in ran) == (pad == 1)
        outs.append(ctx.download(dC, C.shape))
        for x in (dA, dB, dC):
            ctx.free(x)
    np.testing.assert_array_equal(outs[0].view(np.uint32), outs[1].view(np.uint32))


@pytest.mark.parametrize("N,K,pad", [(60, 40, 1), (129, 64, 1), (700, 80, 1), (60, 40, 0), (130, 96, 1)])
def test_host_panels_off_boundaries(ctx, N, K, pad):
    M = 2100  # panels of 512 rows, whose own shape would choose otherwise
    rng = np.random.default_rng(N + K)
    A = rng.uniform(-1, 1, (M, K + pad)).astype(np.float32)
    B = rng.uniform(-1, 1, (K, N + pad)).astype(np.float32)
    C = rng.uniform(-1, 1, (M, N + pad)).astype(np.float32)
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(C)
    ctx.gemm(P, M, N, K, 1.5, dA, K + pad, dB, N + pad, 0.5, dC, N + pad)
    ctx.synchronize()
    out = C.copy()
    ctx.gemm_host(P, M, N, K, 1.5, A, K + pad, B, N + pad, 0.5, out, N + pad)
    ctx.synchronize()
    np.testing.assert_array_equal(out, ctx.download(dC, C.shape))
    for x in (dA, dB, dC):
        ctx.free(x)
