"""CTA pairs on 256 x 128 tiles, launches of one unit per CTA (C through TMA in
the pipeline's stages), and the K split of all their tiles.

Whole tiles sum the same chunks in the same order in every configuration, so
without a K split the results are bitwise those of the 1-CTA 128 x 128 ones;
with it only the order of two partial sums differs (1e-6 relative, the bound
the other K-split tests use)."""
import numpy as np
import pytest

from gbpoly import Op, Precision

pytestmark = pytest.mark.gpu

# form -> (1-CTA 128 x 128, pairs 256 x 256, pairs 256 x 128)
FORMS = {Precision.BF16X3: (2, 3, 6), Precision.TF32X3: (2, 3, 6), Precision.BF16X6: (0, 3, 6),
         Precision.TF32: (2, 3, 6), Precision.FP16X3: (1, 2, 3)}


def matrices(shape, seed, symmetric=False):
    M, N, K = shape
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((M, K)).astype(np.float32)
    B = rng.standard_normal((N, K) if symmetric else (K, N)).astype(np.float32)
    return A, B, rng.standard_normal((M, N)).astype(np.float32)


def run(ctx, prec, config, A, B, C, beta, tail, ldc=None, op=None):
    M, N = C.shape
    K = A.shape[1]
    ldc = ldc or N
    Cp = np.zeros((M, ldc), np.float32)
    Cp[:, :N] = C
    Cp[:, N:] = 7.0
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(Cp)
    ctx.config_set(prec, M, N, K, config)
    ctx.tail_split(tail)
    try:
        if op == "syrk":
            ctx.syrk(prec, N, K, 1.5, dA, K, beta, dC, ldc)
        elif op == "syr2k":
            ctx.syr2k(prec, N, K, 1.5, dA, K, dB, K, beta, dC, ldc)
        else:
            ctx.gemm(prec, M, N, K, 1.5, dA, K, dB, N, beta, dC, ldc)
        ctx.synchronize()
    finally:
        ctx.tail_split(True)
    out = ctx.download(dC, Cp.shape)
    for b in (dA, dB, dC):
        ctx.free(b)
    assert (out[:, N:] == 7.0).all()
    return out[:, :N]


@pytest.mark.parametrize("prec", list(FORMS), ids=lambda p: p.name.lower())
@pytest.mark.parametrize("beta", [0.0, -0.5])
@pytest.mark.parametrize("shape,ldc", [((1, 4, 1), 4), ((129, 132, 65), 132), ((257, 260, 200), 264), ((300, 131, 129), 131),
                                       ((700, 1028, 600), 1028)], ids=str)
def test_single_round_is_bitwise_the_square_tiles(ctx, prec, beta, shape, ldc):
    A, B, C = matrices(shape, sum(shape))
    square, *pairs = (run(ctx, prec, c, A, B, C, beta, False, ldc) for c in FORMS[prec])
    staged = run(ctx, prec, FORMS[prec][0], A, B, C, beta, False, ldc + 1)  # rows TMA cannot address
    np.testing.assert_array_equal(staged.view(np.uint32), square.view(np.uint32))
    for got in pairs:
        np.testing.assert_array_equal(got.view(np.uint32), square.view(np.uint32))


@pytest.mark.parametrize("prec", list(FORMS), ids=lambda p: p.name.lower())
@pytest.mark.parametrize("op", ["syrk", "syr2k"])
@pytest.mark.parametrize("n,k", [(4, 3), (128, 64), (260, 70), (516, 200), (901, 90)])
def test_symmetric_updates_are_bitwise_the_square_tiles(ctx, prec, op, n, k):
    # the halves of a 256 x 128 tile on, below and above the diagonal; n = 901:
    # staged C.  (256 x 256 tiles compute both triangles of their diagonal tile,
    # where the two cross products add in the other order: not the same bits.)
    A, B, C = matrices((n, n, k), n + k, symmetric=True)
    square, pair, narrow = (run(ctx, prec, c, A, B, C, 0.75, False, op=op) for c in FORMS[prec])
    np.testing.assert_array_equal(narrow.view(np.uint32), square.view(np.uint32))
    assert np.linalg.norm(pair - square) / np.linalg.norm(square) < 1e-6


@pytest.mark.parametrize("prec", list(FORMS), ids=lambda p: p.name.lower())
@pytest.mark.parametrize("op,shape", [(None, (130, 260, 2100)), (None, (520, 131, 3000)), ("syrk", (388, 388, 2500)),
                                      ("syr2k", (260, 260, 2000))], ids=str)
def test_k_split_of_all_tiles(ctx, prec, op, shape):
    A, B, C = matrices(shape, sum(shape), symmetric=op is not None)
    for config in FORMS[prec][1:]:
        whole = run(ctx, prec, config, A, B, C, -0.5, False, op=op)
        split, again = (run(ctx, prec, config, A, B, C, -0.5, True, op=op) for _ in range(2))
        np.testing.assert_array_equal(split.view(np.uint32), again.view(np.uint32))
        assert (split != whole).any()  # K was split
        assert np.linalg.norm(split - whole) / np.linalg.norm(whole) < 1e-6


def test_host_panels_split_like_the_whole_call(ctx):
    # two panels of 512 rows of a call whose every tile splits its K
    M, N, K = 1024, 256, 2048
    A, B, C = matrices((M, N, K), 3)
    dA, dB, dC = ctx.upload(A), ctx.upload(B), ctx.upload(C)
    for prec in (Precision.BF16X3, Precision.TF32X3, Precision.BF16X6):
        ctx.config_set(prec, M, N, K, 6)
        ctx.h2d(dC, C)
        ctx.gemm(prec, M, N, K, 1.0, dA, K, dB, N, 0.5, dC, N, op_a=Op.N, op_b=Op.N)
        ctx.synchronize()
        out = C.copy()
        ctx.gemm_host(prec, M, N, K, 1.0, A, K, B, N, 0.5, out, N)
        ctx.synchronize()
        np.testing.assert_array_equal(out.view(np.uint32), ctx.download(dC, C.shape).view(np.uint32))
    for b in (dA, dB, dC):
        ctx.free(b)


@pytest.mark.parametrize("prec", list(FORMS), ids=lambda p: p.name.lower())
@pytest.mark.parametrize("beta", [0.0, -0.5])
def test_rounds_of_boxes_are_bitwise_the_square_tiles(ctx, prec, beta):
    # more pair tiles than pairs: C box by box, ragged in rows and columns; and
    # the same through rows TMA cannot address
    A, B, C = matrices((2570, 2436, 100), 11)
    square, *pairs = (run(ctx, prec, c, A, B, C, beta, False) for c in FORMS[prec])
    staged = run(ctx, prec, FORMS[prec][1], A, B, C, beta, False, ldc=2437)
    for got in (*pairs, staged):
        np.testing.assert_array_equal(got.view(np.uint32), square.view(np.uint32))


@pytest.mark.parametrize("op", ["syrk", "syr2k"])
@pytest.mark.parametrize("prec", [Precision.BF16X3, Precision.FP16X3], ids=lambda p: p.name.lower())
def test_rounds_of_mirrored_boxes(ctx, prec, op):
    # 91 and 182 pair tiles; 256 x 256 tiles as in the symmetric test above
    A, B, C = matrices((3212, 3212, 70), 12, symmetric=True)
    square, pair, narrow = (run(ctx, prec, c, A, B, C, 0.75, False, op=op) for c in FORMS[prec])
    np.testing.assert_array_equal(narrow.view(np.uint32), square.view(np.uint32))
    assert np.linalg.norm(pair - square) / np.linalg.norm(square) < 1e-6
    tail = run(ctx, prec, FORMS[prec][1], A, B, C, 0.75, True, op=op)  # a split last round, where it pays
    assert np.linalg.norm(tail - square) / np.linalg.norm(square) < 1e-6


@pytest.mark.parametrize("mnk", [(1300, 2500, 130), (2450, 2308, 300)], ids=str)
def test_fp8_boxes_are_bitwise_the_square_tiles(ctx, mnk):
    M, N, K = mnk
    A, B, C = matrices(mnk, M)
    outs = [run(ctx, Precision.FP8, c, A, B, C, 0.5, True) for c in (0, 1)]
    staged = run(ctx, Precision.FP8, 1, A, B, C, 0.5, True, ldc=N + 1)
    np.testing.assert_array_equal(outs[1].view(np.uint32), outs[0].view(np.uint32))
    np.testing.assert_array_equal(staged.view(np.uint32), outs[0].view(np.uint32))
