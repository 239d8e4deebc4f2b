"""The K split of a launch's last round of CTA-pair tiles, with K long enough that
the library splits it: every way of writing C (boxes of several rounds, the ring
of one round, staged rows), ragged edges, mirrored tiles and the halves of
256 x 128 tiles above the diagonal, the scaled form included.

The split shows as a result that differs from the whole tiles' in some element
(another order of two partial sums, 1e-6 relative, the bound the other K-split
tests use), is the same on every run, and is as close to the FP64 product."""
import numpy as np
import pytest

from gbpoly import Op, Precision

pytestmark = pytest.mark.gpu

# form -> (pairs on 256 x 256, pairs on 256 x 128); normwise error bound against FP64 of the form
FORMS = {Precision.BF16X3: (3, 6, 2e-5), Precision.TF32X3: (3, 6, 5e-6), Precision.BF16X6: (3, 6, 5e-6),
         Precision.TF32: (3, 6, 1e-3), Precision.FP16X3: (2, 3, 5e-6)}


class Case:
    def __init__(self, ctx, op, M, N, K, ldc, seed):
        rng = np.random.default_rng(seed)
        self.ctx, self.op, self.M, self.N, self.K, self.ldc = ctx, op, M, N, K, ldc
        A = rng.standard_normal((M, K)).astype(np.float32)
        B = rng.standard_normal((N, K)).astype(np.float32)
        self.C = rng.standard_normal((M, ldc)).astype(np.float32)
        self.dA, self.dB, self.dC = ctx.upload(A), ctx.upload(B), ctx.upload(self.C)
        self.d64 = [ctx.alloc(x.size * 8) for x in (A, B, self.C)]
        for d, s, n in zip(self.d64, (self.dA, self.dB, self.dC), (A.size, B.size, self.C.size)):
            ctx.convert_f32_f64(s, d, n)
        a, b, c = self.d64
        if op == "syr2k":
            ctx.syr2k_f64(N, K, 1.5, a, K, b, K, -0.5, c, ldc)
        else:
            ctx.gemm_f64(M, N, K, 1.5, a, K, a if op == "syrk" else b, K, -0.5, c, ldc, op_b=Op.T)
        ctx.synchronize()

    def run(self, prec, config, tail):
        """(result, its normwise error against FP64)"""
        ctx, M, N, K = self.ctx, self.M, self.N, self.K
        ctx.h2d(self.dC, self.C)
        ctx.config_set(prec, M, N, K, config)
        ctx.tail_split(tail)
        try:
            if self.op == "syrk":
                ctx.syrk(prec, N, K, 1.5, self.dA, K, -0.5, self.dC, self.ldc)
            elif self.op == "syr2k":
                ctx.syr2k(prec, N, K, 1.5, self.dA, K, self.dB, K, -0.5, self.dC, self.ldc)
            else:
                ctx.gemm(prec, M, N, K, 1.5, self.dA, K, self.dB, K, -0.5, self.dC, self.ldc, op_b=Op.T)
            ctx.synchronize()
        finally:
            ctx.tail_split(True)
        out = ctx.download(self.dC, self.C.shape)
        np.testing.assert_array_equal(out[:, N:], self.C[:, N:])  # padding untouched
        return out[:, :N], ctx.error_norms(self.dC, self.ldc, self.d64[2], self.ldc, M, N)[1]

    def free(self):
        for b in (self.dA, self.dB, self.dC, *self.d64):
            self.ctx.free(b)


# op, M, N, K, ldc, which of the form's configurations: tiles on 76 resident pairs
CASES = {
    "boxes_256": (None, 2500, 2436, 2100, 2436, 0),     # 100 tiles: 24 split, ragged
    "staged_256": (None, 2500, 2435, 2100, 2435, 0),    # the same through rows TMA cannot address
    "ring_256": (None, 1500, 1396, 2100, 1400, 0),      # 36 tiles, all split
    "boxes_128": (None, 2500, 1204, 2100, 1204, 1),     # 100 tiles of 256 x 128
    "staged_128": (None, 2500, 1203, 2100, 1203, 1),
    "ring_128": (None, 900, 1148, 2100, 1148, 1),       # 36
    "mirrored_256": ("syrk", 3212, 3212, 2100, 3212, 0),  # 91 of the lower triangle
    "mirrored_128": ("syrk", 2300, 2300, 2100, 2300, 1),  # 90, their halves mirrored by themselves
    "mirrored_staged_128": ("syrk", 2299, 2299, 2100, 2299, 1),
    "mirrored_ring_128": ("syrk", 1200, 1200, 2100, 1200, 1),  # 30, all split
    "two_products_256": ("syr2k", 3212, 3212, 1100, 3212, 0),
    "two_products_128": ("syr2k", 2300, 2300, 1100, 2300, 1),
}


@pytest.mark.parametrize("name", list(CASES))
def test_split_rounds(ctx, name):
    if ctx.device_props()["sm_count"] != 152:
        pytest.skip("tile counts of a 152-SM device")
    op, M, N, K, ldc, which = CASES[name]
    case = Case(ctx, op, M, N, K, ldc, sum(map(ord, name)))
    try:
        for prec, (*configs, bound) in FORMS.items():
            config = configs[which]
            whole, e_whole = case.run(prec, config, False)
            split, e_split = case.run(prec, config, True)
            again, _ = case.run(prec, config, True)
            np.testing.assert_array_equal(split.view(np.uint32), again.view(np.uint32), err_msg=prec.name)
            assert (split != whole).any(), prec.name  # K was split
            assert np.linalg.norm(split - whole) / np.linalg.norm(whole) < 1e-6, prec.name
            assert e_whole < bound and e_split < bound, (prec.name, e_whole, e_split)
            ctx.config_set(prec, M, N, K, 0)
    finally:
        case.free()
