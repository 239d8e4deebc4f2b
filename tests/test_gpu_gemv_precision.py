"""Column sums of matrix-vector products are at least as close to FP64 as sums of
64 rows in sequence (one rounding per fused multiply-add) that are then added
exactly: how many rows a CTA takes must not lengthen the chains of additions.

Uniform inputs; the two errors are compared as norms over thousands of columns,
where they vary by about a per cent."""
import numpy as np
import pytest

from gbpoly import Op

pytestmark = pytest.mark.gpu


def chains_of(A, x, n):
    """A^T x with FP32 sums of n rows in sequence, added in FP64."""
    rows, cols = A.shape
    pad = -rows % n
    a = np.pad(A, ((0, pad), (0, 0))).reshape(-1, n, cols).astype(np.float64)
    v = np.pad(x, (0, pad)).reshape(-1, n).astype(np.float64)
    acc = np.zeros((a.shape[0], cols), np.float32)
    for k in range(n):
        acc = (acc.astype(np.float64) + a[:, k] * v[:, k, None]).astype(np.float32)
    return acc.astype(np.float64).sum(0)


@pytest.mark.parametrize("rows,cols,both", [(3832, 7834, True), (4096, 4096, True), (4500, 6000, False), (2300, 9001, True)])
def test_column_sums(ctx, rows, cols, both):
    rng = np.random.default_rng(rows)
    A = rng.uniform(-1, 1, (rows, cols)).astype(np.float32)
    x = rng.uniform(-1, 1, rows).astype(np.float32)
    p = rng.uniform(-1, 1, cols).astype(np.float32)
    dA, dx, dp, dy, dq = ctx.upload(A), ctx.upload(x), ctx.upload(p), ctx.alloc(cols * 4), ctx.alloc(rows * 4)
    if both:
        ctx.gemv_pair(rows, cols, dA, cols, [(Op.T, 1.0, 0.0, dx, dy), (Op.N, 1.0, 0.0, dp, dq)])
    else:
        ctx.gemv(Op.T, rows, cols, 1.0, dA, cols, dx, 0.0, dy)
    ctx.synchronize()
    want = A.astype(np.float64).T @ x.astype(np.float64)
    got = np.linalg.norm(ctx.download(dy, (cols,)) - want) / np.linalg.norm(want)
    assert got <= np.linalg.norm(chains_of(A, x, 64) - want) / np.linalg.norm(want)
    for b in (dA, dx, dp, dy, dq):
        ctx.free(b)
