"""Column means and standard deviations at the edges of their column blocks,
row chunks and load batches: narrow matrices (partials in global memory) and
wide ones (chunks of a cluster).

Tolerance: a sum of n terms in any order is within n 2^-24 sum |x| of the exact
one; the standard deviation's sum of squares adds the rounding of x - mean and
of the mean (relative 2 (n + 8) 2^-24 of the sum of (|x| + |mean|)^2), halved by
the square root."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("shape", [(1, 1), (7, 33), (65, 31), (513, 40), (1, 1300), (63, 1249), (130, 1216), (1030, 1217),
                                   (129, 2050), (3073, 70)], ids=str)
def test_mean_and_stddev(ctx, shape, pad):
    rows, cols = shape
    rng = np.random.default_rng(rows + cols + pad)
    X = (rng.standard_normal((rows, cols + pad)) + 2.0).astype(np.float32)
    dX, dm, ds = ctx.upload(X), ctx.alloc(cols * 4), ctx.alloc(cols * 4)
    ctx.column_mean(rows, cols, dX, cols + pad, float(rows), dm)
    ctx.column_stddev(rows, cols, dX, cols + pad, dm, float(rows), 1e-3, ds)
    ctx.synchronize()
    mean, sd = ctx.download(dm, (cols,)).astype(np.float64), ctx.download(ds, (cols,)).astype(np.float64)
    x = X[:, :cols].astype(np.float64)
    assert (np.abs(mean - x.mean(0)) <= (rows + 2) * U * np.abs(x).mean(0)).all()
    var = np.square(x - mean).mean(0)  # about the mean the kernel was given
    bound = 2 * (rows + 8) * U * np.square(np.abs(x) + np.abs(mean)).mean(0)
    want = np.sqrt(var)
    clear = np.abs(want - 1e-3) > 1e-4  # away from the eps clamp
    low, high = np.sqrt(np.maximum(var - bound, 0)) * (1 - 4 * U), np.sqrt(var + bound) * (1 + 4 * U)
    one = clear & (want < 1e-3) & (high < 1e-3)
    assert (sd[one] == 1.0).all()
    rest = clear & (low > 1e-3)
    assert ((sd[rest] >= low[rest]) & (sd[rest] <= high[rest])).all()
    for b in (dX, dm, ds):
        ctx.free(b)
