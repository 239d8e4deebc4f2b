"""Column means and standard deviations on both sides of the line between the
two reductions (clusters up to 4096 x 4096, partial sums in global memory
beyond) and far beyond it.

Inputs are whole numbers below 8 with rows a power of two or whole sums below
2^24, so every sum, and with a mean of exactly 3 every sum of squares, is exact
in FP32 in any order: the results are the correctly rounded quotients and roots."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(4096, 70), (4097, 70), (4096, 4096), (64, 4097), (1030, 4128), (30000, 1300),
                                       (500, 9000), (7, 33)])
def test_exact_columns(ctx, rows, cols):
    rng = np.random.default_rng(rows + cols)
    X = rng.integers(0, 7, (rows, cols + 1)).astype(np.float32)
    dX, dm, ds, d3 = ctx.upload(X), ctx.alloc(cols * 4), ctx.alloc(cols * 4), ctx.upload(np.full(cols, 3, np.float32))
    ctx.column_mean(rows, cols, dX, cols + 1, float(rows), dm)
    ctx.column_stddev(rows, cols, dX, cols + 1, d3, float(rows), 0.0, ds)
    ctx.synchronize()
    x = X[:, :cols]
    np.testing.assert_array_equal(ctx.download(dm, (cols,)), x.sum(0, dtype=np.float64).astype(np.float32) / np.float32(rows))
    var = np.square(x - 3).sum(0, dtype=np.float64).astype(np.float32) / np.float32(rows)
    np.testing.assert_array_equal(ctx.download(ds, (cols,)), np.where(var > 0, np.sqrt(var), np.float32(1)))
    for b in (dX, dm, ds, d3):
        ctx.free(b)
