"""Column statistics of columns whose sum or mean is not finite.

A column of finite values whose FP32 sum overflows has the mean +inf, and
every (x - mean)^2 is +inf, so its standard deviation is +inf: no term of the
sum may be inf - inf.  The same for a mean that the caller gives.  A column
that itself holds an infinity has x - mean = NaN there, hence NaN.  The other
columns of the same block are unaffected."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INF = np.float32(np.inf)


# chunks of rows with every kind of remainder (128 rows are one batch of loads),
# as clusters (low or wide matrices) and through global partial sums (high, narrow ones)
@pytest.mark.parametrize("rows,cols", [(1, 1), (63, 5), (129, 40), (1000, 33), (2999, 70), (1024, 1300), (3000, 1300),
                                       (5000, 40), (40003, 70)])
@pytest.mark.parametrize("given", [False, True], ids=["overflowed", "given"])
def test_infinite_means_give_infinite_deviations(ctx, rows, cols, given):
    rng = np.random.default_rng(rows + cols)
    X = rng.uniform(-1, 1, (rows, cols)).astype(np.float32)
    big, holds = 0, cols - 1
    if not given:
        X[:, big] = 3e38  # the sum overflows (a single row is given its mean instead)
    if holds != big:
        X[rows // 2, holds] = INF
    dX = ctx.upload(X)
    dm, ds = ctx.alloc(cols * 4), ctx.alloc(cols * 4)
    ctx.column_mean(rows, cols, dX, cols, float(rows), dm)
    ctx.synchronize()
    mean = ctx.download(dm, (cols,))
    if given or rows == 1:
        mean[big] = INF
        ctx.h2d(dm, mean)
        ctx.synchronize()
    ctx.column_stddev(rows, cols, dX, cols, dm, float(rows), 0.005, ds)
    ctx.synchronize()
    sd = ctx.download(ds, (cols,))
    for b in (dX, dm, ds):
        ctx.free(b)
    assert mean[big] == INF and sd[big] == INF
    if holds != big:
        assert mean[holds] == INF and np.isnan(sd[holds])
    rest = slice(1, cols - 1)
    if cols > 2:
        ref = np.sqrt(((X[:, rest].astype(np.float64) - X[:, rest].astype(np.float64).mean(0)) ** 2).mean(0))
        ref[ref <= 0.005] = 1.0
        np.testing.assert_allclose(sd[rest], ref, rtol=1e-5)
