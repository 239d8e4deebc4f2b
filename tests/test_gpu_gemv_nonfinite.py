"""atax with infinities in its input vector: an infinite element of x makes
every tmp infinite, and y follows IEEE arithmetic row by row, whatever the
rows of a CTA's last, part-filled group.

Every case is exact: the matrix is positive, so tmp and y are +inf (or, at a
zero of the matrix, 0 * inf = NaN) in any order of summation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INF = np.float32(np.inf)


# one to eight column tiles (16, 8 or 4 rows at a time), rows that leave every
# kind of remainder, and rows below one group
@pytest.mark.parametrize("rows,cols,pad", [(1, 2, 0), (3, 5, 1), (17, 100, 0), (37, 1500, 0), (311, 3000, 4),
                                           (613, 4097, 1), (1001, 8192, 0), (1300, 1024, 0), (5, 9000, 0)])
def test_atax_keeps_infinities(ctx, rows, cols, pad):
    rng = np.random.default_rng(rows + cols)
    A = rng.uniform(0.5, 1.5, (rows, cols + pad)).astype(np.float32)
    x = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    x[cols // 2] = INF
    dA, dx = ctx.upload(A), ctx.upload(x)
    dt, dy = ctx.upload(np.zeros(rows, np.float32)), ctx.upload(np.zeros(cols, np.float32))
    ctx.atax(rows, cols, dA, cols + pad, dx, dt, dy)
    ctx.synchronize()
    tmp, y = ctx.download(dt, (rows,)), ctx.download(dy, (cols,))
    for b in (dA, dx, dt, dy):
        ctx.free(b)
    np.testing.assert_array_equal(tmp, np.full(rows, INF))
    np.testing.assert_array_equal(y, np.full(cols, INF))


def test_atax_at_the_largest_row_count(ctx):
    """2^31 - 1 rows, the most a call takes: the row counter of the last group
    stays inside the matrix (one column, so that A and tmp are 8.6 GB each)."""
    rows = 2 ** 31 - 1
    dA, dt = ctx.alloc(rows * 4), ctx.alloc(rows * 4)
    one = np.ones(1, np.float32)
    dx, dy = ctx.upload(one), ctx.upload(np.zeros(1, np.float32))
    ctx.memset(dA, 0, rows * 4)
    ctx.memset(dt, 0, rows * 4)
    set_rows = [0, 12345, rows - 17, rows - 16, rows - 2, rows - 1]
    for r in set_rows:
        ctx.h2d(dA.ptr + 4 * r, one)
    ctx.synchronize()
    ctx.atax(rows, 1, dA, 1, dx, dt, dy)
    ctx.synchronize()
    assert ctx.download(dy, (1,))[0] == len(set_rows)
    for r in set_rows:
        assert ctx.download(dt.ptr + 4 * r, (1,))[0] == 1
    for b in (dA, dt, dx, dy):
        ctx.free(b)
