"""Column statistics at the most rows a call takes: the last chunk of rows,
whose end lies beyond 2^31, is part of the sums (one column of 8.6 GB)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROWS = 2 ** 31 - 1
SET = [0, 12345, ROWS // 2, ROWS - 3000000, ROWS - 100000, ROWS - 65, ROWS - 33, ROWS - 9, ROWS - 1]


def test_sums_of_all_rows(ctx):
    dX = ctx.alloc(ROWS * 4)
    ctx.memset(dX, 0, ROWS * 4)
    one = np.ones(1, np.float32)
    for r in SET:
        ctx.h2d(dX.ptr + 4 * r, one)
    dm, ds, zero = ctx.upload(one * 0), ctx.upload(one * 0), ctx.upload(one * 0)
    ctx.column_mean(ROWS, 1, dX, 1, 1.0, dm)
    ctx.column_stddev(ROWS, 1, dX, 1, zero, 1.0, 0.0, ds)
    ctx.synchronize()
    assert ctx.download(dm, (1,))[0] == 9
    assert ctx.download(ds, (1,))[0] == 3
    for b in (dX, dm, ds, zero):
        ctx.free(b)
