"""Matrix-vector passes at the most rows a call takes: the last group of rows,
whose end lies beyond 2^31, is still read and written (one column, so that a
matrix and a vector of rows are 8.6 GB each)."""
import numpy as np
import pytest

from gbpoly import Context, Op

pytestmark = pytest.mark.gpu
ROWS = 2 ** 31 - 1
SET = [0, 12345, ROWS // 2, ROWS - 3000000, ROWS - 100000, ROWS - 33, ROWS - 17, ROWS - 16, ROWS - 1]


@pytest.fixture
def own():  # its scratch of 8.6 GB and more goes with it
    c = Context(0)
    yield c
    c.close()


def zeros_but_ones(c):
    d = c.alloc(ROWS * 4)
    c.memset(d, 0, ROWS * 4)
    one = np.ones(1, np.float32)
    for r in SET:
        c.h2d(d.ptr + 4 * r, one)
    return d


def ones_at(c, d, value):
    for r in SET:
        assert c.download(d.ptr + 4 * r, (1,))[0] == value, r
    for r in (1, ROWS - 2, ROWS - 18, ROWS - 200000):
        assert c.download(d.ptr + 4 * r, (1,))[0] == 0, r


def test_row_and_column_sums(own):
    c = own
    dA, dx, dq = zeros_but_ones(c), zeros_but_ones(c), c.alloc(ROWS * 4)
    two, ds = c.upload(np.full(1, 2, np.float32)), c.upload(np.zeros(1, np.float32))
    c.gemv_pair(ROWS, 1, dA, 1, [(Op.T, 1.0, 0.0, dx, ds), (Op.N, 1.0, 0.0, two, dq)])
    c.synchronize()
    assert c.download(ds, (1,))[0] == len(SET)
    ones_at(c, dq, 2)
    for b in (dA, dx, dq, two, ds):
        c.free(b)


def test_gesummv(own):
    c = own
    dA, dB, dt, dy = (zeros_but_ones(c) for _ in range(4))
    two = c.upload(np.full(1, 2, np.float32))
    c.gesummv(ROWS, 1, 1.0, dA, 1, dB, 1, two, 1.0, dt, dy)  # tmp = 1 + 2, y = tmp + (1 + 2)
    c.synchronize()
    ones_at(c, dt, 3)
    ones_at(c, dy, 6)
    for b in (dA, dB, dt, dy, two):
        c.free(b)
