"""Matrix-vector kernels at the edges of their row groups, column tiles and
load widths, aligned and not.

Tolerance: a dot of K terms summed in any order, scaled, plus beta * y: at most
(K + 8) 2^-24 (|alpha| |A||x| + |beta| |y|) elementwise.  atax's y adds the
error of tmp carried through |A^T|."""
import numpy as np
import pytest

from gbpoly import Op

pytestmark = pytest.mark.gpu

U = 2.0 ** -24
SHAPES = [(1, 1), (3, 5), (15, 1024), (17, 1025), (31, 255), (613, 2047), (1300, 2049), (40, 4100), (33, 8192), (700, 4096)]


def make(rows, cols, pad, seed):
    rng = np.random.default_rng(seed)
    return rng, rng.uniform(-1, 1, (rows, cols + pad)).astype(np.float32)


def f64(a):
    return a.astype(np.float64)


@pytest.mark.parametrize("pad", [0, 3, 4])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_atax(ctx, shape, pad):
    rows, cols = shape
    rng, A = make(rows, cols, pad, rows + cols + pad)
    x, tmp, y = (rng.uniform(-1, 1, n).astype(np.float32) for n in (cols, rows, cols))
    dA, dx, dt, dy = (ctx.upload(v) for v in (A, x, tmp, y))
    ctx.atax(rows, cols, dA, cols + pad, dx, dt, dy)
    ctx.synchronize()
    a = f64(A[:, :cols])
    t = f64(tmp) + a @ f64(x)
    tb = (cols + 8) * U * (np.abs(a) @ np.abs(f64(x)) + np.abs(f64(tmp)))
    assert (np.abs(f64(ctx.download(dt, (rows,))) - t) <= tb).all()
    yb = (rows + 8) * U * (np.abs(a).T @ np.abs(t) + np.abs(f64(y))) + np.abs(a).T @ tb * (1 + 1e-3)
    assert (np.abs(f64(ctx.download(dy, (cols,))) - (f64(y) + a.T @ t)) <= yb).all()
    for b in (dA, dx, dt, dy):
        ctx.free(b)


@pytest.mark.parametrize("pad", [0, 1, 4])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_pair_and_gesummv(ctx, shape, pad):
    rows, cols = shape
    rng, A = make(rows, cols, pad, 7 * rows + cols + pad)
    B = rng.uniform(-1, 1, A.shape).astype(np.float32)
    xc, xr, s, q = (rng.uniform(-1, 1, n).astype(np.float32) for n in (cols, rows, cols, rows))
    dA, dB, dxc, dxr, ds, dq, dt = (ctx.upload(v) for v in (A, B, xc, xr, s, q, q))
    ctx.gemv_pair(rows, cols, dA, cols + pad, [(Op.T, 1.5, 0.5, dxr, ds), (Op.N, -1.0, 0.25, dxc, dq)])
    ctx.synchronize()
    a, b = f64(A[:, :cols]), f64(B[:, :cols])
    aa = np.abs(a)
    assert (np.abs(f64(ctx.download(ds, (cols,))) - (0.5 * f64(s) + 1.5 * a.T @ f64(xr)))
            <= (rows + 8) * U * (1.5 * aa.T @ np.abs(f64(xr)) + 0.5 * np.abs(s))).all()
    assert (np.abs(f64(ctx.download(dq, (rows,))) - (0.25 * f64(q) - a @ f64(xc)))
            <= (cols + 8) * U * (aa @ np.abs(f64(xc)) + 0.25 * np.abs(q))).all()
    ctx.h2d(dq, q)
    ctx.gesummv(rows, cols, 1.5, dA, cols + pad, dB, cols + pad, dxc, 0.5, dt, dq)
    ctx.synchronize()
    t = f64(q) + a @ f64(xc)
    tb = (cols + 8) * U * (aa @ np.abs(f64(xc)) + np.abs(q))
    assert (np.abs(f64(ctx.download(dt, (rows,))) - t) <= tb).all()
    yb = (cols + 8) * U * (1.5 * np.abs(t) + 0.5 * (np.abs(q) + np.abs(b) @ np.abs(f64(xc)))) + 1.5 * tb
    assert (np.abs(f64(ctx.download(dq, (rows,))) - (1.5 * t + 0.5 * (f64(q) + b @ f64(xc)))) <= yb).all()
    for v in (dA, dB, dxc, dxr, ds, dq, dt):
        ctx.free(v)
