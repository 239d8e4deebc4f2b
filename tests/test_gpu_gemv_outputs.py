"""The final pass of the matrix-vector kernels where it changes how many warps
share an output: many outputs of few partials, few outputs of many, both sides
of a call at once, and no outputs or no partials at all.

Tolerance: a dot of K terms summed in any order, scaled, plus beta * y: at most
(K + 8) 2^-24 (|alpha| |A||x| + |beta| |y|) elementwise."""
import numpy as np
import pytest

from gbpoly import Op

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


def f64(a):
    return a.astype(np.float64)


# (rows, cols): one partial per row output; per column output; 2, 9 and 17 column
# tiles; 1, 16 and more row groups; vectors of one element
@pytest.mark.parametrize("rows,cols", [(78000, 5), (5, 78000), (9000, 1100), (1500, 8300), (40, 17000), (16, 2000),
                                       (250, 600), (5000, 64), (1, 4097), (4097, 1)])
def test_both_sides_of_a_pass(ctx, rows, cols):
    rng = np.random.default_rng(rows + cols)
    A, B = (rng.uniform(-1, 1, (rows, cols)).astype(np.float32) for _ in range(2))
    xc, xr, s, q = (rng.uniform(-1, 1, n).astype(np.float32) for n in (cols, rows, cols, rows))
    dA, dB, dxc, dxr, ds, dq, dt = (ctx.upload(v) for v in (A, B, xc, xr, s, q, q))
    a, b = f64(A), f64(B)
    aa, ab, ax, ar = np.abs(a), np.abs(b), np.abs(f64(xc)), np.abs(f64(xr))
    # bicg: a column term and a row term
    ctx.gemv_pair(rows, cols, dA, cols, [(Op.T, 1.5, 0.5, dxr, ds), (Op.N, -1.0, 0.25, dxc, dq)])
    ctx.synchronize()
    got_s, got_q = ctx.download(ds, (cols,)), ctx.download(dq, (rows,))
    assert (np.abs(f64(got_s) - (0.5 * f64(s) + 1.5 * a.T @ f64(xr)))
            <= (rows + 8) * U * (1.5 * aa.T @ ar + 0.5 * np.abs(s))).all()
    assert (np.abs(f64(got_q) - (0.25 * f64(q) - a @ f64(xc))) <= (cols + 8) * U * (aa @ ax + 0.25 * np.abs(q))).all()
    # mvt: two row terms
    ctx.gemv_pair(rows, cols, dA, cols, [(Op.N, 1.0, 0.0, dxc, dq), (Op.N, 2.0, 1.0, dxc, dt)])
    ctx.synchronize()
    assert (np.abs(f64(ctx.download(dq, (rows,))) - a @ f64(xc)) <= (cols + 8) * U * (aa @ ax)).all()
    assert (np.abs(f64(ctx.download(dt, (rows,))) - (2 * a @ f64(xc) + f64(q)))
            <= (cols + 8) * U * (2 * aa @ ax + np.abs(q))).all()
    # gesummv: two matrices
    ctx.h2d(dt, q)
    ctx.h2d(dq, q)
    ctx.gesummv(rows, cols, 1.5, dA, cols, dB, cols, dxc, 0.5, dt, dq)
    ctx.synchronize()
    t = f64(q) + a @ f64(xc)
    tb = (cols + 8) * U * (aa @ ax + np.abs(q))
    assert (np.abs(f64(ctx.download(dt, (rows,))) - t) <= tb).all()
    yb = 1.5 * tb + 0.5 * (cols + 8) * U * (ab @ ax + np.abs(q)) + 4 * U * (1.5 * np.abs(t) + 0.5 * np.abs(q) + ab @ ax)
    assert (np.abs(f64(ctx.download(dq, (rows,))) - (1.5 * t + 0.5 * (f64(q) + b @ f64(xc)))) <= yb).all()
    for x in (dA, dB, dxc, dxr, ds, dq, dt):
        ctx.free(x)


@pytest.mark.parametrize("rows,cols", [(0, 7), (700, 0)])
def test_empty_matrices_scale_the_outputs(ctx, rows, cols):
    n, op = (cols, Op.T) if rows == 0 else (rows, Op.N)
    y = np.arange(n, dtype=np.float32)
    dA, dx, dy = ctx.alloc(64), ctx.alloc(64), ctx.upload(y)
    ctx.gemv(op, rows, cols, 2.0, dA, max(cols, 1), dx, 0.5, dy)
    ctx.synchronize()
    np.testing.assert_array_equal(ctx.download(dy, (n,)), 0.5 * y)
    for x in (dA, dx, dy):
        ctx.free(x)
