"""Advection by columns of four rows per thread (large grids, and every grid of a batch):
the splat sums what neighbouring cells add to one target before its atomics, and the finish
takes four cells of a row at a time. Sizes at the edges of a warp's 32 columns, of four
rows and of a block's 32, and the smallest grid that takes four rows by itself.

Tolerance. A target receives n values and the order of their sum is free: two orders of an
n-term FP32 sum differ by at most 2 (n - 1) 2^-24 times the sum of the values' magnitudes.
Densities are non-negative, so that is relative to the sum itself. The flows below compress
by less than a factor of two a side: at most 9 source cells reach a target's four cells,
n <= 9, giving 1e-6; the smoothing adds five roundings of 2^-24 (3e-7). The backtrace has no
free order and is compared bit for bit.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

TOL = 1.3e-6


def flow(rows, cols, kind, dt):
    """Density and a velocity whose displacement is a few cells: "smooth" (neighbours land
    next to each other), "rough" (up to 0.45 cells apart in any direction), "shift" (a
    uniform one that carries a whole border out of the grid)."""
    rng = np.random.default_rng(rows * 131 + cols)
    cells = 1.0 / (np.sqrt(np.float64(rows) * cols) * dt)  # velocity of one cell per step
    y, x = np.mgrid[0:rows, 0:cols].astype(np.float64)
    d = rng.random((rows, cols)).astype(np.float32)
    if kind == "smooth":
        u, v = 2.3 * np.sin(0.05 * y), 1.7 * np.cos(0.05 * x)
    elif kind == "rough":
        u, v = rng.uniform(-0.45, 0.45, (2, rows, cols))
    else:
        u, v = np.full((rows, cols), 3.25), np.full((rows, cols), -2.5)
    return d, (u * cells).astype(np.float32), (v * cells).astype(np.float32)


@pytest.mark.parametrize("kind", ["smooth", "rough", "shift"])
@pytest.mark.parametrize("rows,cols", [(1449, 1449), (1030, 2045)])
def test_large_grid(fluid, rows, cols, kind):
    dt = 0.05
    d, u, v = flow(rows, cols, kind, dt)
    with fluid.Solver(rows, cols, device=0) as s:
        s.upload(d, u, v)
        s.stage(fluid.STAGE_ADVECT_DENSITY, 0.0, dt)
        gd, _, _ = s.download()
        s.upload(d, u, v)
        s.stage(fluid.STAGE_ADVECT_VELOCITY, 0.0, dt)
        _, gu, gv = s.download()
    want = oracle.smooth(oracle.advect_trace(d, u, v, dt))
    assert oracle.rel_linf(gd, want, skip_corners=False) <= TOL
    wu, wv = oracle.advect_velocity(u, v, dt)
    np.testing.assert_array_equal(gu, wu)
    np.testing.assert_array_equal(gv, wv)


@pytest.mark.parametrize("kind", ["smooth", "rough", "shift"])
def test_batch(fluid, kind):
    """A batch's step with no diffusion and no projection: one advection of each field."""
    shapes = [(3, 3), (4, 31), (5, 32), (6, 33), (31, 34), (32, 35), (33, 64), (34, 65), (37, 129), (65, 130)]
    dt = 0.05
    states = [flow(r, c, kind, dt) for r, c in shapes]
    with fluid.Batch(shapes, diffuse_iterations=0, pressure_iterations=0, device=0) as b:
        for k, state in enumerate(states):
            b.upload(k, *state)
        b.step(0.0, 0.0, dt, 1)
        got = [b.download(k) for k in range(len(shapes))]
    for shape, (d, u, v), (gd, gu, gv) in zip(shapes, states, got):
        z = np.zeros(shape, np.float32)
        od, ou, ov = oracle.gpu_solve(d, z, 0.0, u, v, z, z, 0.0, dt, kd=0, kp=0)
        assert oracle.rel_linf(gd, od) <= TOL, shape
        assert oracle.rel_linf(gu, ou) <= 1e-6 and oracle.rel_linf(gv, ov) <= 1e-6, shape
