"""Residual-driven pressure solves that run two passes as one (small and middle grids) or not:
a solve stopped after k sweeps equals a solve of k fixed sweeps bit for bit, and it stops where
a solve of single passes stops. Grids of one to all 64-row regions an SM each, of 128-row ones,
and beyond; caps of an even and an odd number of passes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(fluid, w, **cfg):
    with fluid.Solver(w.rows, w.cols, diffuse_iterations=8, device=0, **cfg) as s:
        s.upload(*w.state())
        s.upload_sources(*w.sources())
        try:
            s.step(w.diffusion, w.viscosity, w.dt)
        except fluid.FluidError as e:
            if e.code != fluid.FS_ERR_NOT_CONVERGED:
                raise
        return s.download(), s.stats()


@pytest.mark.parametrize("n,sweeps", [(33, 8), (128, 8), (128, 3), (512, 8), (512, 14), (768, 8), (1000, 8), (1024, 8),
                                      (1300, 8)])
@pytest.mark.parametrize("passes", [1, 2, 5, 8])
def test_stopped_solve_is_the_fixed_solve(fluid, wl, n, sweeps, passes):
    w = wl.small_sources(n, seed=n + sweeps)
    got, st = run(fluid, w, pressure_tolerance=1e-30, pressure_max_iterations=sweeps * passes, sweeps_per_pass=sweeps)
    assert tuple(st["pressure_iterations_last"]) == (sweeps * passes,) * 2
    want, _ = run(fluid, w, pressure_iterations=sweeps * passes, sweeps_per_pass=sweeps)
    for g, o in zip(got[1:], want[1:]):
        np.testing.assert_array_equal(g, o)


@pytest.mark.parametrize("n", [128, 512, 1024])
def test_stops_after_every_second_pass(fluid, wl, n):
    """The target is tested after passes 2, 4, ...: with a target between two of those
    residuals the solve stops at the second one."""
    w = wl.small_sources(n, seed=n)
    res = []
    for passes in (2, 4, 6):
        _, st = run(fluid, w, pressure_tolerance=1e-30, pressure_max_iterations=8 * passes, sweeps_per_pass=8)
        res.append(st["pressure_residual_last"][0])
    assert res[0] > res[1] > res[2]
    tol = float(np.sqrt(res[1] * res[2]))
    _, st = run(fluid, w, pressure_tolerance=tol, pressure_max_iterations=400, sweeps_per_pass=8)
    assert st["pressure_iterations_last"][0] == 48
