"""The Gauss-Seidel solves at the sizes where their form changes (GPU required): one CTA for
all bands against a CTA per band, last bands of one row and of all 32, arrays in shared and
in global memory, more sweeps than a launch has warps; and the splat of cells that receive
many sources (a thread's own list, several passes over the lists, the in-order form).
Everything must equal the host solver's restatement bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _step(fluid, n, fields, args, kd, kp, steps=1):
    d, u, v, ds, us, vs = fields
    with fluid.FluidSolverGaussSeidel(n, diffuse_iterations=kd, pressure_iterations=kp, device=0) as s:
        s.upload(d, u, v)
        s.upload_sources(ds, us, vs)
        s.step(*args, steps)
        return s.download()


@pytest.mark.parametrize("n,kd,kp", [(5, 3, 50), (34, 20, 20), (35, 60, 1), (66, 24, 25), (98, 7, 49), (130, 20, 20),
                                     (141, 20, 24), (142, 20, 24), (161, 30, 20), (162, 2, 49), (900, 3, 26)])
def test_bands(fluid, wl, n, kd, kp):
    f = wl.random_state(n, n, n + kp, vmax=0.3)
    got = _step(fluid, n, f, (0.03, 0.01, 0.1), kd, kp)
    want = oracle.cpu_solve(f[0], f[3], 0.03, f[1], f[2], f[4], f[5], 0.01, 0.1, kd=kd, kp=kp, nsteps=1)
    for g, o in zip(got, want):
        np.testing.assert_array_equal(g, o)


@pytest.mark.parametrize("radius", [3, 5, 12])
def test_splat_of_cells_with_many_sources(fluid, radius):
    """All cells within `radius` of the centre move into one cell: ~28, 80 and 450 sources."""
    n, dt = 64, 0.1
    i, j = np.mgrid[0:n, 0:n].astype(np.float32)
    dt0 = np.float32(n) * np.float32(dt)
    near = ((i - 30) ** 2 + (j - 33) ** 2 <= radius * radius).astype(np.float32)
    rng = np.random.default_rng(radius)
    u = (near * (33.4 - j) / dt0).astype(np.float32)
    v = (near * (30.6 - i) / dt0).astype(np.float32)
    d = rng.uniform(0, 1, (n, n)).astype(np.float32)
    z = np.zeros((n, n), np.float32)
    got = _step(fluid, n, (d, u, v, z, z, z), (1e-3, 1e-3, dt), 20, 20)
    want = oracle.cpu_solve(d, z, 1e-3, u, v, z, z, 1e-3, dt, kd=20, kp=20, nsteps=1)
    for g, o in zip(got, want):
        np.testing.assert_array_equal(g, o)
