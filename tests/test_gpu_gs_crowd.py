"""The Gauss-Seidel splat of crowded cells, which receive more sources than a thread sorts (GPU
required): few sources in a wide flow (lists sorted by a CTA), many, or a short reach (every
source near enough looked at), cells at edges and corners, several crowds at once, all sources
in one cell, densities that are not finite. Everything must equal the host solver's restatement
bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

DT = 0.1


def _velocity(n, target_i, target_j, moves):
    """The velocity that carries the cells where `moves` to (target_i, target_j)."""
    i, j = np.mgrid[0:n, 0:n].astype(np.float32)
    dt0 = np.float32(n) * np.float32(DT)
    m = moves.astype(np.float32)
    return (m * (target_j - j) / dt0).astype(np.float32), (m * (target_i - i) / dt0).astype(np.float32)


def _check(fluid, n, d, u, v):
    z = np.zeros((n, n), np.float32)
    with fluid.FluidSolverGaussSeidel(n, diffuse_iterations=0, pressure_iterations=1, device=0) as s:
        s.upload(d, u, v)
        s.upload_sources(z, z, z)
        s.step(0.0, 0.0, DT)
        got = s.download()
    want = oracle.cpu_solve(d, z, 0.0, u, v, z, z, 0.0, DT, kd=0, kp=1, nsteps=1)
    for g, o in zip(got, want):
        np.testing.assert_array_equal(g, o)


def _density(n):
    return np.random.default_rng(n).uniform(0, 1, (n, n)).astype(np.float32)


@pytest.mark.parametrize("far", [0, 150])
@pytest.mark.parametrize("block", [5, 8, 12, 33])
def test_many_crowds(fluid, block, far):
    """Every block of cells moves to its middle; with `far`, one source moves that much, so that
    a cell's sources could be anywhere."""
    n = 200
    i, j = np.mgrid[0:n, 0:n].astype(np.float32)
    ti, tj = ((x // block) * block + np.float32(block / 2 + 0.3) for x in (i, j))
    moves = np.ones((n, n), bool)
    moves[:, 160:] = False
    u, v = _velocity(n, np.minimum(ti, n - 2), np.minimum(tj, n - 2), moves)
    if far:
        u[20, 30] = np.float32(far + 0.25) / (np.float32(n) * np.float32(DT))
    _check(fluid, n, _density(n), u, v)


@pytest.mark.parametrize("n", [8, 33, 66])
@pytest.mark.parametrize("ti,tj", [(0.6, 0.7), (0.6, 4.5), (1.2, 1.4), (-1.6, -1.7), (-2.3, 3.4), (3.2, -2.1)])
def test_at_edges_and_corners(fluid, n, ti, tj):
    u, v = _velocity(n, ti % n, tj % n, np.ones((n, n), bool))
    _check(fluid, n, _density(n), u, v)


@pytest.mark.parametrize("n", [130, 300])
def test_all_sources_in_one_cell(fluid, n):
    u, v = _velocity(n, n / 2 + 0.4, n / 3 + 0.7, np.ones((n, n), bool))
    _check(fluid, n, _density(n), u, v)


@pytest.mark.parametrize("radius", [2, 4, 9])
@pytest.mark.parametrize("value", [np.inf, np.nan, -0.0])
def test_densities_that_are_not_finite(fluid, radius, value):
    n = 64
    i, j = np.mgrid[0:n, 0:n].astype(np.float32)
    u, v = _velocity(n, 30.6, 33.4, (i - 30) ** 2 + (j - 33) ** 2 <= radius * radius)
    d = _density(n)
    d[30, 32] = value
    _check(fluid, n, d, u, v)
