"""fs_sync of a handle with nothing to report costs what its one stream synchronisation costs,
whatever the method (GPU required). A Gauss-Seidel handle's asked the device about 140 sizes at
each sync: 5.8 us against 0.9."""
import time

import pytest

pytestmark = pytest.mark.gpu


def _idle_sync_us(solver):
    with solver as s:
        s.step(1e-4, 1e-4, 0.1)
        best = float("inf")
        for _ in range(40):
            t = time.perf_counter()
            for _ in range(100):
                s.sync()
            best = min(best, (time.perf_counter() - t) / 100)
    return 1e6 * best


@pytest.mark.parametrize("n", [100, 300])
def test_idle_sync(fluid, n):
    jacobi = _idle_sync_us(fluid.Solver(n, n, device=0))
    assert _idle_sync_us(fluid.FluidSolverGaussSeidel(n, device=0)) <= 2.5 * jacobi
