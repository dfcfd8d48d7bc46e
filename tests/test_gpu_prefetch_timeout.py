"""The stencil passes' waits for their prefetched tiles (GPU required): bounded, and a wait that
gives up is reported as FS_ERR_TIMEOUT whether or not the handle checks for non-finite values.

The bound is one poll, which runs out before any tile can have arrived; the kernels then wait
for their copies, fill in NaN and end as usual. With the default bound back the same handle
steps like the oracle. (The solve's grid barriers have the same bound; the tiles' report comes
first.)"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,tile_rows", [(32, 0), (128, 0), (1500, 0), (300, 128)])
@pytest.mark.parametrize("check_finite", [0, 1])
def test_a_wait_that_gives_up_is_reported(fluid, wl, n, tile_rows, check_finite):
    w = wl.small_sources(n, seed=17)
    tol = 2e-2
    with fluid.Solver(w.rows, w.cols, pressure_tolerance=tol, pressure_max_iterations=20000, check_finite=check_finite,
                      tile_rows=tile_rows, sweeps_per_pass=8, device=0) as s:
        s.upload(*w.state())
        s.upload_sources(*w.sources())
        s.step(w.diffusion, w.viscosity, w.dt)  # captures the step
        s.set_barrier_poll_limit(1)
        s.upload(*w.state())
        with pytest.raises(fluid.FluidError, match="tile") as e:
            s.step(w.diffusion, w.viscosity, w.dt)
        assert e.value.code == fluid.FS_ERR_TIMEOUT
        s.sync()  # reported once
        assert not np.isfinite(s.download()[0]).all()
        s.set_barrier_poll_limit(0)
        s.upload(*w.state())
        s.step(w.diffusion, w.viscosity, w.dt)
        got = s.download()
        k1, k2 = s.stats()["pressure_iterations_last"]
    want = oracle.gpu_solve_ex(*w.state()[:1], w.ds, w.diffusion, *w.state()[1:], w.us, w.vs, w.viscosity, w.dt, 15, k1,
                               k2)
    for g, o in zip(got, want):
        assert oracle.rel_linf(g, o) <= 1e-5
