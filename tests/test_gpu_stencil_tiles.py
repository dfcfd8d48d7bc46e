"""The stencil passes at the sizes where their tiling changes (GPU required): grids just
below, at and above one region (128 columns, 64 or 128 rows) and two, every position of the
last column in its group of four, and few rows in the last warp. Projections have no
division substitute and must equal the oracle bit for bit; diffusion differs from it by at
most the last bit of a few quotients (1e-6 of the largest value)."""
import ctypes as C

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SIZES = [(3, 3), (9, 127), (17, 128), (63, 129), (64, 130), (65, 131), (66, 132), (71, 133), (72, 236), (127, 237),
         (128, 238), (129, 239), (161, 240), (113, 241), (112, 5)]


@pytest.mark.parametrize("rows,cols", SIZES)
@pytest.mark.parametrize("sweeps,tile_rows", [(8, 64), (3, 64), (29, 64), (8, 128)])
def test_tiles_match_the_oracle(fluid, wl, rows, cols, sweeps, tile_rows):
    d, u, v, ds, us, vs = wl.random_state(rows, cols, 5 * rows + cols, vmax=1.0)
    k, rate, dt = sweeps + sweeps // 2 + 1, 2e-3, 0.1  # two passes of uneven depth
    with fluid.Solver(rows, cols, diffuse_iterations=k, pressure_iterations=k, sweeps_per_pass=sweeps,
                      tile_rows=tile_rows, device=0) as s:
        s.upload(d, u, v)
        s.upload_sources(ds, us, vs)
        s.stage(fluid.STAGE_DIFFUSE_DENSITY, rate, dt)
        s.stage(fluid.STAGE_PROJECT, 0.0, dt)
        gd, gu, gv = s.download()
    wd = oracle.diffuse(oracle.add_sources(d, ds, dt), oracle.BND_CONT, rate, dt, k)
    wu, wv, _, _ = oracle.project(u, v, k)
    assert oracle.rel_linf(gd, wd) <= 1e-6
    np.testing.assert_array_equal(gu, wu)
    np.testing.assert_array_equal(gv, wv)
    assert gd[0, 0] == d[0, 0] and gd[0, -1] == d[0, -1] and gd[-1, 0] == d[-1, 0] and gd[-1, -1] == d[-1, -1]


@pytest.mark.parametrize("rows,cols,iters", [(64, 130, 20), (65, 129, 5), (17, 128, 8), (129, 131, 3)])
def test_one_pass_projection_epilogue(fluid, wl, rows, cols, iters):
    _, u, v, _, _, _ = wl.random_state(rows, cols, rows + cols, vmax=1.0)
    with fluid.Solver(rows, cols, pressure_iterations=iters, sweeps_per_pass=iters, device=0) as s:
        s.upload(np.zeros_like(u), u, v)
        s.stage(fluid.STAGE_PROJECT, 0.0, 0.1)
        _, gu, gv = s.download()
    wu, wv, _, _ = oracle.project(u, v, iters)
    np.testing.assert_array_equal(gu, wu)
    np.testing.assert_array_equal(gv, wv)


@pytest.mark.parametrize("rows,cols,pitch", [(66, 130, 132), (66, 130, 131), (70, 129, 132), (64, 128, 160)])
def test_caller_rows_keep_their_padding(fluid, wl, rows, cols, pitch):
    """fs_project_noalloc writes the caller's rows up to the last column and no further."""
    import torch

    _, u, v, _, _, _ = wl.random_state(rows, cols, rows + pitch, vmax=1.0)
    src = [torch.zeros((rows, pitch), device="cuda") for _ in range(2)]
    dst = [torch.full((rows, pitch), 7.0, device="cuda") for _ in range(2)]
    for t, x in zip(src, (u, v)):
        t[:, :cols].copy_(torch.from_numpy(x))
    torch.cuda.synchronize()
    L = fluid.load()
    assert L.fs_project_noalloc(*(C.c_void_p(t.data_ptr()) for t in src + dst), rows, cols, pitch, 12, None) == 0
    torch.cuda.synchronize()
    wu, wv, _, _ = oracle.project(u, v, 12)
    for t, w in zip(dst, (wu, wv)):
        np.testing.assert_array_equal(t[:, :cols].cpu().numpy(), w)
        assert bool((t[:, cols:] == 7.0).all())
