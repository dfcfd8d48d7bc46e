"""The host call on grids below the overlapped form's size moves its nine grids by kernels over
the link: the same step as upload, step, download, at row lengths and base addresses of every
alignment, and nothing outside the caller's grids is written.

The velocity has no free order and is compared bit for bit; the density's splat adds with
atomics in any order (n values to a target, n <= 9 in this flow: 2 (n - 1) 2^-24 = 1e-6)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def placed(a, offset):
    """A copy of a whose first element lies `offset` floats past a 64-byte boundary, with
    sentinels around it; returns the view and the whole buffer."""
    n = a.size
    buf = np.full(n + 64, np.float32(-77.0))
    start = (-buf.ctypes.data // 4) % 16 + 16 + offset
    v = buf[start:start + n].reshape(a.shape)
    v[:] = a
    return v, buf, start


@pytest.mark.parametrize("offset", [0, 1, 2])
@pytest.mark.parametrize("rows,cols", [(3, 3), (5, 7), (33, 31), (130, 130), (67, 129), (70, 1021), (41, 254)])
def test_host_call_is_upload_step_download(fluid, wl, rows, cols, offset):
    d, u, v, ds, us, vs = wl.random_state(rows, cols, rows, vmax=0.02)
    diff, visc, dt = 1e-3, 1e-3, 0.05
    with fluid.Solver(rows, cols, device=0) as s:
        s.upload(d, u, v)
        s.upload_sources(ds, us, vs)
        s.step(diff, visc, dt)
        want = s.download()
    grids = [placed(g, offset if k % 2 == 0 else 0) for k, g in enumerate((d, u, v, ds, us, vs))]
    a = [g[0] for g in grids]
    with fluid.Solver(rows, cols, device=0) as s:
        s.solve(a[0], a[3], diff, a[1], a[2], a[4], a[5], visc, dt)
    np.testing.assert_array_equal(a[1], want[1])
    np.testing.assert_array_equal(a[2], want[2])
    assert oracle.rel_linf(a[0], want[0], skip_corners=False) <= 1e-6
    for g, src in zip(a[3:], (ds, us, vs)):
        np.testing.assert_array_equal(g, src)
    for view, buf, start in grids:
        assert (buf[:start] == -77.0).all() and (buf[start + view.size:] == -77.0).all()
