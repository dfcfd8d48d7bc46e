"""Host grids wherever a caller may hold them (GPU required): at addresses that are no multiple
of four bytes (a packed record, a byte buffer), at any multiple of four, page-locked. The host
call and a batch's downloads give what they give for ordinary arrays, and write nothing else.

The velocity has no free order and is compared bit for bit; the density's splat adds with
atomics in any order (n values to a target, n <= 9 in this flow: 2 (n - 1) 2^-24 = 1e-6)."""
import ctypes as C

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

MARK = 0xA5


def placed(shape, offset, values=None):
    """A float32 view that begins `offset` bytes past a 64-byte boundary of a buffer of MARK
    bytes; returns the view, the buffer and the view's place in it."""
    n = 4 * shape[0] * shape[1]
    buf = np.full(n + 192, MARK, np.uint8)
    start = -buf.ctypes.data % 64 + 64 + offset
    view = buf[start:start + n].view(np.float32).reshape(shape)
    if values is not None:
        view[:] = values
    return view, buf, (start, start + n)


def untouched(buf, place):
    return (buf[:place[0]] == MARK).all() and (buf[place[1]:] == MARK).all()


@pytest.mark.parametrize("offset", [1, 2, 6])
@pytest.mark.parametrize("rows,cols", [(3, 3), (34, 37), (130, 130)])
def test_host_call_on_grids_off_the_float_grid(fluid, wl, rows, cols, offset):
    fields = wl.random_state(rows, cols, rows, vmax=0.02)
    diff, visc, dt = 1e-3, 1e-3, 0.05
    a = [f.copy() for f in fields]
    with fluid.Solver(rows, cols, device=0) as s:
        s.solve(a[0], a[3], diff, a[1], a[2], a[4], a[5], visc, dt)
    for moved in (range(6), [0], [4]):  # all six grids, one that is written, one that is read
        g = [placed((rows, cols), offset if k in moved else 0, f) for k, f in enumerate(fields)]
        b = [x[0] for x in g]
        with fluid.Solver(rows, cols, device=0) as s:
            s.solve(b[0], b[3], diff, b[1], b[2], b[4], b[5], visc, dt)
        np.testing.assert_array_equal(b[1], a[1])
        np.testing.assert_array_equal(b[2], a[2])
        assert oracle.rel_linf(b[0], a[0], skip_corners=False) <= 1e-6
        for k in (3, 4, 5):
            np.testing.assert_array_equal(b[k], fields[k])
        assert all(untouched(buf, place) for _v, buf, place in g)


@pytest.mark.parametrize("offset", [0, 1, 4, 7, 8])
def test_batch_download_to_any_address(fluid, wl, offset):
    shapes = [(3, 3), (41, 254), (130, 67)]
    L = fluid.load()
    with fluid.Batch(shapes, device=0) as b:
        fields = [wl.random_state(r, c, r, vmax=0.02)[:3] for r, c in shapes]
        for k, f in enumerate(fields):
            b.upload(k, *f)
        for k, f in enumerate(fields):
            for moved in ((0, 1, 2), (1,)):
                g = [placed(shapes[k], offset if i in moved else 0) for i in range(3)]
                assert L.fs_batch_download(b._h, k, *(C.c_void_p(x[0].ctypes.data) for x in g)) == 0
                # pageable memory is complete on return
                for (view, buf, place), want in zip(g, f):
                    np.testing.assert_array_equal(view, want)
                    assert untouched(buf, place)


def test_batch_download_to_page_locked_memory(fluid, wl):
    shapes = [(41, 254), (130, 67)]
    L = fluid.load()
    with fluid.Batch(shapes, device=0) as b:
        fields = [wl.random_state(r, c, r, vmax=0.02)[:3] for r, c in shapes]
        pinned = [[fluid.PinnedArray(r, c) for _ in range(3)] for r, c in shapes]
        for k, f in enumerate(fields):
            b.upload(k, *f)
        for k, p in enumerate(pinned):
            assert L.fs_batch_download(b._h, k, *(C.c_void_p(x.array.ctypes.data) for x in p)) == 0
        assert L.fs_batch_sync(b._h) == 0
        for f, p in zip(fields, pinned):
            for x, want in zip(p, f):
                np.testing.assert_array_equal(x.array, want)
