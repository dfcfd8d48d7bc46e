"""The tensor-core weight gradient with activations or gradients that are not finite (GPU
required): which of its entries are infinite or NaN is what the CUDA-core kernel says, and the
others are right. A pixel of an image's first or last column must not reach the taps of the
columns that do not exist.

Tolerance as for finite values: two FP32 sums of the same n products differ by at most
2 n 2^-24 times the sum of the products' magnitudes."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


@pytest.mark.parametrize("imgs,img_h,W,up", [(1, 8, 8, 0), (3, 1, 1, 0), (2, 4, 126, 0), (1, 5, 129, 0), (3, 6, 14, 1),
                                             (1, 300, 257, 0)])
@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan")])
@pytest.mark.parametrize("where", ["x", "dz"])
def test_entries_that_are_not_finite(fluid, imgs, img_h, W, up, value, where):
    import torch

    L = fluid.load()
    rng = np.random.default_rng(imgs + 10 * img_h + 100 * W)
    H = imgs * img_h
    bf = lambda *s: torch.from_numpy(rng.uniform(0.5, 1.5, s).astype(np.float32)).to(torch.bfloat16).cuda()
    x, dz = bf(H >> up, W >> up, 32), bf(H, W, 32)
    t = x if where == "x" else dz
    rows, cols = t.shape[:2]
    # the first column, the last one, and an inner pixel, in a channel each
    for ch, (i, j) in enumerate([(rows // 2, 0), (rows - 1, cols - 1), (0, cols // 2)]):
        t[i, j, 5 + 7 * ch] = value
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    work = torch.empty(int(L.fs_net_weight_grad_tc_work_floats(H, W)), dtype=torch.float32, device="cuda")
    g, want, size = (torch.zeros(9248, dtype=torch.float32, device="cuda") for _ in range(3))
    assert L.fs_net_weight_grad_tc(_ptr(dz), _ptr(x), _ptr(g), _ptr(g[9216:]), _ptr(work), work.numel(), H, W, img_h,
                                   up, _ptr(err), None) == 0
    assert L.fs_net_weight_grad(_ptr(dz.float()), _ptr(x), _ptr(want), _ptr(want[9216:]), H, W, img_h, up, None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert torch.equal(torch.isnan(g), torch.isnan(want))
    inf = torch.isinf(want)
    assert torch.equal(torch.isinf(g), inf) and torch.equal(g[inf], want[inf])
    ok = torch.isfinite(want)
    # all values are between 0.5 and 1.5, so the finite sums are their own magnitudes
    assert bool(((g - want).abs()[ok] <= 2 * H * W * 2.0 ** -24 * want[ok]).all())
