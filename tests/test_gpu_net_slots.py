"""The network's tensor-core convolution and weight gradient in border-column slots, at the
sizes where slots, tiles of 128 and images end in different places, and the fused launches
of the training step against the launches they stand for.

Tolerance: two FP32 sums of the same n products differ by at most 2 n 2^-24 times the sum of
the products' magnitudes, which the CUDA-core kernels give for the absolute values. The
fused launches do the same operations on the same values and are compared bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24
# images, rows per image, columns, upsampled input
SHAPES = [(1, 1, 1, 0), (1, 3, 1, 0), (5, 2, 2, 1), (3, 1, 125, 0), (2, 2, 126, 0), (1, 2, 127, 0), (3, 1, 128, 0),
          (1, 5, 129, 0), (2, 4, 254, 1), (1, 1, 300, 0), (9, 6, 14, 1)]


def _ptr(t):
    import ctypes

    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _bf(rng, *shape):
    import torch

    return torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).to(torch.bfloat16).cuda()


def _pack(L, w):
    import torch

    wpk = torch.empty(32 * 288, dtype=torch.bfloat16, device="cuda")
    assert L.fs_conv_pack_weights(_ptr(w), _ptr(wpk), None) == 0
    return wpk


@pytest.mark.parametrize("imgs,img_h,W,up", SHAPES)
def test_convolution_and_weight_gradient(fluid, imgs, img_h, W, up):
    import torch

    L = fluid.load()
    rng = np.random.default_rng(imgs + 10 * img_h + 100 * W)
    H = imgs * img_h
    x = _bf(rng, H >> up, W >> up, 32)
    w = _bf(rng, 32, 9, 32).float()
    dzb = _bf(rng, H, W, 32)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def conv(xx, ww, tc):
        y = torch.full((H, W, 32), np.nan, dtype=torch.float32, device="cuda")
        assert L.fs_conv3x3(_ptr(xx), _ptr(_pack(L, ww)), _ptr(ww), None, None, None, _ptr(y), H, W, img_h, up, 0, tc,
                            _ptr(err), None) == 0
        return y

    size = conv(x.abs(), w.abs(), 0)
    assert bool(((conv(x, w, 1) - conv(x, w, 0)).abs() <= 2 * 288 * EPS * size).all())

    def wgrad_ref(xx, dz):
        g = torch.zeros(9248, dtype=torch.float32, device="cuda")
        assert L.fs_net_weight_grad(_ptr(dz), _ptr(xx), _ptr(g), _ptr(g[9216:]), H, W, img_h, up, None) == 0
        return g

    work = torch.empty(int(L.fs_net_weight_grad_tc_work_floats(H, W)), dtype=torch.float32, device="cuda")
    g = torch.zeros(9248, dtype=torch.float32, device="cuda")
    assert L.fs_net_weight_grad_tc(_ptr(dzb), _ptr(x), _ptr(g), _ptr(g[9216:]), _ptr(work), work.numel(), H, W, img_h,
                                   up, _ptr(err), None) == 0
    size = wgrad_ref(x.abs(), dzb.float().abs())
    assert bool(((g - wgrad_ref(x, dzb.float())).abs() <= 2 * H * W * EPS * size).all())
    assert int(err.item()) == 0


def test_packed_layers(fluid):
    import torch

    L = fluid.load()
    rng = np.random.default_rng(3)
    layers, stride = 3, 9248
    params = torch.from_numpy(rng.standard_normal(layers * stride).astype(np.float32)).cuda()
    wpk = torch.empty((layers, 9216), dtype=torch.bfloat16, device="cuda")
    wflip = torch.empty((layers, 9216), dtype=torch.float32, device="cuda")
    wflip_pk = torch.empty_like(wpk)
    assert L.fs_net_pack_layers(_ptr(params), layers, stride, _ptr(wpk), _ptr(wflip), _ptr(wflip_pk), None) == 0
    for li in range(layers):
        w = params[li * stride:li * stride + 9216]
        f = torch.empty(9216, dtype=torch.float32, device="cuda")
        assert L.fs_net_flip_weights(_ptr(w), _ptr(f), None) == 0
        assert torch.equal(wflip[li], f)
        assert torch.equal(wpk[li], _pack(L, w)) and torch.equal(wflip_pk[li], _pack(L, f))
    assert L.fs_net_pack_layers(_ptr(params), 0, stride, _ptr(wpk), _ptr(wflip), _ptr(wflip_pk), None) != 0


@pytest.mark.parametrize("rows,w", [(2, 2), (6, 10), (64, 34)])
@pytest.mark.parametrize("skip", [0, 1])
def test_fused_relu_backward(fluid, rows, w, skip):
    import torch

    L = fluid.load()
    rng = np.random.default_rng(rows + w)
    f32 = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32)).cuda()
    act = torch.relu(_bf(rng, rows, w, 32))
    da2 = f32(rows, w, 32) if skip else None
    n = rows * w * 32

    def two_steps(da):
        dz, dzb = torch.empty_like(da), torch.empty_like(act)
        assert L.fs_net_relu_bwd(_ptr(da), _ptr(da2), _ptr(act), _ptr(dz), _ptr(dzb), n, 1, None) == 0
        return dz, dzb

    da = {0: f32(rows, w, 32), 1: f32(rows // 2, w // 2, 32), 2: f32(2 * rows, 2 * w, 32)}
    full = {0: da[0], 1: torch.empty((rows, w, 32), device="cuda"), 2: torch.empty((rows, w, 32), device="cuda")}
    assert L.fs_net_avgpool2_bwd(_ptr(da[1]), _ptr(full[1]), rows, w, None) == 0
    assert L.fs_net_upsample2_bwd(_ptr(da[2]), _ptr(full[2]), rows, w, None) == 0
    for src in (0, 1, 2):
        dz, dzb = torch.empty((rows, w, 32), device="cuda"), torch.empty_like(act)
        want, wantb = two_steps(full[src])
        assert L.fs_net_relu_bwd_from(_ptr(da[src]), src, _ptr(da2), _ptr(act), _ptr(dz), _ptr(dzb), rows, w, 1,
                                      None) == 0
        assert torch.equal(dz, want) and torch.equal(dzb, wantb)
    # the convolution's epilogue
    dzb, wt = _bf(rng, rows, w, 32), _bf(rng, 32, 9, 32).float()
    wpk = _pack(L, wt)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    da = torch.empty((rows, w, 32), device="cuda")
    assert L.fs_conv3x3(_ptr(dzb), _ptr(wpk), _ptr(wt), None, None, None, _ptr(da), rows, w, rows, 0, 0, 1, _ptr(err),
                        None) == 0
    da2 = None
    want, wantb = two_steps(da)
    dz, got = torch.empty_like(da), torch.empty_like(act)
    assert L.fs_conv3x3_relu_bwd(_ptr(dzb), _ptr(wpk), _ptr(act), _ptr(got), _ptr(dz), rows, w, rows, _ptr(err), None) == 0
    assert torch.equal(dz, want) and torch.equal(got, wantb) and int(err.item()) == 0
