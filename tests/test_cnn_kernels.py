"""The warm-start network's convolution kernels against FP64 convolutions, through the C ABI.

Tolerance, elementwise: a chain of n FP32 fused multiply-adds is within n 2^-24 of the sum of its
products' magnitudes (first order), so |error| <= (n + 4) 2^-24 (sum |a b| + |bias| + |skip|)."""
import numpy as np
import pytest

import gpair_b200 as g
from gpair_b200 import warmstart

pytestmark = pytest.mark.gpu

# (B, Cin, Cout, H, W): every tile configuration, widths that are no multiple of 4 or of a tile,
# channels that fill no block, one pixel, and many images
SHAPES = [(1, 1, 1, 1, 1), (2, 3, 5, 7, 9), (1, 4, 16, 33, 34), (3, 16, 24, 8, 8), (1, 40, 17, 12, 20),
          (40, 8, 33, 16, 32), (2, 9, 16, 65, 70), (1, 128, 130, 9, 16), (20, 16, 16, 40, 48)]


def _torch():
    import torch
    warmstart._declare(g.lib())
    return torch, g.lib()


def _case(shape, offset=0):
    torch, L = _torch()
    B, Ci, Co, H, W = shape
    gen = torch.Generator().manual_seed(B * 1000 + Ci)
    r = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731

    def put(t):  # on the device at a float offset from an aligned address
        buf = torch.zeros(t.numel() + offset, device="cuda")
        buf[offset:] = t.reshape(-1).cuda()
        return buf[offset:].view(t.shape)

    x, w, b = put(r(B, Ci, H, W)), r(Co, Ci, 3, 3).to(torch.bfloat16).cuda(), put(r(Co))
    skip, gy = put(r(B, Co, H, W)), put(r(B, Co, H, W))
    return torch, L, x, w, b, skip, gy, put


def _close(got, ref, mag, n):
    assert (got.double() - ref).abs().max().item() >= 0  # finite
    assert bool(((got.double() - ref).abs() <= (n + 4) * 2.0 ** -24 * mag).all())


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("shape", SHAPES)
def test_forward(shape, offset):
    torch, L, x, w, b, skip, gy, put = _case(shape, offset)
    B, Ci, Co, H, W = shape
    conv = torch.nn.functional.conv2d
    lin = conv(x.double(), w.double(), padding=1)
    mag = conv(x.double().abs(), w.double().abs(), padding=1) + b.double().abs().view(1, -1, 1, 1) + skip.double().abs()
    for use_skip, relu in ((0, 0), (1, 1)):
        y = put(torch.full((B, Co, H, W), float("nan")))
        assert L.gpair_cnn_conv3x3(x.data_ptr(), w.data_ptr(), b.data_ptr(), skip.data_ptr() if use_skip else None,
                                   y.data_ptr(), B, Ci, Co, H, W, relu, None) == 0
        torch.cuda.synchronize()
        ref = lin + b.double().view(1, -1, 1, 1) + (skip.double() if use_skip else 0)
        _close(y, ref.clamp(min=0) if relu else ref, mag, 9 * Ci)


@pytest.mark.parametrize("shape", SHAPES)
def test_gradients(shape):
    torch, L, x, w, b, skip, gy, put = _case(shape)
    B, Ci, Co, H, W = shape
    conv_t = torch.nn.functional.conv_transpose2d
    ref, mag = conv_t(gy.double(), w.double(), padding=1), conv_t(gy.double().abs(), w.double().abs(), padding=1)
    first = torch.randn(B, Ci, H, W, device="cuda")
    for accumulate in (0, 1):
        gx = first.clone()
        assert L.gpair_cnn_conv3x3_bwd_data(gy.data_ptr(), w.data_ptr(), gx.data_ptr(), B, Ci, Co, H, W, accumulate,
                                            None) == 0
        torch.cuda.synchronize()
        f = first.double() if accumulate else torch.zeros_like(ref)
        _close(gx, ref + f, mag + f.abs(), 9 * Co)
    unfold = lambda t: torch.nn.functional.unfold(t, 3, padding=1)  # noqa: E731
    cols, gf = unfold(x.double()), gy.double().reshape(B, Co, -1)
    dw, mw = torch.einsum("bop,bkp->ok", gf, cols), torch.einsum("bop,bkp->ok", gf.abs(), cols.abs())
    for floats in (1 << 22, -(-B // max(1, min(B, 65536 // (H * W)))) * (Co * Ci * 9 + Co)):  # ample, the least accepted
        scratch = torch.full((floats,), float("nan"), device="cuda")
        gw, gb = torch.empty(Co * Ci * 9, device="cuda"), torch.empty(Co, device="cuda")
        args = (x.data_ptr(), gy.data_ptr(), gw.data_ptr(), gb.data_ptr(), scratch.data_ptr())
        assert L.gpair_cnn_conv3x3_bwd_weight(*args, floats, B, Ci, Co, H, W, None) == 0
        torch.cuda.synchronize()
        _close(gw.view(Co, Ci * 9), dw, mw, B * H * W)
        _close(gb, gf.sum((0, 2)), gf.abs().sum((0, 2)), B * H * W)
        assert L.gpair_cnn_conv3x3_bwd_weight(*args, Co * Ci * 9 + Co - 1, B, Ci, Co, H, W, None) != 0
