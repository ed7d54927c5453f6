"""The network's kernels at channel counts beyond one pass or one dimension of a grid, against FP64.

Tolerances as in test_cnn_kernels: n 2^-24 of the sum of the products' magnitudes for a chain of n FP32 products; for the head, whose sums
are FP64, a few roundings (64 x 2^-24) of each term's magnitude.
"""
import pytest

from test_cnn_kernels import _torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ci,Co", [(70000, 2), (65536, 5), (3, 70000)])
def test_weight_gradient_of_many_channels(Ci, Co):
    torch, L = _torch()
    gen = torch.Generator().manual_seed(Ci)
    x, gy = torch.randn(1, Ci, 2, 2, generator=gen).cuda(), torch.randn(1, Co, 2, 2, generator=gen).cuda()
    n = Co * Ci * 9 + Co
    dw, db, sc = torch.full((Co, Ci, 3, 3), float("nan"), device="cuda"), torch.empty(Co, device="cuda"), torch.empty(n, device="cuda")
    assert L.gpair_cnn_conv3x3_bwd_weight(x.data_ptr(), gy.data_ptr(), dw.data_ptr(), db.data_ptr(), sc.data_ptr(), n, 1, Ci, Co, 2, 2,
                                          None) == 0
    torch.cuda.synchronize()
    pad = torch.nn.functional.pad(x.double(), (1, 1, 1, 1))
    for ky in range(3):
        for kx in range(3):
            part = pad[0, :, ky:ky + 2, kx:kx + 2].reshape(Ci, 4)
            ref, mag = gy.double().reshape(Co, 4) @ part.T, gy.double().abs().reshape(Co, 4) @ part.abs().T
            assert bool(((dw[:, :, ky, kx].double() - ref).abs() <= 8 * 2.0 ** -24 * mag).all())
    assert torch.allclose(db.double(), gy.double().sum(dim=(0, 2, 3)), rtol=0, atol=1e-5)


@pytest.mark.parametrize("B,C,HW", [(1, 1, 1), (2, 15, 9), (3, 16, 64), (2, 17, 65), (1, 33, 300), (2, 40, 4097), (1, 300, 50)])
def test_head_and_its_backward(B, C, HW):
    """Channels in passes of 16: none, one and several full passes, remainders, and more gradients than threads in a block."""
    torch, L = _torch()
    gen = torch.Generator().manual_seed(100 * C + HW)
    d, w, bias = torch.randn(B, C, HW, generator=gen).cuda(), torch.randn(C, generator=gen).cuda() / C ** 0.5, torch.randn(1, generator=gen).cuda()
    gout = torch.randn(B, HW, generator=gen).cuda()
    nan = float("nan")
    z, out = torch.full((B, HW), nan, device="cuda"), torch.full((B, HW), nan, device="cuda")
    asum, gd, dw = torch.full((B,), nan, device="cuda"), torch.full((B, C, HW), nan, device="cuda"), torch.full((C + 1,), nan, device="cuda")
    sc = torch.empty(B * (C + 1), device="cuda")
    assert L.gpair_cnn_head(d.data_ptr(), w.data_ptr(), bias.data_ptr(), z.data_ptr(), out.data_ptr(), asum.data_ptr(), B, C, HW, None) == 0
    assert L.gpair_cnn_head_bwd(d.data_ptr(), w.data_ptr(), z.data_ptr(), out.data_ptr(), asum.data_ptr(), gout.data_ptr(), gd.data_ptr(),
                                dw.data_ptr(), sc.data_ptr(), B, C, HW, None) == 0
    torch.cuda.synchronize()
    e = 2.0 ** -24
    zr = torch.einsum("bcp,c->bp", d.double(), w.double()) + bias.double()
    zm = torch.einsum("bcp,c->bp", d.double().abs(), w.double().abs()) + bias.double().abs()
    assert bool(((z.double() - zr).abs() <= (C + 4) * e * zm).all())
    # from the kernel's own z on, so that one bound holds for each step
    a = torch.nn.functional.softplus(z.double(), threshold=40.0)
    S = a.sum(1, keepdim=True)
    assert torch.allclose(asum.double(), S[:, 0], rtol=64 * e, atol=0)
    assert torch.allclose(out.double(), a / S, rtol=64 * e, atol=1e-30)
    dot = (gout.double() * out.double()).sum(1, keepdim=True)
    gz = (gout.double() - dot) / S * torch.sigmoid(z.double())
    gzm = (gout.double().abs() + dot.abs()) / S  # what its difference is rounded against
    wd = w.double().abs().view(1, C, 1)
    assert bool(((gd.double() - w.double().view(1, C, 1) * gz[:, None]).abs() <= 64 * e * wd * gzm[:, None]).all())
    ref = torch.cat([torch.einsum("bp,bcp->c", gz, d.double()), gz.sum().view(1)])
    mag = torch.cat([torch.einsum("bp,bcp->c", gzm, d.double().abs()), gzm.sum().view(1)])
    assert bool(((dw.double() - ref).abs() <= (64 + B) * e * mag).all())
