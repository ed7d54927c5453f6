"""The network's kernels at channel counts beyond one dimension of a grid, against FP64.

Tolerances as in test_cnn_kernels: n 2^-24 of the sum of the products' magnitudes for a chain of n FP32 products.
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
