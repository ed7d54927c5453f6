"""The weight gradient's chunks (csrc/warmstart_cnn.cu): several images in one, a last chunk of a few images, strips of an
image with widths that do and do not divide 256, images too wide for a chunk. Reference and tolerance as in
test_cnn_kernels."""
import pytest

from test_cnn_kernels import test_gradients as check_gradients

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [
    (60, 4, 8, 8, 8),       # 51 images a chunk, then 9
    (7, 3, 5, 17, 15),      # whole images, an odd width
    (2, 2, 3, 100, 128),    # strips of whole rows
    (1, 3, 4, 100, 129),    # strips that begin within a row
    (1, 2, 20, 3, 1270),    # a strip of less than a row
    (2, 2, 3, 2, 1400),     # too wide
    (1, 150, 9, 70, 72),    # one output channel, groups of two: an odd number of channels
    (16, 16, 16, 64, 64)])
def test_chunks(shape):
    check_gradients(shape)


def test_masked_infinities():
    """A pixel whose gradient is 0 adds nothing, also where the input is infinite, and a tap outside the image is left out,
    also of an infinite gradient."""
    import numpy as np
    from test_cnn_kernels import _case
    for shape in ((2, 3, 5, 16, 16), (2, 2, 3, 64, 64), (1, 2, 3, 20, 19), (1, 1, 2, 3, 1400)):
        torch, L, x, w, b, skip, gy, put = _case(shape)
        B, Ci, Co, H, W = shape
        x[0, 0, 1, 1] = float("inf")
        gy[0, :, 0:3, 0:3] = 0.0
        gy[0, 1, 1, W - 1] = float("inf")  # at the right edge: taps 2, 5 and 8 lie outside
        dw, db = torch.empty(Co, Ci, 3, 3, device="cuda"), torch.empty(Co, device="cuda")
        sc = torch.empty(1 << 20, device="cuda")
        assert L.gpair_cnn_conv3x3_bwd_weight(x.data_ptr(), gy.data_ptr(), dw.data_ptr(), db.data_ptr(), sc.data_ptr(),
                                              1 << 20, B, Ci, Co, H, W, None) == 0
        torch.cuda.synchronize()
        got = np.isfinite(dw.cpu().numpy())
        want = np.ones((Co, Ci, 3, 3), bool)
        want[1] = False
        want[1, :, :, 2] = True
        assert np.array_equal(got, want)
        assert np.array_equal(np.isfinite(db.cpu().numpy()), np.arange(Co) != 1)
