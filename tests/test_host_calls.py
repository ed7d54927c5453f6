"""Host side of the blocking calls: staged copies, results written by the kernels, batch parameters in one launch.

No tolerances: copies return the same bytes, and a run in a batch of one kind repeats itself bit for bit.
"""
import numpy as np
import pytest

import gpair_b200 as g
from gpair_b200 import api
from test_uvgrid import _image, _problem

pytestmark = pytest.mark.gpu


def _small(N, seed, precision):
    rng = np.random.default_rng(seed)
    r = g.Reconstructor(0)
    r.set_problem(_problem(N, rng.uniform(-0.2, 0.2, (40, 2)), 20, seed))
    r.set_precision(precision)
    return r


@pytest.mark.parametrize("N", [8, 255, 256, 257])  # around the size that is staged (256 x 256)
def test_copies(N):
    r = _small(N, 1, g.PREC_FP32)
    rng = np.random.default_rng(2)
    buf = np.empty(N * N, np.float32)
    for i in range(6):  # the caller's array is its own again once the call returns
        buf[:] = rng.uniform(1, 2, N * N)
        want = buf.copy()
        r.set_image(buf)
        r.set_image(buf[::-1].copy(), g.IMG_TEMP)
        buf[:] = -1
        assert np.array_equal(r.get_image(), want)
        assert np.array_equal(r.get_image(g.IMG_TEMP), want[::-1])
    r.close()


@pytest.mark.parametrize("precision", [g.PREC_FP32, g.PREC_SPLIT16])
@pytest.mark.parametrize("N", [33, 160])
def test_results_follow_their_own_evaluation(N, precision):
    r = _small(N, 3, precision)
    img = _image(N, 4)
    r.set_image(img)
    want = r.criterion()
    r.gradient()
    grad = r.full_gradient()
    bad = img.copy()
    bad[N + 3] = np.nan
    r.set_image(bad)
    with pytest.raises(g.GpairError):
        r.criterion()
    r.set_image(img)  # the flag of the last evaluation does not stay
    assert r.criterion() == want
    r.gradient()
    assert np.array_equal(r.full_gradient(), grad)
    first = r.update_pixel(2, 1, float(img[2 + N]))  # no change of the image: rounding of V alone
    again = r.update_pixel(2, 1, float(img[2 + N]))
    assert np.isfinite(first).all() and np.isfinite(again).all()
    r.close()


def test_batch_takes_queued_images_and_new_parameters():
    recs = [_small(N, 5 + N, g.PREC_SPLIT16) for N in (48, 64, 130)]
    imgs = [_image(r.problem.width, 6) for r in recs]

    def go(b, iterations):
        for r, im in zip(recs, imgs):
            r.set_image(im)  # still in flight when the run starts
        out = b.run(iterations)
        return [(o["J"], o["chi2"], o["criterion_evals"], o["iterations"]) for o in out], \
            [r.get_image() for r in recs]

    for r, im in zip(recs, imgs):
        r.set_image(im)
    b = api.Batch(recs, line_search=g.LS_BATCH)
    one = go(b, 1)
    three = go(b, 3)
    again = go(b, 3)
    assert [o[3] for o in one[0]] == [1] * 3 and all(b[2] > a[2] for a, b in zip(one[0], three[0]))
    assert three[0] == again[0] and all(np.array_equal(x, y) for x, y in zip(three[1], again[1]))
    b.close()
    for r in recs:
        r.close()
