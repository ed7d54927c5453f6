"""The CUDA-core path's contractions (csrc/kernels_core.cu) at the edges of their tiles: 64 or 32 pixels, 32 or 16 uv
points, splits of the uv points whose last one is short, more blocks than SMs and fewer.

Tolerances: FP32 sums of at most N (N pixels of a row, N rows) or 64 terms a split, 2^-24 each and random: V 1e-6 of the flux,
the adjoint of given weights 2e-6 of its norm, both against direct FP64 sums.
"""
import numpy as np
import pytest

import gpair_b200 as g
from test_uvgrid import _adjoint, _direct, _image, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nuv,nbis", [(1, 3, 1), (31, 15, 4), (32, 16, 0), (33, 17, 9), (63, 900, 1200), (64, 901, 1201),
                                        (65, 2369, 40), (64, 4753, 10), (95, 33, 5), (130, 31, 7), (64, 1, 0)])
def test_contractions(N, nuv, nbis):
    rng = np.random.default_rng(N * 1000 + nuv)
    p = _problem(N, rng.uniform(-0.1, 0.1, (nuv, 2)), nbis, N)
    img = _image(N, N + 1)
    V, chi2, _ = _direct(p, img)
    w = (rng.standard_normal(nuv) + 1j * rng.standard_normal(nuv)).astype(np.complex64)
    want = _adjoint(p, w)
    with g.Reconstructor(0) as r:
        r.set_problem(p)
        r.set_image(img)
        got, S = r.criterion()
        assert np.abs(r.visibilities() - V).max() <= 1e-6
        assert abs(got / chi2 - 1) <= 2e-5
        I, m = img.astype(np.float64), p.model.astype(np.float64)
        want_S = np.sum(I - m - I * np.log(I / m))
        assert abs(S - want_S) <= 1e-12 * np.sum(np.abs(I) + m + np.abs(I * np.log(I / m)))
        assert np.linalg.norm(r.adjoint_image(w) - want) <= 2e-6 * np.linalg.norm(want)
