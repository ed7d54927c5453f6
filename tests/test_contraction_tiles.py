"""The tensor contractions where an image's last tile is cut (csrc/umma_dft.cu): widths around the 32-row steps of the
tile's columns, one image and a stack of trial images, single CTAs and pairs.

Tolerances, against direct FP64 sums: V 1e-5 of the flux (E4M3 cross terms: 1e-4), the library's bound, and the adjoint
of given weights 1e-5 of its norm; chi2 12 times V's bound (residuals are about 0.5 and a triple product moves by three
times V's error, chi2 by twice the relative change of a residual).
"""
import numpy as np
import pytest

import gpair_b200 as g
from test_uvgrid import _adjoint, _direct, _image, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("precision", [g.PREC_SPLIT16, g.PREC_TF32X3, g.PREC_SPLIT16F8])
@pytest.mark.parametrize("N", [7, 32, 33, 63, 65, 97, 128, 129, 160, 161, 192, 225, 255, 257, 300])
def test_cut_tiles(N, precision, pair):
    rng = np.random.default_rng(N)
    p = _problem(N, rng.uniform(-0.02, 0.02, (213, 2)), 60, N)  # a bright image's short baselines: well conditioned
    img = _image(N, N + 1)
    tol = 1e-4 if precision == g.PREC_SPLIT16F8 else 1e-5
    V, chi2, _ = _direct(p, img)
    w = (rng.standard_normal(213) + 1j * rng.standard_normal(213)).astype(np.complex64)
    want = _adjoint(p, w)
    r = g.Reconstructor(0)
    r.set_problem(p)
    r.set_precision(precision)
    r.set_tc_pair(pair)
    r.set_image(img)
    got = r.criterion()[0]
    assert np.abs(r.visibilities() - V).max() <= tol
    assert abs(got / chi2 - 1) <= 12 * tol
    assert np.linalg.norm(r.adjoint_image(w) - want) <= 1e-5 * np.linalg.norm(want)
    out = r.cg(3, method=2, trace=True, line_search=g.LS_BATCH)
    assert np.all(np.diff(out["trace_J"]) <= 0)  # a trial misjudged by a wrong column would be accepted uphill
    r.close()
