"""The uv grid's sums over runs of points (csrc/uvgrid.cu): cells with many runs and with a last run of a few points, and
the trials of the batched search.

Tolerances: the adjoint of given weights against direct FP64 sums, 2e-6 of its norm in FP32 (window 1e-7 and FP32 sums of at
most a few hundred terms a stage), 1e-5 on the tensor path; a batched search never accepts a rise of the objective.
"""
import numpy as np
import pytest

import gpair_b200 as g
from test_uvgrid import _adjoint, _freq, _image, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nuv,nbis,kind,precision", [
    (100, 8200, 100, "cell", g.PREC_FP32),      # one cell or two: 256 runs each, a last run of 8 points
    (280, 8231, 300, "cell", g.PREC_SPLIT16),
    (147, 1904, 3801, "inner", g.PREC_FP32),    # a few points a cell
    (281, 9001, 65, "inner", g.PREC_TF32X3),
    (401, 12545, 1, "inner", g.PREC_SPLIT16F8),  # no triangles to speak of
    (256, 9221, 30011, "wrapped", g.PREC_SPLIT16)])
def test_runs_and_trials(N, nuv, nbis, kind, precision):
    p = _problem(N, _freq(kind, nuv, N), nbis, N)
    rng = np.random.default_rng(N)
    w = (rng.standard_normal(nuv) + 1j * rng.standard_normal(nuv)).astype(np.complex64)
    want = _adjoint(p, w)
    with g.Reconstructor(0) as r:
        r.set_problem(p)
        r.set_precision(precision)
        r.set_image(_image(N, N + 1))
        tol = 2e-6 if precision == g.PREC_FP32 else 1e-5
        assert np.linalg.norm(r.adjoint_image(w) - want) <= tol * np.linalg.norm(want)
        out = r.cg(3, method=2, trace=True, line_search=g.LS_BATCH)
        assert np.all(np.diff(out["trace_J"]) <= 0)
        one = r.get_image()
        r.set_image(_image(N, N + 1))
        r.cg(3, method=2, line_search=g.LS_BATCH)
        assert np.array_equal(r.get_image(), one)  # the same sums every time
