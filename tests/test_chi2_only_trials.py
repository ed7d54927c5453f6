"""A captured Wolfe search over large data forms chi2 alone at its trials (csrc/kernels_core.cu, k_vis_chi2): the run
on the device against the same run driven by the host, which evaluates everything at every trial. No tolerance: the same bits,
also of what the run leaves behind (V, mock data, the gradient of the last evaluation's weights)."""
import numpy as np
import pytest

import gpair_b200 as g
from test_uvgrid import _freq, _image, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nuv,nbis,precision", [
    (64, 1501, 900_000, g.PREC_FP32),       # direct, one partial entry
    (130, 2003, 890_003, g.PREC_SPLIT16),   # direct tensor path, two entries
    (300, 1501, 890_001, g.PREC_SPLIT16),   # three or more: V summed beforehand
    (150, 3001, 950_000, g.PREC_FP32)])     # the uv grid
def test_device_run_equals_host_driven_run(N, nuv, nbis, precision):
    p = _problem(N, _freq("inner", nuv, N), nbis, N)
    got = []
    for host_loop in (1, 0):
        with g.Reconstructor(0) as r:
            r.set_problem(p)
            r.set_precision(precision)
            r.set_image(_image(N, 3))
            out = r.cg(3, method=2, line_search=g.LS_WOLFE, host_loop=host_loop)
            V, mock = r.visibilities(), r.mock()
            got.append((out["J"], out["criterion_evals"], out["grad_evals"], r.get_image(), V, mock, r.criterion()))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
