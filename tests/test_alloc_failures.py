"""Calls that run out of device memory fail with an error and leave a context that works once there is memory again.

Device memory is taken by one tensor up to a few MB, so that another of a call's allocations is the first to fail each time;
nothing is written to it. No tolerances: the results afterwards are those of a context that never failed, bit for bit.
"""
import numpy as np
import pytest

import gpair_b200 as g
from test_uvgrid import _freq, _image, _problem

pytestmark = pytest.mark.gpu

MB = 1 << 20


class _Full:
    """Device memory taken up to `leave` bytes."""

    def __init__(self, leave):
        import torch
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        for spare in range(0, 64 * MB, 2 * MB):  # not all of what is free can be had
            try:
                self.t = torch.empty(max(0, (free - leave - spare) // (2 * MB) * 2 * MB), dtype=torch.uint8, device="cuda")
                break
            except torch.OutOfMemoryError:
                pass

    def __enter__(self):
        return self

    def __exit__(self, *a):
        import torch
        self.t = None
        torch.cuda.empty_cache()


def _context(N, nuv, precision=g.PREC_FP32):
    r = g.Reconstructor(0)
    r.set_problem(_problem(N, _freq("inner", nuv, N), nuv // 4, N))
    if precision != g.PREC_FP32:
        r.set_precision(precision)
    r.set_image(_image(N, 5))
    return r


def _evaluation(r):
    value = r.criterion()
    r.gradient()
    return value, r.full_gradient()


# direct contractions (operands of 8 and 16 MB each), and the uv grid in every mode
@pytest.mark.parametrize("N,nuv", [(250, 8000), (450, 30000)])
@pytest.mark.parametrize("precision", [g.PREC_SPLIT16, g.PREC_SPLIT16F8, g.PREC_TF32X3])
def test_set_precision(N, nuv, precision):
    with _context(N, nuv, precision) as r:
        want = _evaluation(r)
    with _context(N, nuv) as r:
        fp32 = _evaluation(r)
    failed = 0
    for leave in (0, 6, 18, 30, 48, 66):
        r = _context(N, nuv)
        assert _evaluation(r)[0] == fp32[0]
        with _Full(leave * MB):
            try:
                r.set_precision(precision)
            except g.GpairError:
                failed += 1
                assert r._L.gpair_get_precision(r.h) == g.PREC_FP32
        if r._L.gpair_get_precision(r.h) == g.PREC_FP32:
            value, grad = _evaluation(r)
            assert value == fp32[0] and np.array_equal(grad, fp32[1])
            r.set_precision(precision)
        value, grad = _evaluation(r)
        assert value == want[0] and np.array_equal(grad, want[1])
        r.close()
    assert failed or N == 450  # a tensor mode's operands on the grid may fit into what was left


@pytest.mark.parametrize("N,nuv", [(250, 8000), (450, 30000)])
@pytest.mark.parametrize("precision", [g.PREC_FP32, g.PREC_SPLIT16, g.PREC_SPLIT16F8])
@pytest.mark.parametrize("method", [2, 4])
def test_batched_run(N, nuv, precision, method):
    with _context(N, nuv, precision) as r:
        want = r.cg(2, method=method, line_search=g.LS_BATCH)["J"], r.get_image()
    failed = 0
    for leave in (0, 4, 10, 20, 60):
        r = _context(N, nuv, precision)
        _evaluation(r)
        with _Full(leave * MB):
            try:
                r.cg(2, method=method, line_search=g.LS_BATCH)
            except g.GpairError:
                failed += 1
        r.set_image(_image(N, 5))
        got = r.cg(2, method=method, line_search=g.LS_BATCH)["J"], r.get_image()
        assert got[0] == want[0] and np.array_equal(got[1], want[1])
        r.close()
    assert failed
