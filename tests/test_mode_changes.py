"""Changes of the precision mode between runs: a run after them is the run of a context that was never changed.

No tolerances: the same sums in the same order give the same bits.
"""
import numpy as np
import pytest

import gpair_b200 as g
from test_uvgrid import _freq, _image, _problem

pytestmark = pytest.mark.gpu


def _context(N, nuv, precision):
    r = g.Reconstructor(0)
    r.set_problem(_problem(N, _freq("inner", nuv, N), nuv // 2, N))
    r.set_precision(precision)
    return r


def _run(r, N, search):
    r.set_image(_image(N, 3))
    out = r.cg(2, method=2, line_search=search)
    return out["J"], r.get_image()


# direct contractions, and the uv grid in every mode
@pytest.mark.parametrize("N,nuv", [(64, 700), (330, 20001)])
@pytest.mark.parametrize("search", [g.LS_WOLFE, g.LS_BATCH])
@pytest.mark.parametrize("mode,other", [(g.PREC_SPLIT16, g.PREC_TF32X3), (g.PREC_SPLIT16F8, g.PREC_TF32)])
def test_run_after_a_change_and_back(N, nuv, search, mode, other):
    with _context(N, nuv, mode) as r, _context(N, nuv, mode) as fresh:
        want = _run(r, N, search)
        r.set_precision(other)  # frees the operands that the first run's graph holds
        taken = _context(N, nuv, mode)  # takes memory that became free
        r.set_precision(mode)
        got = _run(r, N, search)
        first = _run(fresh, N, search)
        assert got[0] == want[0] == first[0]
        assert np.array_equal(got[1], want[1]) and np.array_equal(got[1], first[1])
        taken.close()


@pytest.mark.parametrize("precision", [g.PREC_FP32, g.PREC_SPLIT16])
@pytest.mark.parametrize("search", [g.LS_WOLFE, g.LS_BATCH])
def test_batch_after_a_new_problem_is_refused(precision, search):
    """The batch's graph holds the buffers of the problem that it was made for."""
    recs = [_context(64, 700, precision) for _ in range(2)]
    for r in recs:
        r.set_image(_image(64, 3))
    b = g.api.Batch(recs, line_search=search)
    b.run(1)
    recs[1].set_problem(_problem(64, _freq("inner", 900, 1), 300, 2))
    recs[1].set_image(_image(64, 3))
    with pytest.raises(g.GpairError):
        b.run(1)
    b.close()
    for r in recs:
        r.close()


def _devices():
    import torch
    return torch.cuda.device_count() if torch.cuda.is_available() else 0


@pytest.mark.skipif(_devices() < 2, reason="needs two devices")
def test_mode_of_a_context_on_another_device():
    """One thread with a context on each device: a change of the first one's mode allocates on its own device."""
    p = _problem(330, _freq("inner", 20001, 1), 300, 2)
    recs = [g.Reconstructor(d) for d in (0, 1)]
    for r in recs:
        r.set_problem(p)
        r.set_image(_image(330, 3))
    got = []
    for r in recs[::-1] + recs:  # the current device is the other one's at every second step
        r.set_precision(g.PREC_SPLIT16)
        got.append(r.criterion()[0])
        r.set_precision(g.PREC_FP32)
    assert len(set(got)) == 1
    for r in recs:
        r.close()
