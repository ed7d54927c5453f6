"""Which path a problem takes: the uv grid or direct sums, by the context's own answer (gpair_uv_grid).

No tolerances here: paths are compared with what the rule says, runs with runs bit for bit.
"""
import numpy as np
import pytest

import gpair_b200 as g
import test_uvgrid as U
import test_uvgrid_runs as R
from test_uvgrid import _freq, _image, _problem

pytestmark = pytest.mark.gpu


def _context(N, nuv, kind="inner", nbis=10):
    r = g.Reconstructor(0)
    r.set_problem(_problem(N, _freq(kind, nuv, N), nbis, N))
    return r


# the last uv count below a mode's least direct work 2 N^2 nuv (4e7, 1.2e9, 4e9) and the first one at it
@pytest.mark.parametrize("N,nuv,mode", [(128, 1221, g.PREC_FP32), (256, 9156, g.PREC_SPLIT16), (256, 9156, g.PREC_TF32),
                                        (256, 9156, g.PREC_TF32X3), (256, 30518, g.PREC_SPLIT16F8)])
def test_least_work(N, nuv, mode):
    for k, grid in ((nuv - 1, False), (nuv, True)):
        with _context(N, k) as r:
            assert r.uv_grid(mode) == grid
            r.set_precision(mode)
            assert r.uv_grid() == grid
            r.set_image(_image(N, 1))
            assert np.isfinite(r.criterion()).all()


def test_least_width():
    for N, grid in ((95, False), (96, True)):
        with _context(N, 20000) as r:
            assert r.uv_grid() == grid


def test_answer_follows_the_mode():
    with _context(256, 12000) as r:  # between the lines of split-f16 and split-f16/E4M3
        for mode, grid in ((g.PREC_FP32, True), (g.PREC_SPLIT16, True), (g.PREC_SPLIT16F8, False),
                           (g.PREC_FP32, True), (g.PREC_SPLIT16F8, False), (g.PREC_TF32X3, True)):
            r.set_precision(mode)
            assert r.uv_grid() == grid and r.uv_grid(g.PREC_SPLIT16) and not r.uv_grid(g.PREC_SPLIT16F8)
    with g.Reconstructor(0) as r:
        with pytest.raises(g.GpairError):
            r.uv_grid()  # no problem


@pytest.mark.parametrize("case", [c for c in U.CASES if c[0] >= 96])
def test_fp32_cases_are_on_the_grid(case):
    with _context(case[0], case[1], case[3]) as r:
        assert r.uv_grid()


def test_one_cell_on_the_grid():
    """The problem of test_fp32_grid_matches_direct_sums whose points share a cell or two, at a width that takes the grid."""
    case = (100, 8200, 100, "cell")
    with _context(case[0], case[1], case[3]) as r:
        assert r.uv_grid()
    U.test_fp32_grid_matches_direct_sums(case)


@pytest.mark.parametrize("case", [m.args[1] for m in R.test_runs_and_trials.pytestmark if m.name == "parametrize"][0])
def test_run_cases_are_on_the_grid(case):
    N, nuv, nbis, kind, mode = case
    with _context(N, nuv, kind) as r:
        assert r.uv_grid(mode)


@pytest.mark.parametrize("search", [g.LS_BATCH, g.LS_WOLFE])
def test_runs_between_changes_of_the_path(search):
    """One context from direct sums to the grid and back between runs: each run is a fresh context's."""
    N, nuv = 256, 12000
    want = {}
    for mode in (g.PREC_SPLIT16F8, g.PREC_SPLIT16, g.PREC_FP32):
        with _context(N, nuv, nbis=3000) as r:
            r.set_precision(mode)
            r.set_image(_image(N, 2))
            want[mode] = r.cg(2, line_search=search)["J"], r.get_image()
    with _context(N, nuv, nbis=3000) as r:
        for mode in (g.PREC_SPLIT16F8, g.PREC_SPLIT16, g.PREC_SPLIT16F8, g.PREC_FP32, g.PREC_SPLIT16, g.PREC_FP32):
            r.set_precision(mode)
            r.set_image(_image(N, 2))
            out = r.cg(2, line_search=search)
            assert out["J"] == want[mode][0] and np.array_equal(r.get_image(), want[mode][1])


def test_wolfe_batch_with_instances_on_the_grid():
    recs = [_context(N, nuv, nbis=nuv // 2) for N, nuv in ((96, 1500), (330, 9001), (128, 900), (256, 9200))]
    try:
        alone = []
        for r in recs:
            r.set_precision(g.PREC_SPLIT16)
        assert [r.uv_grid() for r in recs] == [False, True, False, True]
        for r in recs:
            r.set_image(r.problem.start_image())
            alone.append((r.cg(3, method=2, line_search=g.LS_WOLFE), r.get_image()))
        with g.api.Batch(recs, line_search=g.LS_WOLFE) as b:
            for _ in range(2):
                for r in recs:
                    r.set_image(r.problem.start_image())
                for r, o, (a, img) in zip(recs, b.run(3), alone):
                    assert o["J"] == a["J"] and np.array_equal(r.get_image(), img)
    finally:
        for r in recs:
            r.close()
