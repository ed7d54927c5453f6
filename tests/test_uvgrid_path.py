"""Which path a problem takes: the uv grid or direct sums, by the context's own answer (gpair_uv_grid).

Paths are compared with what the rule says, runs with runs bit for bit; the one tolerance is the library's 1e-5.
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


def _extent(p):
    """Grid columns and rows each way (nbx, J) of a problem: first window points floor(2 N |f|) - 3, 8 of them."""
    f = U.RPMAS * np.float64(np.float32(p.pixellation)) * p.uv[:, :2].astype(np.float64)
    f -= np.rint(f)
    f[f[:, 0] < 0] *= -1
    j = np.floor(f * 2 * p.width).astype(int) - 3
    return j[:, 0].max() - j[:, 0].min() + 8, max((-j[:, 1]).max(), (j[:, 1] + 7).max())


@pytest.mark.parametrize("N", [256, 301])
@pytest.mark.parametrize("mode,ratio", [(g.PREC_SPLIT16, 300), (g.PREC_SPLIT16F8, 450), (g.PREC_TF32, 450)])
def test_wide_coverage_line(N, mode, ratio):
    """A few points at the edge of the plane, the others inside: the last uv count left to the direct sums, the first on the grid."""
    edge = np.array([[0.49, 0.49], [0.49, -0.49], [0.0, 0.0]])

    def problem(nuv):
        f = _freq("inner", nuv, 1)
        f[:3] = edge
        return _problem(N, f, 10, 2)

    nbx, J = _extent(problem(10))
    first = int(np.ceil(ratio * nbx * J / (2 * N)))
    for nuv, grid in ((first - 1, False), (first, True)):
        p = problem(nuv)
        assert _extent(p) == (nbx, J)
        with g.Reconstructor(0) as r:
            r.set_problem(p)
            assert r.uv_grid(mode) == grid
            assert r.uv_grid(g.PREC_FP32) and r.uv_grid(g.PREC_TF32X3)


@pytest.mark.parametrize("N,nuv", [(515, 9001), (330, 8200)])
def test_wide_coverage_on_either_path(N, nuv):
    """Points over the whole plane: V, chi2 and the adjoint of given weights within 1e-5 on the path that each mode takes."""
    p = _problem(N, _freq("full", nuv, 5), 500, 6)
    img = _image(N, 7)
    V, chi2, _ = U._direct(p, img)
    rng = np.random.default_rng(4)
    w = (rng.standard_normal(nuv) + 1j * rng.standard_normal(nuv)).astype(np.complex64)
    adj = U._adjoint(p, w)
    with g.Reconstructor(0) as r:
        r.set_problem(p)
        for mode, grid in ((g.PREC_SPLIT16, False), (g.PREC_FP32, True), (g.PREC_SPLIT16F8, False), (g.PREC_TF32X3, True)):
            r.set_precision(mode)
            assert r.uv_grid() == grid
            r.set_image(img)
            c, _ = r.criterion()
            assert np.abs(r.visibilities() - V).max() <= 1e-5
            assert abs(c - chi2) <= 1e-5 * chi2
            assert np.linalg.norm(r.adjoint_image(w) - adj) <= 1e-5 * np.linalg.norm(adj)
