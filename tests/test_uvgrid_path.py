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


def _used():
    import torch
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_plan_is_built_by_the_mode_that_takes_it():
    """1024 pixels and points over the whole plane: the grid for FP32, direct sums for split-f16. The plan (S alone is
    2 x 8.5 MB, the x contraction's sums 8.5 MB) exists once FP32 has been set, and not in a context that was split-f16 before the
    problem was loaded."""
    p = _problem(1024, _freq("full", 9500, 5), 100, 6)
    img = _image(1024, 7)
    want = []
    used = []
    for fp32 in (False, True):
        with g.Reconstructor(0) as r:
            u0 = _used()
            r.set_precision(g.PREC_FP32 if fp32 else g.PREC_SPLIT16)
            r.set_problem(p)
            r.set_precision(g.PREC_SPLIT16)
            assert r.uv_grid(g.PREC_FP32) and not r.uv_grid()
            used.append(_used() - u0)
            r.set_image(img)
            one = r.criterion()
            r.set_precision(g.PREC_FP32)
            want += [one, r.criterion()]
            r.set_precision(g.PREC_SPLIT16)
            assert r.criterion() == one
    assert want[:2] == want[2:]
    assert used[1] - used[0] >= 16 << 20


@pytest.mark.parametrize("first", ["criterion", "adjoint", "cg", "host_loop", "batch", "batched_search", "time_stages",
                                   "time_batch_stages", "autotune", "checkpoint"])
def test_first_call_in_fp32(first):
    """Each entry point as a new context's first: the results are those after an evaluation."""
    N, nuv = 147, 1904
    rng = np.random.default_rng(4)
    w = (rng.standard_normal(nuv) + 1j * rng.standard_normal(nuv)).astype(np.complex64)
    got = []
    for warm in (True, False):
        with _context(N, nuv, nbis=900) as r:
            assert r.uv_grid()
            r.set_image(_image(N, 2))
            if warm:
                r.criterion()
                r.gradient()
                r.set_image(_image(N, 2))
            if first == "criterion":
                out = r.criterion()
            elif first == "adjoint":
                out = r.adjoint_image(w).tolist()
            elif first == "cg":
                out = r.cg(2)["J"]
            elif first == "host_loop":
                out = r.cg(2, host_loop=1)["J"]
            elif first == "batch":
                with g.api.Batch([r]) as b:
                    out = b.run(2)[0]["J"]
            elif first == "batched_search":
                out = r.cg(2, line_search=g.LS_BATCH)["J"]
            elif first == "time_stages":
                out = len(r.time_stages(2))
            elif first == "time_batch_stages":
                out = len(r.time_batch_stages(2))
            elif first == "autotune":
                r.autotune(g.api.TUNE_SPLITS)
                out = r.criterion()
            else:
                with _context(N, nuv, nbis=900) as other:
                    other.set_image(_image(N, 2))
                    other.cg(1)
                    r.restore(other.checkpoint())
                out = r.cg(1, resume=True)["J"]
            got.append((out, r.get_image().tolist()))
    assert got[0] == got[1]


@pytest.mark.parametrize("mode", [g.PREC_FP32, g.PREC_TF32X3])
def test_memory_of_a_wide_image(mode):
    """1,500 pixels, a grid of 371 x 731 points: images (9 + 8 trials of 9 MB), the x contraction's sums as many as the mode takes (FP32
    one of 744 floats a row; TF32X3 eight, and eight of its operand stack of 1,536 rows an image), grids and points."""
    N, nuv = 1500, 20000
    f = np.random.default_rng(1).uniform(-0.12, 0.12, (nuv, 2))
    p = _problem(N, f, 100, 2)
    nbx, J = _extent(p)
    with g.Reconstructor(0) as r:
        u0 = _used()
        r.set_precision(mode)
        r.set_problem(p)
        assert r.uv_grid()
        r.set_image(_image(N, 3))
        r.cg(1, line_search=g.LS_BATCH)
        sums = 4 * (2 * nbx + 4) * (N * 9 if mode == g.PREC_FP32 else 8 * (N + 8 * 1536))
        operands = 0 if mode == g.PREC_FP32 else 8 * (9 * 1536 + 2 * nbx + 128) * 1504
        rest = 8 * nbx * (2 * J + 1) * 10 + 8 * N * nbx + 1000 * nuv
        assert _used() - u0 <= 17 * 4 * N * N + sums + operands + rest + (64 << 20)  # allocations in blocks of 2 MB, the run's graph


def test_sums_of_both_kinds_of_core():
    """FP32 and tensor modes on the grid keep sums of their own: changes between batched runs leave the other's alone, and a batch of a
    mode still runs after evaluations in another."""
    N, nuv = 330, 20001
    want = {}
    for mode in (g.PREC_FP32, g.PREC_SPLIT16):
        with _context(N, nuv, nbis=2000) as r:
            r.set_precision(mode)
            r.set_image(_image(N, 2))
            want[mode] = r.cg(2, line_search=g.LS_BATCH)["J"], r.get_image()
    with _context(N, nuv, nbis=2000) as r:
        r.set_precision(g.PREC_SPLIT16)
        assert r.uv_grid() and r.uv_grid(g.PREC_FP32)
        r.set_image(_image(N, 2))
        with g.api.Batch([r], line_search=g.LS_BATCH) as b:
            for mode in (g.PREC_SPLIT16, g.PREC_FP32, g.PREC_SPLIT16):
                r.set_precision(mode)
                r.set_image(_image(N, 2))
                out = r.cg(2, line_search=g.LS_BATCH)
                assert out["J"] == want[mode][0] and np.array_equal(r.get_image(), want[mode][1])
            r.set_image(_image(N, 2))
            assert b.run(2)[0]["J"] == want[g.PREC_SPLIT16][0]


def test_tuned_choice_is_not_taken_over_by_another_path():
    """Equal widths and uv counts: a compact coverage on the grid, one too wide for it, and one on the grid in FP32 alone."""
    flags = g.api.TUNE_PRECISION | g.api.TUNE_SPLITS | g.api.TUNE_TILE | g.api.TUNE_CACHE
    seen = []
    for kind, nuv, grid in (("inner", 5000, (True, False, True)), ("full", 5000, (False, False, True)),
                            ("inner", 5001, (True, False, True))):
        with _context(512, nuv, kind) as r:
            assert (r.uv_grid(g.PREC_SPLIT16), r.uv_grid(g.PREC_SPLIT16F8), r.uv_grid(g.PREC_FP32)) == grid
            r.set_image(_image(512, 3))
            t = r.autotune(flags, reps=2)
            seen.append(t)
            tune = r.uv_grid(t["precision"])
            assert (t["adjoint_splits"] == 0) == tune
            for prec, splits, tile, _ in t["candidates"]:
                assert (splits == 0) == r.uv_grid(prec)
                assert tile == 0 if prec == g.PREC_FP32 else tile in ((128,) if r.uv_grid(prec) else (128, 256))
            assert np.isfinite(r.criterion()).all()
    assert [t["from_cache"] for t in seen] == [False, False, True]
    assert seen[2]["precision"] == seen[0]["precision"]
    # S16 and FP32 on the grid: one candidate each; F8 directly: two tiles, up to three splits each
    assert sum(c[0] != g.PREC_SPLIT16F8 for c in seen[0]["candidates"]) == 2


def test_tuning_on_the_grid_leaves_the_tile():
    with _context(512, 20000) as r:
        assert all(r.uv_grid(m) for m in (g.PREC_FP32, g.PREC_SPLIT16, g.PREC_SPLIT16F8))
        r.set_image(_image(512, 3))
        for pair in (True, False):
            r.set_tc_pair(pair)
            t = r.autotune(g.api.TUNE_PRECISION | g.api.TUNE_SPLITS | g.api.TUNE_TILE, reps=2)
            assert len(t["candidates"]) == 3 and t["adjoint_splits"] == 0
            assert r._L.gpair_get_tc_pair(r.h) == pair
