"""Runs of several contexts are in a line: with their loops in flight side by side a call now and then never returned."""
import time

import numpy as np
import pytest

import gpair_b200 as g
from gpair_b200.instances import instance

pytestmark = pytest.mark.gpu


@pytest.fixture
def contexts():
    recs, ps = [], [instance(20_000_000 + k) for k in range(12)]
    try:
        for p in ps:
            r = g.Reconstructor(0)
            recs.append(r)
            r.set_tc_pair(False)
            r.set_problem(p)
            r.set_precision(g.PREC_SPLIT16)
        yield recs, ps
    finally:
        for r in recs:
            r.close()


def _start(recs, ps):
    for r, p in zip(recs, ps):
        r.set_image(p.start_image())


@pytest.mark.parametrize("flags,search,layout", [
    ({}, g.LS_BATCH, 2), ({"forwards_only": True}, g.LS_BATCH, 1), ({"mixed": True}, g.LS_BATCH, 1),
    ({"independent": True}, g.LS_BATCH, 0), ({}, g.LS_WOLFE, 0)])
def test_batch_graph_is_one_line(contexts, flags, search, layout):
    """No level of the graph has two roots, or two nodes that wait for the same one."""
    recs, ps = contexts
    flags = dict(flags)
    if flags.pop("mixed", False):
        recs[1].set_precision(g.PREC_FP32)
        recs[2].set_precision(g.PREC_SPLIT16F8)
    _start(recs, ps)
    with g.api.Batch(recs, line_search=search, **flags) as b:
        assert (b.grouped, b.branches) == (layout, 1)


def test_runs_of_one_call_do_not_overlap(contexts):
    """The device times of the runs, start to end, fit one after another into the call; the results are the separate runs'."""
    recs, ps = contexts
    _start(recs, ps)
    single = [(r.cg(20, method=2, line_search=g.LS_BATCH)["J"], r.get_image()) for r in recs]
    _start(recs, ps)
    t0 = time.perf_counter()
    many = g.cg_many(recs, 20, method=2, line_search=g.LS_BATCH)
    wall = (time.perf_counter() - t0) * 1e3
    assert sum(r.last_run_stats()[0] for r in recs) <= wall
    for r, (J, img), m in zip(recs, single, many):
        assert m["status"] == 0 and m["iterations"] == 20 and m["J"] == J
        assert np.array_equal(r.get_image(), img)
