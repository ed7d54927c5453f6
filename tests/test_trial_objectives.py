"""The objectives of the batched search's trials against FP64 sums, on the uv grid and directly.

A checkpoint holds the steps that an iteration tried with their objectives, and the direction; the trial images follow from them.
Tolerance: that of a single evaluation, 2e-6 of chi2 in FP32 and 1e-5 in the tensor modes (tests/test_uvgrid.py).
"""
import ctypes as C

import numpy as np
import pytest

import gpair_b200 as g
from test_uvgrid import RPMAS, _freq, _image, _problem

pytestmark = pytest.mark.gpu

TRIALS, ROUNDS, PAIRS = 8, 6, 4


class _CgState(C.Structure):
    """The controller state of a checkpoint (CgState of csrc/gpair_internal.cuh)."""
    _fields_ = [(n, C.c_int) for n in ("method", "max_zoom", "max_bracket", "run_limit")] + \
               [(n, C.c_double) for n in ("alpha", "minvalue", "c1", "c2", "step_max")] + \
               [("ls_mode", C.c_int), ("target_J", C.c_double), ("batch_step_max", C.c_double), ("it", C.c_int)] + \
               [(n, C.c_double) for n in ("J", "chi2", "entropy", "beta", "wolfe1", "prev_nn")] + \
               [(n, C.c_int) for n in ("phase", "ls_it", "action", "zoom_counter", "zoom_trials", "bracket_trials")] + \
               [(n, C.c_double) for n in ("s", "s_old", "J_init", "J_old", "Jt", "lo", "hi", "J_lo", "z_s", "z_s_old", "z_J_old",
                                          "sel")] + \
               [(n, C.c_int) for n in ("criterion_evals", "grad_evals", "run_it", "batches", "reached", "stopped", "bphase",
                                       "bround", "npts", "force_sd")] + \
               [("s_c", C.c_double), ("ts", C.c_double * TRIALS), ("pts_s", C.c_double * (ROUNDS * TRIALS)),
                ("pts_J", C.c_double * (ROUNDS * TRIALS))] + \
               [(n, C.c_int) for n in ("lb_count", "lb_xvalid", "lb_drop")] + [("lb_slot", C.c_int * (PAIRS + 1))] + \
               [("lb_sy", C.c_double * PAIRS ** 2), ("lb_yy", C.c_double * PAIRS ** 2), ("lb_gamma", C.c_double),
                ("lb_cq", C.c_double), ("lb_cs", C.c_double * PAIRS), ("lb_cy", C.c_double * PAIRS)]


def _state(data, npix):
    """(controller state, direction) of a checkpoint's bytes."""
    head = np.frombuffer(data, np.uint32, 2, 8 + 6 * 4)
    assert head[0] == C.sizeof(_CgState) and head[1] == 5
    at = 8 + 8 * 4
    s = _CgState.from_buffer_copy(data, at)
    return s, np.frombuffer(data, np.float32, npix, at + C.sizeof(_CgState) + 4 * npix)


def _objective(p, images, tables):
    """chi2 - alpha S and chi2 of images, in FP64."""
    import torch
    fx, fy = tables
    N = p.width
    out = []
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    d, w, at, sg = up(p.data).double(), up(p.data_err).double(), up(p.uvpnt), up(p.sign) < 0
    ph, m = up(p.phasor).to(torch.complex128), up(p.model).double()
    for img in images:
        I = up(img).double()
        V = ((fx @ I.reshape(N, N).T.to(torch.complex128)) * fy).sum(1) / I.sum()
        side = torch.where(sg, V[at].conj(), V[at])
        t3 = side[:, 0] * side[:, 1] * side[:, 2] * ph
        mock = torch.empty_like(d)
        mock[:p.npow], mock[p.npow::2], mock[p.npow + 1::2] = V[:p.npow].abs() ** 2, t3.real, t3.imag
        chi2 = float((((mock - d) * w) ** 2).sum())
        out.append((chi2 - float(np.float32(p.alpha)) * float((I - m - I * torch.log(I / m)).sum()), chi2))
    return out


# grid: wide images, whose trials' blocks fill the device without partial sums; direct: below the lines
@pytest.mark.parametrize("N,nuv,mode,grid", [
    (1024, 1500, g.PREC_FP32, True), (147, 1904, g.PREC_FP32, True), (130, 600, g.PREC_FP32, False),
    (1024, 6000, g.PREC_SPLIT16, True), (300, 9001, g.PREC_TF32X3, True), (200, 3000, g.PREC_SPLIT16, False),
    (1100, 9000, g.PREC_SPLIT16F8, True), (200, 3000, g.PREC_SPLIT16F8, False)])
def test_trials(N, nuv, mode, grid):
    import torch
    p = _problem(N, _freq("inner", nuv, N), nuv, N)
    img = _image(N, 2)
    s = RPMAS * np.float64(np.float32(p.pixellation))
    x = torch.arange(N, dtype=torch.float64, device="cuda")
    u, v = (torch.from_numpy(p.uv[:, i].astype(np.float64) * s).cuda()[:, None] * x * (2 * np.pi) for i in (0, 1))
    tables = torch.complex(u.cos(), u.sin()), torch.complex(v.cos(), -v.sin())
    with g.Reconstructor(0) as r:
        r.set_precision(mode)
        r.set_problem(p)
        assert r.uv_grid() == grid
        r.set_image(img)
        r.cg(1, method=2, line_search=g.LS_BATCH)
        st, d = _state(r.checkpoint(), N * N)
    assert st.npts >= TRIALS and st.minvalue > 0
    steps = np.array(st.pts_s[:st.npts])
    trials = [np.maximum(img.astype(np.float64) + a * d.astype(np.float64), st.minvalue).astype(np.float32) for a in steps]
    tol = 2e-6 if mode == g.PREC_FP32 else 1e-5
    for a, got, (want, chi2) in zip(steps, st.pts_J, _objective(p, trials, tables)):
        assert abs(got - want) <= tol * chi2, (a, got, want)
