"""The DFT and its adjoint through the uv grid (csrc/uvgrid.cu) against direct FP64 sums.

Tolerances, derived from the method before any run:
  window      interpolation from grid values by the 8-point Kaiser-Bessel window at twofold
              oversampling: 1e-7 of the flux (FP64 model, CPU)
  FP32        V: the window (1e-7) plus FP32 rounding of sums of at most a few hundred terms per
              stage (a few 2^-24 each): 1e-6 of the flux; gradient 2e-6 relative
  tensor      V 1e-5 of the flux, chi2 and gradient 1e-5 relative, the library's bounds
"""
import numpy as np
import pytest

import gpair_b200 as g

RPMAS = (np.pi / 180.0) / 3600000.0


def _problem(N, freq, nbis, seed, pix=0.1):
    """A problem whose uv points sit at `freq` (cycles per pixel, [nuv, 2]); data near a random image's."""
    rng = np.random.default_rng(seed)
    nuv = len(freq)
    uv = np.zeros((nuv, 4), np.float32)
    uv[:, :2] = freq / (RPMAS * np.float64(np.float32(pix)))
    tri = rng.integers(0, nuv, (nbis, 3)).astype(np.int64)
    sign = rng.choice(np.array([1, -1], np.int16), (nbis, 3))
    data = rng.uniform(0, 0.5, nuv + 2 * nbis).astype(np.float32)
    err = rng.uniform(5, 50, nuv + 2 * nbis).astype(np.float32)
    phasor = np.exp(1j * rng.uniform(-np.pi, np.pi, nbis)).astype(np.complex64)
    model = np.full(N * N, 1.0 / N ** 2, np.float32)
    return g.Problem(N, pix, uv, nuv, nbis, data, err, phasor, tri, sign, model, 1e-3)


def _image(N, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:N, 0:N] / N
    img = 0.5 + np.exp(-((x - 0.4) ** 2 + (y - 0.6) ** 2) / 0.02) * 20 + rng.uniform(0, 1, (N, N))
    return (img / img.sum()).astype(np.float32).ravel()


def _direct(p, img):
    """(V, chi2, data gradient) by direct FP64 sums."""
    N = p.width
    s = RPMAS * np.float64(np.float32(p.pixellation))
    x = np.arange(N)
    fx = np.exp(2j * np.pi * s * np.outer(p.uv[:, 0].astype(np.float64), x))
    fy = np.exp(-2j * np.pi * s * np.outer(p.uv[:, 1].astype(np.float64), x))
    I = img.astype(np.float64).reshape(N, N)
    F = I.sum()
    V = np.einsum("kx,yx,ky->k", fx, I, fy, optimize=True) / F
    d, w = p.data.astype(np.float64), p.data_err.astype(np.float64)
    side = np.where(p.sign < 0, V[p.uvpnt].conj(), V[p.uvpnt])
    ph = p.phasor.astype(np.complex128)
    t3 = side[:, 0] * side[:, 1] * side[:, 2] * ph
    mock = np.empty(p.npow + 2 * p.nbis)
    mock[:p.npow], mock[p.npow::2], mock[p.npow + 1::2] = np.abs(V[:p.npow]) ** 2, t3.real, t3.imag
    chi2 = np.sum(((mock - d) * w) ** 2)
    c = np.zeros(p.nuv, np.complex128)
    c[:p.npow] = 4 * w[:p.npow] ** 2 * (mock[:p.npow] - d[:p.npow]) * V[:p.npow].conj() / F
    re, im = slice(p.npow, None, 2), slice(p.npow + 1, None, 2)
    gt = (2 * w[re] ** 2 * (mock[re] - d[re]) - 2j * w[im] ** 2 * mock[im]) * ph / F
    for j in range(3):
        b = gt * side[:, (j + 1) % 3] * side[:, (j + 2) % 3]
        np.add.at(c, p.uvpnt[:, j], np.where(p.sign[:, j] < 0, b.conj(), b))
    G = np.einsum("ky,k,kx->yx", fy, c, fx, optimize=True).real
    return V, chi2, (G - (c * V).real.sum()).ravel()


def _adjoint(p, w):
    s = RPMAS * np.float64(np.float32(p.pixellation))
    x = np.arange(p.width)
    fx = np.exp(2j * np.pi * s * np.outer(p.uv[:, 0].astype(np.float64), x))
    fy = np.exp(-2j * np.pi * s * np.outer(p.uv[:, 1].astype(np.float64), x))
    return np.einsum("ky,k,kx->yx", fy, w.astype(np.complex128), fx, optimize=True).real.ravel()


def _freq(kind, nuv, seed):
    rng = np.random.default_rng(seed)
    if kind == "inner":  # an ordinary coverage: a small disk
        r, t = 0.06 * np.sqrt(rng.uniform(0, 1, nuv)), rng.uniform(0, 2 * np.pi, nuv)
        return np.stack([r * np.cos(t), r * np.sin(t)], axis=1)
    if kind == "wrapped":  # beyond half a cycle per pixel: the phase of whole cycles drops out
        return rng.uniform(-0.05, 0.05, (nuv, 2)) + rng.integers(-2, 3, (nuv, 2))
    if kind == "full":  # the whole plane, its edges and axes among it
        f = rng.uniform(-0.5, 0.5, (nuv, 2))
        f[:6] = [[0, 0], [0, 0.3], [0.3, 0], [0.5, -0.5], [-0.5, 0.25], [0.25, 0.5]]
        return f
    f = rng.uniform(0, 1e-4, (nuv, 2)) + [0.031, -0.017]  # "cell": all in one grid cell or two
    return f


# width, uv points, triangles: even and odd widths, not multiples of any tile, below and above one 32-pixel or
# 64-row tile; uv counts beside a warp's and a block's
CASES = [(147, 1904, 3800, "inner"), (64, 8200, 100, "cell"), (201, 1025, 0, "wrapped"), (150, 3001, 777, "full"),
         (257, 4097, 4000, "inner")]


@pytest.mark.parametrize("N", [33, 64, 150])
def test_window_error_bound(N):
    """FP64 model: V from the grid of spacing 1 / (2 N) by the 8 x 8 window, points over the whole plane."""
    rng = np.random.default_rng(N)
    M, W = 2 * N, 8
    beta = np.pi * W * (1 - N / (2 * M))
    xp = np.arange(N) - (N - 1) / 2
    z = np.sqrt(beta ** 2 - (np.pi * W * xp / M) ** 2)
    phi = W * np.sinh(z) / z / np.i0(beta)
    img = rng.uniform(0, 1, (N, N)) ** 4
    ab = rng.uniform(-0.5, 0.5, (300, 2))
    direct = np.einsum("kx,yx,ky->k", np.exp(2j * np.pi * np.outer(ab[:, 0], xp)), img,
                       np.exp(-2j * np.pi * np.outer(ab[:, 1], xp)), optimize=True)
    j = np.arange(-N - W, N + W + 1)
    G = (np.exp(-2j * np.pi * np.outer(j, xp) / M) / phi) @ img @ (np.exp(2j * np.pi * np.outer(xp, j) / M) / phi[:, None])
    gx, gy = ab[:, 0] * M, ab[:, 1] * M
    jx, jy = np.floor(gx).astype(int) - 3, np.floor(gy).astype(int) - 3
    V = np.zeros(300, complex)
    for a in range(W):
        for b in range(W):
            wx = np.i0(beta * np.sqrt(np.maximum(0, 1 - (2 * (gx - jx - b) / W) ** 2))) / np.i0(beta)
            wy = np.i0(beta * np.sqrt(np.maximum(0, 1 - (2 * (gy - jy - a) / W) ** 2))) / np.i0(beta)
            V += wx * wy * G[jy + a - j[0], jx + b - j[0]]
    assert np.abs(V - direct).max() <= 1e-7 * img.sum()


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_fp32_grid_matches_direct_sums(case):
    N, nuv, nbis, kind = case
    p = _problem(N, _freq(kind, nuv, 1), nbis, 2)
    img = _image(N, 3)
    V, chi2, grad = _direct(p, img)
    with g.Reconstructor(0) as r:
        r.set_problem(p)
        r.set_image(img)
        c, _ = r.criterion()
        assert np.abs(r.visibilities() - V).max() <= 1e-6
        assert abs(c - chi2) <= 2e-6 * chi2
        r.gradient()
        assert np.linalg.norm(r.data_gradient() - grad) <= 2e-6 * np.linalg.norm(grad)
        # the adjoint of given weights
        rng = np.random.default_rng(4)
        w = (rng.standard_normal(nuv) + 1j * rng.standard_normal(nuv)).astype(np.complex64)
        ref = _adjoint(p, w)
        assert np.linalg.norm(r.adjoint_image(w) - ref) <= 2e-6 * np.linalg.norm(ref)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [g.PREC_SPLIT16, g.PREC_TF32X3, g.PREC_SPLIT16F8])
@pytest.mark.parametrize("case", [(322, 20001, 3000, "inner"), (515, 9001, 500, "full")])
def test_tensor_grid_matches_direct_sums_and_precision_switches(case, prec):
    """The gradient of the second case is ill-conditioned (a noise image over the whole plane, |V| near 1e-3): its
    adjoint is checked on given weights."""
    N, nuv, nbis, kind = case
    p = _problem(N, _freq(kind, nuv, 5), nbis, 6)
    img = _image(N, 7)
    V, chi2, grad = _direct(p, img)
    rng = np.random.default_rng(4)
    w = (rng.standard_normal(nuv) + 1j * rng.standard_normal(nuv)).astype(np.complex64)
    adj = _adjoint(p, w)
    with g.Reconstructor(0) as r:
        r.set_problem(p)
        for mode in (prec, g.PREC_FP32, prec):
            r.set_precision(mode)
            r.set_image(img)
            c, _ = r.criterion()
            r.gradient()
            assert np.abs(r.visibilities() - V).max() <= 1e-5
            assert abs(c - chi2) <= 1e-5 * chi2
            if kind == "inner":
                assert np.linalg.norm(r.data_gradient() - grad) <= 1e-5 * np.linalg.norm(grad)
            assert np.linalg.norm(r.adjoint_image(w) - adj) <= 1e-5 * np.linalg.norm(adj)


@pytest.mark.gpu
@pytest.mark.parametrize("independent,fwd_only", [(False, False), (False, True), (True, False)])
def test_batches_with_grid_and_direct_instances_equal_separate_runs(independent, fwd_only):
    """One instance on the grid between direct ones, in every batch layout: the separate runs bit for bit."""
    ps = [_problem(N, _freq("inner", nuv, 8 + N), nuv // 2, N) for N, nuv in ((96, 1500), (330, 9001), (128, 900))]
    recs = [g.Reconstructor(0) for _ in ps]
    try:
        for r, p in zip(recs, ps):
            r.set_problem(p)
            r.set_precision(g.PREC_SPLIT16)
        alone = []
        for r, p in zip(recs, ps):
            r.set_image(p.start_image())
            alone.append((r.cg(3, method=2, line_search=g.LS_BATCH), r.get_image()))
        with g.api.Batch(recs, line_search=g.LS_BATCH, independent=independent, forwards_only=fwd_only) as b:
            assert b.grouped == (0 if independent else 1 if fwd_only else 2)
            for _ in range(2):
                for r, p in zip(recs, ps):
                    r.set_image(p.start_image())
                for r, o, (a, img) in zip(recs, b.run(3), alone):
                    assert o["J"] == a["J"] and np.array_equal(r.get_image(), img)
    finally:
        for r in recs:
            r.close()


@pytest.mark.gpu
def test_single_pixel_moves_on_the_grid():
    """update_pixel without tables: V of the changed image by direct FP64 sums."""
    p = _problem(147, _freq("inner", 1904, 1), 500, 2)
    img = _image(147, 3)
    with g.Reconstructor(0) as r:
        r.set_problem(p)
        r.set_image(img)
        r.criterion()
        c, _ = r.update_pixel(31, 140, float(img.max()) * 3)
        img[140 * 147 + 31] = np.float32(float(img.max()) * 3)
        V, chi2, _ = _direct(p, img)
        assert np.abs(r.visibilities() - V).max() <= 1e-6
        assert abs(c - chi2) <= 2e-6 * chi2
