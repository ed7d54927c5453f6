"""Performance cases: the work a program has this framework do, through its public entry points.

Every case is a dict of plain values. ``prepare`` makes what the program holds before the call
(seeded data of a random telescope array, the device contexts, the network), ``run`` is one pass of
the call itself, ``exact`` is the same result in 64 bits from numpy and torch alone.

The kinds of case:

* ``evaluate``  one objective and gradient for a program that runs its own optimiser: image in,
  chi2, regulariser and full gradient out (``inspect``: also the visibilities and the mock data, what
  a residual plot needs);
* ``moves``     single-pixel moves of an annealing or MCMC sampler, each with its new chi2;
* ``cg``        iterations of a reconstruction under way, on the device, with either line search and
  any direction rule;
* ``many``      independent reconstructions of uneven sizes in one staged batch;
* ``warm``      the learned warm start of one problem: feature maps, network, start image;
* ``train``     one training step of that network.

Widths, array sizes, channels and pixel sizes follow the repository's own workloads
(``gpair_b200.synth``, ``gpair_b200.instances``, ``gpair_b200.warmstart``).
"""
from __future__ import annotations

import itertools
import math

import numpy as np
import torch

import gpair_b200 as g
from gpair_b200 import api, synth, warmstart

RPMAS = math.pi / 180.0 / 3600000.0  # radians per milliarcsecond
PRECISIONS = {"fp32": g.PREC_FP32, "split16": g.PREC_SPLIT16, "tf32x3": g.PREC_TF32X3,
              "split16f8": g.PREC_SPLIT16F8}
SEARCHES = {"wolfe": g.LS_WOLFE, "batch": g.LS_BATCH}


def listed():
    return [
        # An external optimiser on a small image (6 telescopes, 3 channels): latency and launches count.
        {"name": "evaluate_64", "kind": "evaluate", "width": 64, "tel": 6, "ha": 20, "channels": 3,
         "precision": "split16", "inspect": False},
        # A context as it is created (FP32), an odd width, an array in four channels, every result read back.
        {"name": "evaluate_147_default", "kind": "evaluate", "width": 147, "tel": 8, "ha": 17, "channels": 4,
         "precision": "fp32", "inspect": True},
        # The 256-pixel workload: 12 telescopes, 40 hour angles, 8 channels.
        {"name": "evaluate_256", "kind": "evaluate", "width": 256, "tel": 12, "ha": 40, "channels": 8,
         "precision": "split16", "inspect": False},
        # The largest workload: 20 telescopes, 64 hour angles, 16 channels, 1024 pixels.
        {"name": "evaluate_1024", "kind": "evaluate", "width": 1024, "tel": 20, "ha": 64, "channels": 16,
         "precision": "split16f8", "inspect": False},
        # A sampler's sweep over a small image: the smallest calls there are.
        {"name": "moves_64", "kind": "moves", "width": 64, "tel": 6, "ha": 20, "channels": 3,
         "precision": "split16", "moves": 16},
        # The reference's method (PR+, strong-Wolfe search) on a small image.
        {"name": "cg_64_plain", "kind": "cg", "width": 64, "tel": 6, "ha": 20, "channels": 3,
         "precision": "fp32", "method": 2, "search": "wolfe", "iterations": 2},
        # Projected L-BFGS with the batched search at 256 pixels.
        {"name": "cg_256_lbfgs", "kind": "cg", "width": 256, "tel": 12, "ha": 40, "channels": 8,
         "precision": "split16f8", "method": 4, "search": "batch", "iterations": 2},
        # One iteration of the reference's method on the largest workload.
        {"name": "cg_1024_plain", "kind": "cg", "width": 1024, "tel": 20, "ha": 64, "channels": 16,
         "precision": "split16f8", "method": 2, "search": "wolfe", "iterations": 1},
        # The same with the batched search.
        {"name": "cg_1024_batch", "kind": "cg", "width": 1024, "tel": 20, "ha": 64, "channels": 16,
         "precision": "split16f8", "method": 2, "search": "batch", "iterations": 1},
        # A survey: uneven problems of 64 to 256 pixels in one launch.
        {"name": "many_24", "kind": "many", "count": 24, "precision": "split16", "iterations": 2},
        # The learned start of one held-out problem.
        {"name": "warm_128", "kind": "warm", "width": 128, "tel": 8, "ha": 12, "channels": 3,
         "precision": "split16"},
        # A training step on a batch of 64-pixel problems.
        {"name": "train_64", "kind": "train", "width": 64, "batch": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["evaluate", "evaluate", "evaluate", "moves", "cg", "cg", "cg", "many", "warm", "train"])
    if kind == "many":
        return {"kind": kind, "count": rng.randint(6, 24), "precision": "split16", "iterations": rng.randint(1, 2)}
    if kind == "train":
        return {"kind": kind, "width": 8 * rng.randint(6, 16), "batch": rng.randint(3, 12)}
    c = {"kind": kind, "width": _log_int(rng, 48, 1024), "tel": rng.randint(4, 20), "ha": rng.randint(8, 64),
         "channels": rng.randint(1, 16), "precision": rng.choice(["fp32", "split16", "split16", "tf32x3", "split16f8"])}
    if c["width"] > 600 and c["precision"] in ("fp32", "tf32x3"):  # the slow contractions stay below the largest listed case
        c["precision"] = "split16f8"
    if kind == "warm":
        c.update(width=8 * rng.randint(6, 32), precision="split16")
    elif kind == "moves":
        c.update(moves=rng.randint(4, 24))
    elif kind == "evaluate":
        c.update(inspect=rng.random() < 0.3)
    else:
        c.update(method=rng.choice([0, 1, 2, 2, 3, 4]), search=rng.choice(["wolfe", "batch"]), iterations=1)
    return c


# ------------------------------------------------------------------ problems

def _scene(width, rng):
    """(scene of 1-10 disks, Gaussians and points, field of view in mas)."""
    return warmstart.training_scene(rng, 6.4), 20.48 if width >= 512 else 12.8 if width > 128 else 6.4


def _problem(width, tel, ha, channels, rng):
    """A seeded observation of a scene by a random array, packed as the indexer packs it: V2 points in the order
    (hour angle, baseline, channel), every triangle in every channel, the third side conjugated. A triple amplitude
    below its error is given as its error: the phase weight is 1 / (amplitude x phase error)."""
    scene, field = _scene(width, rng)
    pix = field / width
    diameter = 330.0 if width < 128 else 400.0
    pos = synth.random_array(rng, tel, diameter)
    hour = np.linspace(-3.0, 3.0, ha) * (np.pi / 12.0)
    lam = np.linspace(1.45e-6, 1.85e-6, channels) if channels > 1 else np.array([1.65e-6])
    pairs = list(itertools.combinations(range(tel), 2))
    side = {p: i for i, p in enumerate(pairs)}
    tris = np.array([(side[a, b], side[b, c], side[a, c]) for a, b, c in itertools.combinations(range(tel), 3)])
    base = np.array([pos[b] - pos[a] for a, b in pairs])
    um, vm = synth.baseline_uv(base[None, :, :], hour[:, None])  # [ha, baseline], metres
    u = (um[:, :, None] / lam).astype(np.float32)
    v = (vm[:, :, None] / lam).astype(np.float32)
    V = scene.vis(u.astype(np.float64), v.astype(np.float64))
    v2 = np.abs(V) ** 2
    e2 = 0.01 + 0.05 * v2
    t3 = V[:, tris[:, 0]] * V[:, tris[:, 1]] * np.conj(V[:, tris[:, 2]])
    amp = np.abs(t3)
    ea = 0.01 + 0.05 * amp
    npow, nbis = v2.size, t3.size
    f32 = np.float32
    # index of (hour angle, baseline, channel)
    at = (np.arange(ha)[:, None, None] * len(pairs) + tris.T[:, None, :, None]) * channels + np.arange(channels)
    uvpnt = np.ascontiguousarray(at.reshape(3, nbis).T.astype(np.int64))
    sign = np.tile(np.array([1, 1, -1], np.int16), (nbis, 1))
    uv = np.stack([u.ravel(), v.ravel(), np.full(npow, 5e-8, f32),
                   np.broadcast_to(lam.astype(f32), u.shape).ravel()], axis=1)
    ix = api.Indexed(npow, nbis, npow, (v2 + e2 * rng.standard_normal(v2.shape)).ravel().astype(f32),
                     e2.ravel().astype(f32),
                     np.maximum(amp + ea * rng.standard_normal(amp.shape), ea).ravel().astype(f32),
                     ea.ravel().astype(f32), (np.degrees(np.angle(t3)) + rng.standard_normal(amp.shape)).ravel().astype(f32),
                     np.ones(nbis, f32), uv, uvpnt, sign)
    data, err, phasor, _ = api.init_data(ix)
    model = api.set_model(width, pix, 0, 0.0, 1.0)
    return api.Problem(width, pix, uv, npow, nbis, data, err, phasor, uvpnt, sign, model, 1e-3)


def _case_problem(case, seed):
    return _problem(case["width"], case["tel"], case["ha"], case["channels"], np.random.default_rng([seed, 1]))


def _image(p, seed):
    """The image of a reconstruction under way: the scene, softened, on a floor of half the flux."""
    rng = np.random.default_rng([seed, 1])
    N = p.width
    scene, field = _scene(N, rng)  # the scene that _case_problem observed
    pix = field / N
    y, x = (np.mgrid[0:N, 0:N] - (N - 1) / 2.0) * pix
    img = np.zeros((N, N))
    for c in scene.components:
        dx, dy = x - c.x, y - c.y
        r = np.hypot(dx, dy)
        if c.kind == "gauss":
            co, si = math.cos(c.pa), math.sin(c.pa)
            up, vp = co * dx - si * dy, -si * dx - co * dy  # y runs against v
            one = np.exp(-4.0 * math.log(2.0) * ((up / c.size) ** 2 + (vp / (c.size * c.ratio)) ** 2))
        elif c.kind == "point":
            one = np.exp(-((r / (1.5 * pix)) ** 2))
        else:
            one = np.clip((c.size / 2.0 - r) / pix + 0.5, 0.0, 1.0)
        img += c.flux * one / one.sum()
    img = img * (1.0 + 0.05 * np.random.default_rng([seed, 2]).uniform(-1, 1, img.shape))
    img = 0.5 * img / img.sum() + 0.5 / img.size
    return (img / img.sum()).astype(np.float32).ravel()


def _context(p, case):
    rec = g.Reconstructor(0)
    rec.set_problem(p)
    if case["precision"] != "fp32":  # a new context is on the FP32 path
        rec.set_precision(PRECISIONS[case["precision"]])
    return rec


def _many_problems(case, seed):
    """Widths 64 to 256 in turn, 4-telescope arrays in 8 channels, 500 to 8,000 V2 points (gpair_b200.instances)."""
    rng = np.random.default_rng([seed, 3])
    return [_problem((64, 128, 192, 256)[i % 4], 4, max(10, int(rng.integers(500, 8001)) // 48), 8, rng)
            for i in range(case["count"])]


def _train_batch(case, seed):
    rng = np.random.default_rng([seed, 4])
    B, N = case["batch"], case["width"]
    t = torch.from_numpy(rng.standard_normal((B, warmstart.N_FEATURES, N // 8, N // 8)).astype(np.float32))
    x = torch.nn.functional.interpolate(t, size=(N, N), mode="bicubic")
    x = x / x.abs().amax(dim=(2, 3), keepdim=True)
    target = torch.relu(x[:, 0]) + 1e-3
    target = (target / target.sum(dim=(1, 2), keepdim=True)).reshape(B, N * N)
    return x.contiguous(), target.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, target = _train_batch(case, seed)
        return {"case": case, "net": warmstart.WarmStartNet(seed=seed % 1000), "x": x.cuda(), "target": target.cuda()}
    if kind == "many":
        ps = _many_problems(case, seed)
        recs = [_context(p, case) for p in ps]
        for r in recs:
            r.set_tc_pair(False)
        api.shared_splits(recs)
        starts = [p.start_image() for p in ps]  # the flat prior
        for r, s in zip(recs, starts):
            r.set_image(s)
        return {"case": case, "recs": recs, "starts": starts, "batch": api.Batch(recs, line_search=g.LS_BATCH)}
    p = _case_problem(case, seed)
    state = {"case": case, "problem": p, "rec": _context(p, case)}
    if kind == "warm":
        state["net"] = warmstart.WarmStartNet.load()
    else:
        state["image"] = _image(p, seed)
    if kind == "moves":
        state["moves"] = _moves(case, seed)
    return state


def _moves(case, seed):
    rng = np.random.default_rng([seed, 5])
    N = case["width"]
    return [(int(rng.integers(N)), int(rng.integers(N)), float(np.float32(rng.uniform(0.2, 3.0) / N ** 2)))
            for _ in range(case["moves"])]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        net = state["net"]
        loss = net.train_step(state["x"], state["target"], 1e-4)
        return {"loss": loss, "gradient": net.g, "weights": net.p}
    if kind == "many":
        for r, s in zip(state["recs"], state["starts"]):
            r.set_image(s)
        out = state["batch"].run(case["iterations"])
        return {"J": np.array([o["J"] for o in out], np.float32), "images": [r.get_image() for r in state["recs"]]}
    rec = state["rec"]
    if kind == "warm":
        return warmstart.warm_start(state["net"], rec, state["problem"])
    rec.set_image(state["image"])
    if kind == "cg":
        out = rec.cg(case["iterations"], method=case["method"], line_search=SEARCHES[case["search"]])
        return {"J": out["J"], "chi2": out["chi2"], "image": rec.get_image()}
    chi2, S = rec.criterion()
    if kind == "moves":
        return {"chi2": [rec.update_pixel(x, y, v)[0] for x, y, v in state["moves"]], "visibilities": rec.visibilities()}
    rec.gradient()
    out = {"chi2": chi2, "S": S, "gradient": rec.full_gradient()}
    if case["inspect"]:
        out.update(visibilities=rec.visibilities(), mock=rec.mock())
    return out


# ---------------------------------------------------------------------- work

def _sizes(case):
    """(width, V2 points, triangles) of a problem."""
    per = case["ha"] * case["channels"]
    return case["width"], math.comb(case["tel"], 2) * per, math.comb(case["tel"], 3) * per


def _evaluation(N, npow, nbis, gradient, images=1):
    """Least bytes and operations of `images` objectives, one of them with its gradient: the image and the prior, the
    uv points, the data with their errors and the triangles once, the gradient once; a fast transform to the uv points
    (and back) at 5 N^2 log2(N^2) + 8 x 36 operations per uv point, and the V2, T3 and chi2 arithmetic."""
    b = images * 4 * N * N + 4 * N * N + 8 * npow + 8 * npow + nbis * (12 + 8 + 16)
    f = images * (5 * N * N * math.log2(N * N) + 288 * npow + 8 * npow + 40 * nbis + 10 * N * N)
    if gradient:
        b += 4 * N * N
        f += 5 * N * N * math.log2(N * N) + 288 * npow + 60 * nbis + 10 * N * N
    return b, f


def work(case):
    kind = case["kind"]
    if kind == "train":
        n = case["width"] ** 2
        conv = sum(2 * 9 * cin * cout * n / 4 ** ("1234".index(name[1])) for name, cin, cout in warmstart.LAYERS)
        first = 2 * 9 * warmstart.N_FEATURES * 16 * n  # the first layer passes no gradient back
        params = warmstart.n_params()
        return {"bytes": 4 * case["batch"] * n * (warmstart.N_FEATURES + 1) + 4 * 7 * params,
                "flops": case["batch"] * (3 * conv - first)}
    if kind == "many":
        # the mean of the sizes that are drawn: 30,720 pixels, 4,250 V2 points, 2/3 as many triangles
        b, f = _evaluation(175, 4250, 2833, True)
        bt, ft = _evaluation(175, 4250, 2833, False, 8)
        n = case["count"] * case["iterations"]
        return {"bytes": n * (b + bt), "flops": n * (f + ft)}
    N, npow, nbis = _sizes(case)
    if kind == "warm":
        b, f = _evaluation(N, npow, nbis, True)
        conv = sum(2 * 9 * cin * cout * N * N / 4 ** ("1234".index(name[1])) for name, cin, cout in warmstart.LAYERS)
        return {"bytes": 2.5 * b, "flops": 2.5 * f + conv}
    if kind == "moves":
        b, f = _evaluation(N, npow, nbis, False)
        m = case["moves"]
        return {"bytes": b + m * (24 * npow + 36 * nbis), "flops": f + m * (30 * npow + 40 * nbis)}
    if kind == "evaluate":
        b, f = _evaluation(N, npow, nbis, True)
        if case["inspect"]:
            b += 8 * npow + 4 * (npow + 2 * nbis)
        return {"bytes": b, "flops": f}
    # an iteration has one objective with its gradient and at least one trial (eight at once in a batched search)
    b, f = _evaluation(N, npow, nbis, True)
    bt, ft = _evaluation(N, npow, nbis, False, 8 if case["search"] == "batch" else 1)
    return {"bytes": case["iterations"] * (b + bt), "flops": case["iterations"] * (f + ft)}


# --------------------------------------------------------------------- exact

def _tables(p, sl):
    """Fx[k][x] = e^{+2 pi i s u_k x} and Fy[k][y] = e^{-2 pi i s v_k y} of the uv points in `sl`."""
    s = 2.0 * math.pi * RPMAS * float(np.float32(p.pixellation))
    x = torch.arange(p.width, dtype=torch.float64, device="cuda")
    uv = torch.from_numpy(p.uv[sl, :2].astype(np.float64)).cuda() * s
    ax, ay = uv[:, :1] * x, uv[:, 1:2] * x
    return torch.complex(ax.cos(), ax.sin()), torch.complex(ay.cos(), -ay.sin())


def _chunks(p):
    step = max(1, (1 << 24) // p.width)
    return [slice(i, min(p.nuv, i + step)) for i in range(0, p.nuv, step)]


def _exact_vis(p, image):
    I = torch.from_numpy(image.astype(np.float64)).cuda().reshape(p.width, p.width)
    out = []
    for sl in _chunks(p):
        fx, fy = _tables(p, sl)
        out.append(((fx @ I.T.to(torch.complex128)) * fy).sum(1))
    return torch.cat(out) / I.sum()


class _Data:
    """A problem's data arrays in 64 bits on the device."""

    def __init__(self, p):
        d = lambda a, t=torch.float64: torch.from_numpy(np.ascontiguousarray(a)).cuda().to(t)  # noqa: E731
        self.p = p
        self.data, self.w = d(p.data), d(p.data_err)
        self.phasor = d(p.phasor, torch.complex128)
        self.at, self.conj = d(p.uvpnt, torch.int64), d(p.sign) < 0

    def sides(self, V):
        s = V[self.at]
        return torch.where(self.conj, s.conj(), s)

    def mock(self, V):
        p = self.p
        s = self.sides(V)
        t3 = s[:, 0] * s[:, 1] * s[:, 2] * self.phasor
        m = torch.empty(p.npow + 2 * p.nbis, dtype=torch.float64, device="cuda")
        m[:p.npow] = V[:p.npow].abs() ** 2
        m[p.npow::2], m[p.npow + 1::2] = t3.real, t3.imag
        return m

    def chi2(self, V):
        return float((((self.mock(V) - self.data) * self.w) ** 2).sum())

    def weights(self, V, flux):
        """c_k of d chi2 / dI = Re sum_k c_k (Fx Fy - V_k); the T3 imaginary part as the mock value alone."""
        p = self.p
        m, s = self.mock(V), self.sides(V)
        c = torch.zeros(p.nuv, dtype=torch.complex128, device="cuda")
        w2 = self.w ** 2
        c[:p.npow] = 4.0 * w2[:p.npow] * (m[:p.npow] - self.data[:p.npow]) * V[:p.npow].conj() / flux
        re, im = slice(p.npow, None, 2), slice(p.npow + 1, None, 2)
        gt = torch.complex(2.0 * w2[re] * (m[re] - self.data[re]), -2.0 * w2[im] * m[im]) * self.phasor / flux
        for j in range(3):
            b = gt * s[:, (j + 1) % 3] * s[:, (j + 2) % 3]
            c.index_add_(0, self.at[:, j], torch.where(self.conj[:, j], b.conj(), b))
        return c


def _exact_adjoint(p, c):
    G = torch.zeros(p.width, p.width, dtype=torch.float64, device="cuda")
    for sl in _chunks(p):
        fx, fy = _tables(p, sl)
        G += ((fy * c[sl, None]).T @ fx).real
    return G.reshape(-1)


def _exact_gradient(p, image, alpha):
    """(chi2, S, data gradient, full gradient, V) of an image."""
    I = torch.from_numpy(image.astype(np.float64)).cuda()
    m = torch.from_numpy(p.model.astype(np.float64)).cuda()
    V, d = _exact_vis(p, image), _Data(p)
    S = float((I - m - I * torch.log(I / m)).sum())
    c = d.weights(V, float(I.sum()))
    data = _exact_adjoint(p, c) - (c * V).real.sum()
    return d.chi2(V), S, data, data + alpha * torch.log(I / m), V


def _network(params, x):
    """The warm-start network in 64 bits on bf16-rounded weights: unit-flux images."""
    conv, up, pool = torch.nn.functional.conv2d, torch.nn.functional.interpolate, torch.nn.functional.avg_pool2d

    def layer(name, h, skip=None):
        y = conv(h, params[name + ".w"], params[name + ".b"], padding=1)
        return torch.relu(y if skip is None else y + skip)

    def twice(h):
        return up(h, scale_factor=2, mode="nearest")

    e1 = layer("e1b", layer("e1a", x))
    e2 = layer("e2b", layer("e2a", pool(e1, 2)))
    e3 = layer("e3b", layer("e3a", pool(e2, 2)))
    e4 = layer("e4b", layer("e4a", pool(e3, 2)))
    d3 = layer("d3b", layer("d3a", twice(e4), e3))
    d2 = layer("d2b", layer("d2a", twice(d3), e2))
    d1 = layer("d1b", layer("d1a", twice(d2), e1))
    z = (d1 * params["head.w"].view(1, -1, 1, 1)).sum(1) + params["head.b"]
    out = torch.nn.functional.softplus(z, threshold=40.0).flatten(1)
    return out / out.sum(1, keepdim=True)


def _parameters(flat):
    shapes = {name: (cout, cin, 3, 3) for name, cin, cout in warmstart.LAYERS}
    out = {}
    for name, off, n in warmstart.param_layout():
        t = torch.from_numpy(flat[off:off + n].copy()).cuda()
        if name.endswith(".w") and name[:-2] in shapes:
            t = t.to(torch.bfloat16).reshape(shapes[name[:-2]])
        out[name] = t.to(torch.float64).requires_grad_(True)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, target = (t.cuda().to(torch.float64) for t in _train_batch(case, seed))
        flat = warmstart.init_params(seed % 1000)
        params = _parameters(flat)
        out = _network(params, x)
        loss = ((out - target) ** 2).sum(1) / (target ** 2).sum(1)
        loss.mean().backward()
        grad = torch.cat([params[name].grad.reshape(-1) for name, _, _ in warmstart.param_layout()])
        m, v = 0.1 * grad, 0.001 * grad ** 2
        step = 1e-4 * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8)
        return {"loss": loss.detach(), "gradient": grad, "weights": torch.from_numpy(flat).cuda().double() - step}
    if kind in ("many", "cg"):
        return None
    p = _case_problem(case, seed)
    if kind == "warm":
        flat_start = p.start_image()
        _, _, dirty, _, _ = _exact_gradient(p, flat_start, 0.0)
        N = p.width
        u, v = p.uv[:, 0].astype(np.float64), p.uv[:, 1].astype(np.float64)
        w = np.zeros(p.nuv, np.complex128)
        w[:p.npow] = np.maximum(p.data[:p.npow].astype(np.float64), 0.0)
        w *= np.exp(-2j * np.pi * RPMAS * p.pixellation * (u - v) * (N // 2))
        v2map = _exact_adjoint(p, torch.from_numpy(w.astype(np.complex64).astype(np.complex128)).cuda())
        y, x = np.mgrid[0:N, 0:N].astype(np.float64)
        blob = np.exp(-((x - N // 2) ** 2 + (y - N // 2) ** 2) / (2 * (N / 4.0 / 2.3548) ** 2))
        flux = float(np.sum(flat_start, dtype=np.float64))
        _, _, probe, _, _ = _exact_gradient(p, np.maximum(blob / blob.sum() * flux, 1e-8).astype(np.float32).ravel(), 0.0)
        density = torch.from_numpy(warmstart.uv_density(p).astype(np.float64)).cuda().reshape(-1)
        feats = torch.stack([t / t.abs().max() for t in (-dirty, v2map, density, -probe)]).reshape(1, -1, N, N)
        with np.load(warmstart.DEFAULT_WEIGHTS) as z:
            params = _parameters(z["params"])
        return torch.clamp(_network(params, feats)[0].detach() * flux, min=1e-8)
    image = _image(p, seed)
    if kind == "moves":
        d, I, chi2 = _Data(p), image.copy(), []
        V, N = _exact_vis(p, image), p.width
        flux = float(np.sum(I, dtype=np.float64))
        fx, fy = _tables(p, slice(0, p.nuv))
        for x, y, value in _moves(case, seed):
            change = float(np.float32(value)) - float(I[y * N + x])
            V = (flux * V + change * fx[:, x] * fy[:, y]) / (flux + change)
            flux += change
            I[y * N + x] = value
            chi2.append(d.chi2(V))
        return {"chi2": chi2, "visibilities": V}
    chi2, S, _, full, V = _exact_gradient(p, image, p.alpha)
    out = {"chi2": chi2, "S": S, "gradient": full}
    if case["inspect"]:
        out.update(visibilities=V, mock=_Data(p).mock(V))
    return out
