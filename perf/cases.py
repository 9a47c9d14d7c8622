"""The workloads whose speed is tracked: what a program that uses g2s_b200 has it do, through the public entry points.

Kinds of case
  pattern  one query of the per-node device interface (Worker.pattern_kbest), the call that a path loop outside the
           library makes at each node
  batch    one batch of calibration queries (Worker.pattern_kbest_verbatim): weighted terms, exclusion radius
  qs       one whole simulation by the one-call API (g2s_b200.qs): host arrays in, simulation and index image out
  sample   the teacher-forced draw of a sample of path nodes of a prepared Simulation (large 3-D images, where the whole
           simulation takes minutes)
  jobs     several prepared simulations in one call (run_jobs)
  encoder  forward, loss and gradient of the neighbourhood encoder (Encoder.loss_grad)

Inputs are seeded synthetic images of the distributions the package's own generators give: Gaussian random fields with
an exponential covariance (made on the GPU, where the large ones take milliseconds), binary sinuous channels, and a field
stacked with its indicator at the 0.7 quantile.
"""
import math

import numpy as np
import torch

import g2s_b200 as g2s
from g2s_b200 import synthetic

SQLIN, EQ = g2s.QSK_OP_SQLIN, g2s.QSK_OP_EQ


def listed():
    return [
        # the smallest call: one node of a small 2-D image, launch and host latency
        dict(name="pattern grf 100x83 n20", kind="pattern", image="grf", ti="100x83", n=20, k=1),
        # one node of a 3-D reservoir-sized image, as a path loop outside the library asks for it
        dict(name="pattern grf3d 120x150x180 n60", kind="pattern", image="grf", ti="120x150x180", n=60, k=2),
        # one iteration's queries of a parameter calibration
        dict(name="batch channels 250 x256", kind="batch", image="channels", ti="250x250", queries=256, n=80, k=1),
        # a small whole simulation of odd size: few nodes a level, latency of the level chain
        dict(name="qs channels 101x90 plain", kind="qs", image="channels", ti="101x90", grid="67x61", n=20, k=1.5,
             tensor="plain"),
        # a continuous realisation, exact path
        dict(name="qs grf 200 plain", kind="qs", image="grf", ti="200x200", grid="200x200", n=50, k=1.2, tensor="plain"),
        # the same on the tensor cores
        dict(name="qs grf 200 bf16", kind="qs", image="grf", ti="200x200", grid="200x200", n=50, k=1.2, tensor="bf16"),
        # a categorical realisation four times the training image, exact path and tensor cores (tuned prefix)
        dict(name="qs channels 500 plain", kind="qs", image="channels", ti="250x250", grid="500x500", n=80, k=1.5,
             tensor="plain"),
        dict(name="qs channels 500 bf16", kind="qs", image="channels", ti="250x250", grid="500x500", n=80, k=1.5,
             tensor="bf16", prefix=384),
        # nodes of a 3-D continuous simulation on the FP8 form, and of a 3-D bivariate one on the exact path
        dict(name="sample grf3d fp8 x8000", kind="sample", image="grf", ti="120x150x180", grid="80x100x120", n=60, k=1.2,
             nodes=8000, tensor="fp8"),
        dict(name="sample bivar3d plain x512", kind="sample", image="bivariate", ti="128x128x128", grid="64x96x96", n=64,
             k=1.5, nodes=512, tensor="plain"),
        # several realisations of different kinds in one call
        dict(name="jobs x4", kind="jobs", jobs=4, ti=256, grid=128, n=40, tensor="bf16"),
        # a training step's gradient for a batch of 1024 pairs
        dict(name="encoder loss_grad 1024", kind="encoder", nvar=2, pairs=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pattern", "pattern", "batch", "qs", "qs", "qs", "sample", "sample", "jobs", "encoder"])
    if kind == "pattern":
        if rng.random() < 0.5:
            ti = "%dx%d" % (_log(rng, 40, 500), _log(rng, 40, 500))
        else:
            ti = "%dx%dx%d" % (_log(rng, 20, 120), _log(rng, 24, 150), _log(rng, 24, 180))
        return dict(kind=kind, image=rng.choice(["grf", "channels", "bivariate"]) if ti.count("x") == 1 else
                    rng.choice(["grf", "bivariate"]), ti=ti, n=_log(rng, 8, 60), k=rng.randint(1, 4))
    if kind == "batch":
        return dict(kind=kind, image=rng.choice(["channels", "grf"]), ti="%dx%d" % (_log(rng, 80, 250), _log(rng, 80, 250)),
                    queries=rng.randint(40, 256), n=_log(rng, 8, 80), k=rng.randint(1, 2))
    if kind == "qs":
        tensor = rng.choice(["plain", "plain", "bf16"])
        c = dict(kind=kind, image=rng.choice(["grf", "channels", "bivariate"]),
                 ti="%dx%d" % (_log(rng, 64, 250), _log(rng, 64, 250)),
                 grid="%dx%d" % (_log(rng, 40, 200), _log(rng, 40, 200)), n=_log(rng, 10, 60),
                 k=rng.choice([1.0, 1.2, 1.5, 2.5]), tensor=tensor)
        return c
    if kind == "sample":
        tensor = rng.choice(["plain", "fp8", "bf16"])
        return dict(kind=kind, image=rng.choice(["grf", "bivariate"]),
                    ti="%dx%dx%d" % (_log(rng, 40, 96), _log(rng, 48, 110), _log(rng, 48, 128)),
                    grid="%dx%dx%d" % (_log(rng, 32, 64), _log(rng, 40, 96), _log(rng, 40, 96)), n=_log(rng, 16, 64),
                    k=rng.choice([1.0, 1.2, 1.5]), nodes=_log(rng, 200, 512 if tensor == "plain" else 4000), tensor=tensor)
    if kind == "jobs":
        return dict(kind=kind, jobs=rng.randint(2, 4), ti=_log(rng, 100, 256), grid=_log(rng, 48, 128),
                    n=_log(rng, 16, 40), tensor=rng.choice(["plain", "bf16"]))
    return dict(kind=kind, nvar=rng.randint(1, 3), pairs=_log(rng, 64, 1024))


# ---- inputs ---------------------------------------------------------------------------------------------------------

def _dims(text):
    """'AxB[xC]' in numpy order (slowest first)."""
    return tuple(int(v) for v in text.split("x"))


def _grf(shape, seed):
    """Gaussian random field, exponential covariance, range about a sixteenth of the longest side (the vertical one a
    quarter of that in 3-D), filtered on a periodic grid and cropped; mean 0, variance 1."""
    r = max(3.0, max(shape) / 16.0)
    ranges = [r] * len(shape)
    if len(shape) == 3:
        ranges[0] = r / 4.0
    dev = torch.device("cuda", 0)
    big = [s + int(6 * q) for s, q in zip(shape, ranges)]
    big = [b + b % 2 for b in big]
    h2 = torch.zeros(big, dtype=torch.float64, device=dev)
    for d, (b, q) in enumerate(zip(big, ranges)):
        i = torch.arange(b, device=dev, dtype=torch.float64)
        a = torch.minimum(i, b - i) / q
        view = [1] * len(big)
        view[d] = b
        h2 += (a * a).view(view)
    spec = torch.fft.rfftn(torch.exp(-torch.sqrt(h2))).real.clamp_(min=0.0).sqrt_()
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    noise = torch.randn(big, generator=gen, dtype=torch.float64, device=dev)
    f = torch.fft.irfftn(torch.fft.rfftn(noise) * spec, s=big)
    f = f[tuple(slice(0, s) for s in shape)]
    f = (f - f.mean()) / f.std()
    return f.to(torch.float32).cpu().numpy()


def _image(name, shape, seed):
    """(array, variable types)"""
    if name == "channels":
        return synthetic.channels2d(shape, n_channels=max(4, shape[0] * shape[1] // 3000), seed=int(seed)), [1]
    if name == "bivariate":
        return synthetic.bivariate(_grf(shape, seed)), [0, 1]
    return _grf(shape, seed), [0]


def _pattern(rng, tpl, wtab, ti, types, n, density):
    """A neighbourhood taken from the training image itself: a random cell, its template neighbours kept with the given
    probability until there are n (as a calibration sample or a node of a partly simulated grid has them).  Returns
    (offsets, terms, flat cell)."""
    nvar = len(types)
    space = ti.shape if nvar == 1 else ti.shape[:-1]
    src = np.array(space[::-1])
    c = np.array([int(rng.integers(0, s)) for s in src])
    keep = np.flatnonzero(rng.random(len(tpl)) < density)
    p = c + tpl[keep]
    keep = keep[np.all((p >= 0) & (p < src), axis=1)]
    keep = keep[np.any(tpl[keep] != 0, axis=1)][:n]
    offs = tpl[keep]
    vals = ti.reshape(space + (nvar,))[tuple((c + offs).T[::-1])]
    terms = []
    for j in range(len(offs)):
        w = np.float32(wtab[keep[j]])
        for v, t in enumerate(types):
            x = vals[j, v]
            if t == 0:
                terms.append((j, v, SQLIN, -float(w), float(np.float32(2.0) * (w * x))))
            else:
                terms.append((j, v, EQ, float(w), float(x)))
    flat = 0
    for d in reversed(range(len(src))):
        flat = flat * int(src[d]) + int(c[d])
    return np.ascontiguousarray(offs, np.int32), terms, flat


def _query(case, seed):
    """Image, types, patterns, seeds, cells and radius of a pattern or batch case."""
    shape = _dims(case["ti"])
    ti, types = _image(case["image"], shape, seed)
    rng = np.random.default_rng(int(seed) + 77)
    box = [min(s // 2 + 1, 61 if len(shape) == 2 else 25) for s in reversed(shape)]
    tpl, _ = g2s.search_template(box)
    batch = case["kind"] == "batch"
    # a calibration weighs the neighbours with a Gaussian kernel; a path loop's default kernel is uniform
    wtab = np.exp(-(tpl.astype(np.float64) ** 2).sum(1) / 200.0).astype(np.float32) if batch else \
        np.ones(len(tpl), np.float32)
    count = case["queries"] if batch else 1
    pats, cells = [], []
    for q in range(count):
        density = [0.0625, 0.125, 0.25, 0.5][q % 4] if batch else 0.25
        o, t, c = _pattern(rng, tpl, wtab, ti, types, case["n"], density)
        pats.append((o, t))
        cells.append(c)
    seeds = rng.random(count).astype(np.float32)
    radius = (np.prod(shape) * 0.005) ** (1.0 / len(shape))
    return ti, types, pats, seeds, np.array(cells, np.uint32), np.full(count, radius, np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("pattern", "batch"):
        ti, types, pats, seeds, cells, radii = _query(case, seed)
        worker = g2s.Worker(g2s.TrainingImage(ti, types))
        return dict(kind=kind, worker=worker, pats=pats, seeds=seeds, cells=cells, radii=radii, k=case["k"])
    if kind == "qs":
        ti, types = _image(case["image"], _dims(case["ti"]), seed)
        grid = _dims(case["grid"]) + ((len(types),) if len(types) > 1 else ())
        tensor = None if case["tensor"] == "plain" else case["tensor"]
        if tensor and case.get("prefix"):
            tensor = {"mode": tensor, "prefix": case["prefix"]}
        return dict(kind=kind, ti=ti, types=types, di=np.full(grid, np.nan, np.float32), n=case["n"], k=case["k"],
                    seed=100 + int(seed) % 1000, tensor=tensor)
    if kind == "sample":
        ti, types = _image(case["image"], _dims(case["ti"]), seed)
        done, _ = _image(case["image"], _dims(case["grid"]), int(seed) + 1000003)
        sim = g2s.Simulation(ti, np.full(done.shape, np.nan, np.float32), types, n=case["n"], k=case["k"],
                             seed=100 + int(seed) % 1000)
        if case["tensor"] != "plain":
            sim.set_tensor(case["tensor"], audit=0.01)
        cells = int(np.prod(_dims(case["grid"])))
        nodes = (np.arange(case["nodes"], dtype=np.int64) * cells // case["nodes"]).astype(np.int32)
        return dict(kind=kind, sim=sim, done=done, nodes=nodes)
    if kind == "jobs":
        sims = []
        for j in range(case["jobs"]):
            image = ["grf", "channels", "bivariate"][j % 3]
            side = case["ti"]
            ti, types = _image(image, (side, side), int(seed) + j)
            edge = max(16, int(case["grid"] / 2 ** (j / 2.0)))
            grid = (edge, edge) + ((len(types),) if len(types) > 1 else ())
            sim = g2s.Simulation(ti, np.full(grid, np.nan, np.float32), types, n=case["n"], k=1.2,
                                 seed=(100 + int(seed) + j) % 100000)
            if case["tensor"] != "plain":
                sim.set_tensor(case["tensor"], audit=0.01)
            sims.append(sim)
        return dict(kind=kind, sims=sims)
    enc = g2s.Encoder(nvar=case["nvar"], seed=int(seed) % 100000)
    rng = np.random.default_rng(int(seed))
    xq = rng.standard_normal((case["pairs"], enc.input_dim), dtype=np.float32)
    xp = xq + np.float32(0.5) * rng.standard_normal(xq.shape, dtype=np.float32)
    return dict(kind=kind, enc=enc, xq=xq, xp=xp)


def run(state):
    kind = state["kind"]
    if kind == "pattern":
        offs, terms = state["pats"][0]
        sc, ix, mn = state["worker"].pattern_kbest(offs, terms, state["k"], float(state["seeds"][0]))
        return dict(scores=sc, index=ix, min_offset=mn)
    if kind == "batch":
        sc, ix, mn = state["worker"].pattern_kbest_verbatim(state["pats"], state["k"], state["seeds"], state["cells"],
                                                            state["radii"])
        return dict(scores=sc, index=ix, min_offset=mn)
    if kind == "qs":
        out, idx = g2s.qs(state["ti"], state["di"], state["types"], k=state["k"], n=state["n"], s=state["seed"],
                          tensor=state["tensor"])
        return dict(simulation=out, index=idx)
    if kind == "sample":
        sim = state["sim"]
        sim.run_teacher_nodes(state["done"], state["nodes"])
        # the draws of the sampled nodes; the other path nodes are not simulated by this call
        return dict(cells=sim.read()[2][state["nodes"]])
    if kind == "jobs":
        g2s.run_jobs(state["sims"])
        return [list(sim.read()[:2]) for sim in state["sims"]]
    loss, grad = state["enc"].loss_grad(state["xq"], state["xp"], tau=0.5)
    return dict(loss=loss, grad=grad)


# ---- what the path cannot do without --------------------------------------------------------------------------------

def _map_flops(nodes, n, cells, image):
    """Two operations for each layer of a neighbour at each position: squared and linear for a continuous variable, one
    indicator for a binary one."""
    return 2.0 * nodes * n * cells * {"grf": 2, "channels": 1, "bivariate": 3}[image]


def work(case):
    kind = case["kind"]
    if kind == "encoder":
        d0, b = 64 * (case["nvar"] + 4), case["pairs"]
        mats = d0 * 256 + 2 * 256 * 256 + 256 * 64
        params = d0 * 256 + 2 * 256 * 256 + 3 * 256 + 2 * (256 * 64 + 64)
        return {"bytes": 4.0 * (2 * b * d0 + 2 * params), "flops": 6.0 * 2 * b * mats + 6.0 * b * b * 64}
    if kind == "jobs":
        flops = nbytes = 0.0
        for j in range(case["jobs"]):
            image = ["grf", "channels", "bivariate"][j % 3]
            nv = 2 if image == "bivariate" else 1
            edge = max(16, int(case["grid"] / 2 ** (j / 2.0)))
            flops += _map_flops(edge * edge, case["n"], case["ti"] ** 2, image)
            nbytes += 4.0 * (nv * case["ti"] ** 2 + (nv + 1) * edge * edge)
        return {"bytes": nbytes, "flops": flops}
    cells = float(np.prod(_dims(case["ti"])))
    nv = 2 if case["image"] == "bivariate" else 1
    if kind in ("pattern", "batch"):
        q = case.get("queries", 1)
        return {"bytes": 4.0 * nv * cells + q * (case["n"] * nv * 20.0 + 8.0 * case["k"]),
                "flops": _map_flops(q, case["n"], cells, case["image"])}
    grid = float(np.prod(_dims(case["grid"])))
    nodes = grid if kind == "qs" else case["nodes"]
    out = (2 * nv + 1) * grid if kind == "qs" else nv * grid + nodes
    return {"bytes": 4.0 * (nv * cells + out), "flops": _map_flops(nodes, case["n"], cells, case["image"])}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------

def _exact_pattern(case, seed):
    """The k best scores of the pattern over the positions whose neighbourhood lies inside the image."""
    ti, types, pats, _, _, _ = _query(case, seed)
    offs, terms = pats[0]
    nd = offs.shape[1]
    t = torch.from_numpy(ti).to("cuda", torch.float64).reshape(_dims(case["ti"]) + (len(types),))
    lo = np.minimum(offs.min(0), 0) if len(offs) else np.zeros(nd, int)
    hi = np.maximum(offs.max(0), 0) if len(offs) else np.zeros(nd, int)
    src = t.shape[:nd][::-1]
    if any(src[d] - (hi[d] - lo[d]) < 1 for d in range(nd)):
        return None
    score = None
    for j, v, op, a, b in terms:
        view = tuple(slice(int(offs[j][d] - lo[d]), int(offs[j][d] - lo[d] + src[d] - (hi[d] - lo[d])))
                     for d in reversed(range(nd)))
        x = t[view + (v,)]
        s = a * x * x + b * x if op == SQLIN else a * (x == b).to(torch.float64)
        score = s if score is None else score + s
    if score is None or score.numel() < case["k"]:
        return None
    return dict(scores=torch.topk(score.reshape(-1), case["k"]).values.cpu().numpy(), index=None, min_offset=None)


def _exact_encoder(case, seed):
    s = prepare(case, seed)
    d0 = s["enc"].input_dim
    w = torch.from_numpy(s["enc"].weights()).to("cuda", torch.float64)
    shapes = [(256, d0), (256,), (256, 256), (256,), (256, 256), (256,), (64, 256), (64,), (64, 256), (64,)]
    parts, at = [], 0
    for sh in shapes:
        n = int(np.prod(sh))
        parts.append(w[at:at + n].reshape(sh).clone().requires_grad_(True))
        at += n

    def trunk(x):
        h = torch.from_numpy(x).to("cuda", torch.float64)
        for i in (0, 2, 4):
            h = torch.nn.functional.gelu(h @ parts[i].T + parts[i + 1], approximate="tanh")
        return h

    q = trunk(s["xq"]) @ parts[6].T + parts[7]
    p = trunk(s["xp"]) @ parts[8].T + parts[9]
    logits = q @ p.T / 0.5
    label = torch.arange(logits.shape[0], device="cuda")
    loss = 0.5 * (torch.nn.functional.cross_entropy(logits, label) + torch.nn.functional.cross_entropy(logits.T, label))
    grads = torch.autograd.grad(loss, parts)
    return dict(loss=float(loss), grad=torch.cat([x.reshape(-1) for x in grads]).cpu().numpy())


def exact(case, seed):
    if case["kind"] == "pattern":
        return _exact_pattern(case, seed)
    if case["kind"] == "encoder":
        return _exact_encoder(case, seed)
    # batches score excluded positions apart; simulations return copies of training-image values and whole numbers
    return None
