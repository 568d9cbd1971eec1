"""The work that users of lensed_gb300 have it do, as timed cases.

A lens modeller creates a context for one observed image (or one for a batch
of systems) and evaluates candidate parameter vectors: one at a time from a
host sampler, or in batches.  The sampler of the library does the same from
inside; the best candidate is then written out as images.  The models, sizes,
PSFs and quadrature rules are those of the workloads of this repository
(``lensed_gb300/workloads.py``) and of its tests, or lie between them.

``exact`` is a float64 restatement of the model (Tessore, Bellagamba &
Metcalf 2016 and the papers named at the lens profiles) in plain torch.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import lensed_gb300 as lg

# object id -> plugin, in list order: the models of the workloads
MODELS = {
    # galaxy-scale lens, one source (the sampler's workload)
    "sie": (("lens", "sie"), ("src", "sersic"), ("sky", "sky")),
    # the headline model: shear, bulge and disk
    "shear": (("lens", "sie_plus_shear"), ("bulge", "sersic"), ("disk", "exponential"), ("sky", "sky")),
    # power-law lens (the multi-system workload)
    "epl": (("lens", "epl_plus_shear"), ("src", "sersic"), ("sky", "sky")),
    # three lenses, three sources (the large workload)
    "group": (("lens", "epl_plus_shear"), ("sat", "nsie"), ("pert", "point_mass"), ("src1", "sersic"),
              ("src2", "sersic"), ("clump", "gauss"), ("sky", "sky")),
    # cored lens with a de Vaucouleurs source (the plugins the others leave out)
    "cored": (("lens", "nsie"), ("src", "devauc"), ("sky", "sky")),
}
FLAGS = {"exact": 0, "fast": lg.LG_FLAG_FAST_MATH}

# source-level FP32 operations of one ray through a plugin (an elementary
# function counts as one), and of the quadrature sum and lens plane
RAY_FLOPS = {"sie": 26, "sie_plus_shear": 34, "nsie": 30, "point_mass": 9, "epl_plus_shear": 180, "sersic": 17,
             "exponential": 15, "devauc": 16, "gauss": 16, "sky": 6}
RAY_OVERHEAD = 12
RULE_POINTS = {"sub2": 4, "sub3": 9, "sub5": 25, "g3k7": 49}


def listed():
    image = dict(model="shear", width=256, height=256, psf_w=25, psf_h=25, rule="sub5", mode="exact")
    return [
        # a host sampler (MultiNest's role) asking for one point at a time
        # through the reference's callback: latency
        dict(image, name="callback", kind="callback", batch=1),
        # a few walkers at a time on a small cut-out of odd sides, even PSF
        dict(name="walkers", kind="host", model="cored", width=101, height=77, psf_w=12, psf_h=12, rule="sub3",
             batch=7, mode="exact"),
        # the sampler's own batches: unit-cube points, prior transform on the GPU, no PSF
        dict(name="cube_batch", kind="cube", model="sie", width=128, height=128, psf_w=0, psf_h=0, rule="sub3",
             batch=1024, mode="exact"),
        # the headline workload, default arithmetic and the fast mode
        dict(image, name="headline", kind="device", batch=1024),
        dict(image, name="headline_fast", kind="device", batch=1024, mode="fast"),
        # a survey's cut-outs of uneven size and PSF in one call, ragged counts
        dict(name="systems", kind="systems", model="epl", width=512, height=512, psf_w=31, psf_h=31, rule="g3k7",
             batch=40, count=6, mode="exact"),
        dict(name="systems_fast", kind="systems", model="epl", width=512, height=512, psf_w=31, psf_h=31,
             rule="g3k7", batch=40, count=6, mode="fast"),
        # a cluster-scale field: large image and PSF, many objects
        dict(name="large", kind="device", model="group", width=1024, height=1024, psf_w=41, psf_h=41, rule="g3k7",
             batch=24, mode="exact"),
        # an ordinary odd-sized cut-out, ragged batch, host buffers
        dict(name="ragged", kind="host", model="epl", width=333, height=211, psf_w=17, psf_h=21, rule="sub3",
             batch=131, mode="exact"),
        # the result images of the best candidate
        dict(name="layers", kind="layers", model="shear", width=601, height=479, psf_w=25, psf_h=25, rule="g3k7",
             batch=1, mode="exact"),
        # a whole (short) sampler run: proposals, prior transform, likelihood, evidence
        dict(name="sampler", kind="sampler", model="sie", width=96, height=96, psf_w=0, psf_h=0, rule="sub3",
             batch=512, nlive=400, maxiter=1500, mode="exact"),
        # training the learned proposal on a sampler's live points
        dict(name="training", kind="training", points=1000, dims=13, epochs=25),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: kinds by how often they are used, sizes over their range."""
    kind = rng.choice(["device", "device", "host", "host", "cube", "systems", "callback", "layers", "sampler"])
    mode = rng.choice(["exact", "exact", "exact", "fast"])
    model = rng.choice(sorted(MODELS))
    case = dict(kind=kind, model=model, mode=mode, rule=rng.choice(sorted(RULE_POINTS)))
    case["width"], case["height"] = _log_int(rng, 48, 900), _log_int(rng, 48, 900)
    case["psf_w"] = case["psf_h"] = 0
    if rng.random() < 0.75:
        case["psf_w"], case["psf_h"] = rng.randint(5, 41), rng.randint(5, 41)
    case["batch"] = 1
    if kind in ("device", "host", "cube"):
        case["batch"] = _log_int(rng, 1, 1024)
    elif kind == "systems":
        case.update(batch=_log_int(rng, 2, 64), count=rng.randint(2, 6), model="epl",
                    width=_log_int(rng, 64, 512), psf_w=rng.randrange(15, 32, 2))
        case["height"], case["psf_h"] = case["width"], case["psf_w"]
    elif kind == "sampler":
        case.update(model="sie", rule="sub3", psf_w=0, psf_h=0, width=rng.randint(48, 128), batch=512,
                    nlive=rng.randint(200, 500), maxiter=rng.randint(300, 1500), mode="exact")
        case["height"] = case["width"]
    # no dearer than the largest listed case
    limit = _flops(next(c for c in listed() if c["name"] == "headline"))
    while case["batch"] > 1 and _flops(case) > limit:
        case["batch"] = max(1, case["batch"] // 2 + rng.randint(0, 1) * (case["batch"] > 8))
    return case


# ------------------------------------------------------------------ inputs
def _psf(w, h, rng):
    """Gaussian core with wings, slightly elliptical, normalised (float32)."""
    fwhm = rng.uniform(1.8, 3.5)
    y, x = np.mgrid[0:h, 0:w].astype(np.float64)
    x, y = x - (w - 1) / 2, (y - (h - 1) / 2) * rng.uniform(0.9, 1.1)
    s = fwhm / 2.3548200450309493
    r2 = x * x + y * y + 0.1 * x * y
    p = 0.9 * np.exp(-0.5 * r2 / s ** 2) / s ** 2 + 0.1 * np.exp(-0.5 * r2 / (4 * s) ** 2) / (4 * s) ** 2
    return (p / p.sum()).astype(np.float32)


def _mag(snr, re, n, q, sky=10.0):
    """Magnitude of a Sersic profile whose centre has a signal-to-noise ratio over the sky."""
    b = 2 * n - 1 / 3 + 4 / (405 * n)
    log0 = 2 * n * math.log(b) - math.log(math.pi) - 2 * math.log(re) - math.lgamma(2 * n + 1)
    peak = math.exp(log0 - math.exp(math.log(b) - math.log(re) / n + 0.5 / n * math.log(0.25 / q)))
    return -2.5 * math.log10((snr * math.sqrt(sky) + snr * snr / 2) / peak)


def _truth(model, width, height, rng):
    """True parameters and half-widths of the prior box (0: fixed), in object order."""
    u = rng.uniform
    side = min(width, height)
    er = side / 12.8 if side > 128 else side / 6.4
    cx, cy = (width + 1) / 2 + u(-1, 1), (height + 1) / 2 + u(-1, 1)
    sx, sy = cx + u(-0.2, 0.2) * er, cy + u(-0.2, 0.2) * er
    n, re, q = u(1, 4), er * u(0.1, 0.4), u(0.5, 0.9)
    mag = _mag(30.0, re, n, q)
    lens_q, pa = u(0.6, 0.9), u(20, 160)
    sersic = ([sx, sy, re, mag, n, q, u(20, 160)], [0.1 * er, 0.1 * er, re / 5, 0.5, 0.5, 0.08, 20])
    truth = {
        "sie": ([cx, cy, er, lens_q, pa], [1, 1, er / 10, 0.08, 20]),
        "sie_plus_shear": ([cx, cy, er, lens_q, pa, u(0, 0.09), u(0, 0.03)], [1, 1, er / 10, 0.08, 20, 0.03, 0.03]),
        "epl_plus_shear": ([cx, cy, er, u(0.8, 1.2), lens_q, pa, u(-0.05, 0.05), u(-0.05, 0.05)],
                           [1, 1, er / 10, 0.1, 0.08, 20, 0.02, 0.02]),
        "nsie": ([cx, cy, er, u(0.3, 1.0), lens_q, pa], [1, 1, er / 10, 0.2, 0.08, 20]),
        "point_mass": ([cx - 0.9 * er, cy + 0.8 * er, 0.06 * er + 0.5], [0.5, 0.5, 0.2]),
        "sersic": sersic,
        "exponential": ([sx, sy, er * u(0.15, 0.4), mag + 0.5, u(0.4, 0.9), u(20, 160)], [1, 1, er / 20, 0.5, 0.08, 20]),
        "devauc": ([sx, sy, er * u(0.3, 0.6), mag - 1, u(0.5, 0.9), u(20, 160)], [1, 1, er / 20, 0.5, 0.08, 20]),
        "gauss": ([cx + 0.1 * er, cy + 0.3 * er, 0.1 * er + 0.5, mag + 2, u(0.5, 0.9), u(20, 160)],
                  [0.5, 0.5, 0.2, 0.3, 0.08, 10]),
        "sky": ([10.0, -0.0, -0.0], [1, 0, 0]),
    }
    t, h = [], []
    for i, (_, plugin) in enumerate(MODELS[model]):
        a, b = truth[plugin]
        if plugin == "nsie" and i:  # a satellite of the main lens
            a, b = [cx + 1.2 * er, cy - 0.6 * er, 0.16 * er, 1.0, a[4], a[5]], [1, 1, 0.01 * er, 0.2, 0.05, 10]
        if plugin == "sersic" and any(p == "sersic" for _, p in MODELS[model][:i]):  # a fainter second source
            a = [a[0] - 0.2 * er, a[1] + 0.1 * er, 0.6 * a[2], a[3] + 1, 1.0, 0.6, 120.0]
            b = [1, 1, a[2] / 5, 0.3, 0.2, 0.08, 10]
        t += a
        h += b
    return np.float32(t).astype(np.float64), np.float32(h).astype(np.float64)


def _system(model, width, height, psf_w, psf_h, seed):
    """One observed system: image, weight, PSF, true parameters and prior box."""
    rng = random.Random(seed)
    psf = _psf(psf_w, psf_h, rng) if psf_w else None
    truth, half = _truth(model, width, height, rng)
    lo = np.float32(truth - half).astype(np.float64)
    hi = np.float32(truth + half).astype(np.float64)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    p = torch.from_numpy(truth).cuda()[None]
    mock = _render64(model, width, height, p, [(0.0, 0.0, 1.0)], even=_even(psf))
    if psf is not None:
        mock = _convolve64(mock, psf)
    mock = mock[0]
    noise = torch.randn(mock.shape, generator=gen, device="cuda", dtype=torch.float64)
    image = (mock + noise * (mock.clamp(min=0) + 1).sqrt()).float()
    weight = 1.0 / (image.double().clamp(min=-0.5) + 1.0)
    weight[torch.rand(mock.shape, generator=gen, device="cuda") < 0.1] = 0  # masked pixels
    return {"image": image.cpu().numpy(), "weight": weight.float().cpu().numpy(), "psf": psf, "truth": truth,
            "lo": lo, "hi": hi, "model": model}


def _candidates(s, batch, seed):
    """Candidates in object order: half of them near the truth, the rest from
    the whole box; single-precision values, as the model takes them."""
    g = np.random.Generator(np.random.PCG64(seed))
    c = s["lo"] + g.random((batch, len(s["lo"]))) * (s["hi"] - s["lo"])
    c[: batch // 2] = s["truth"] + 0.1 * (c[: batch // 2] - s["truth"])
    c = np.float32(c).astype(np.float64)
    return np.where(s["lo"] == s["hi"], s["truth"], c)


def _map_order(s):
    """Free parameters first, then the fixed ones, each in object order."""
    free = s["lo"] != s["hi"]
    return np.concatenate([np.flatnonzero(free), np.flatnonzero(~free)])


def _counts(case):
    """Sizes, PSF sizes and candidate counts of a multi-system case: ragged, from its own numbers."""
    rng = random.Random("%(width)d %(psf_w)d %(batch)d %(count)d" % case)
    out = []
    for k in range(case["count"]):
        w = case["width"] if k == 0 else max(48, int(case["width"] * rng.choice([0.125, 0.25, 0.5, 0.61])))
        p = case["psf_w"] if k == 0 else rng.randrange(min(15, case["psf_w"]), case["psf_w"] + 1, 2)
        out.append((w, p, case["batch"] if k == 0 else rng.randint(1, case["batch"])))
    return out


def _systems(case, seed):
    return [(_system(case["model"], w, w, p, p, seed * 1000 + k), n) for k, (w, p, n) in enumerate(_counts(case))]


def _live_points(case, seed):
    """A sampler's live points half-way: a curved, correlated cloud in the unit cube."""
    g = np.random.Generator(np.random.PCG64(seed))
    d = case["dims"]
    x = g.normal(size=(case["points"], d)) @ (np.eye(d) + 0.3 * g.normal(size=(d, d)) / math.sqrt(d))
    x[:, 1] += 0.5 * x[:, 0] ** 2
    return 0.5 + 0.05 * x


def _inputs(case, seed):
    s = _system(case["model"], case["width"], case["height"], case["psf_w"], case["psf_h"], seed)
    if case["kind"] in ("cube", "callback"):
        free = np.flatnonzero(s["lo"] != s["hi"])
        s["cube"] = np.random.Generator(np.random.PCG64(seed + 1)).random((case["batch"], len(free)))
        phys = np.tile(s["truth"], (case["batch"], 1))
        phys[:, free] = s["lo"][free] + s["cube"] * (s["hi"] - s["lo"])[free]
        s["phys"] = phys  # object order
    else:
        s["params"] = _candidates(s, case["batch"], seed + 1)
    return s


def _objects(s):
    out, k = [], 0
    for oid, plugin in MODELS[s["model"]]:
        n = len(lg.plugin_params(plugin))
        pri = [repr(float(s["truth"][i])) if s["lo"][i] == s["hi"][i] else
               "unif %r %r" % (float(s["lo"][i]), float(s["hi"][i])) for i in range(k, k + n)]
        out.append((oid, plugin, pri))
        k += n
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "training":
        return {"kind": kind, "points": _live_points(case, seed), "epochs": case["epochs"]}
    flags = FLAGS[case["mode"]]
    if kind == "systems":
        both = _systems(case, seed)
        ctx = lg.Systems([(s["image"], s["weight"], s["psf"], None) for s, _ in both], _box_free(both[0][0]),
                         [n for _, n in both], rule=case["rule"], flags=flags)
        params = [_candidates(s, n, seed + 1 + k)[:, _map_order(s)] for k, (s, n) in enumerate(both)]
        return {"kind": kind, "ctx": ctx, "params": params}
    s = _inputs(case, seed)
    ctx = lg.Context(s["image"], s["weight"], _objects(s), psf=s["psf"], rule=case["rule"], max_batch=case["batch"],
                     flags=flags)
    st = {"kind": kind, "ctx": ctx, "batch": case["batch"]}
    if kind == "callback":
        st["cube"] = s["cube"][0]
    elif kind == "cube":
        st["cube"] = torch.from_numpy(s["cube"]).cuda()
        st["phys"] = torch.empty((case["batch"], ctx.npars), dtype=torch.float64, device="cuda")
        st["logl"] = torch.empty(case["batch"], dtype=torch.float64, device="cuda")
    elif kind == "sampler":
        st["opts"] = dict(nlive=case["nlive"], batch=case["batch"], maxiter=case["maxiter"], seed=seed % 2 ** 31)
    else:
        st["params"] = ctx.to_map_order(s["params"])
        if kind == "device":
            st["params"] = torch.from_numpy(st["params"]).cuda()
            st["logl"] = torch.empty(case["batch"], dtype=torch.float64, device="cuda")
    return st


def _box_free(s):
    """The objects of a multi-system batch: fixed parameters fixed, the others free over their whole range."""
    out, k = [], 0
    for oid, plugin in MODELS[s["model"]]:
        n = len(lg.plugin_params(plugin))
        out.append((oid, plugin, [repr(float(s["truth"][i])) if s["lo"][i] == s["hi"][i] else "unif 0 1000"
                                  for i in range(k, k + n)]))
        k += n
    return out


def run(state):
    kind, ctx = state["kind"], state.get("ctx")
    if kind == "callback":
        logl, phys = ctx.loglike(state["cube"])
        return {"logl": logl, "phys": phys}
    if kind == "host":
        return {"logl": ctx.eval_batch(state["params"])}
    if kind == "device":
        ctx.eval_batch_device(state["params"].data_ptr(), state["batch"], state["logl"].data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
        return {"logl": state["logl"]}
    if kind == "cube":
        ctx.eval_cube_device(state["cube"].data_ptr(), state["batch"], state["phys"].data_ptr(),
                             state["logl"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"logl": state["logl"], "phys": state["phys"]}
    if kind == "systems":
        return {"logl": ctx.eval(state["params"])}
    if kind == "layers":
        return ctx.dump(state["params"][0])
    if kind == "sampler":
        r = ctx.nested(**state["opts"])
        return {k: r[k] for k in ("logz", "logz_err", "information", "max_logl", "ncall", "niter", "mean", "std",
                                  "samples", "logwt")}
    history, kept = lg.flow_fit(state["points"], epochs=state["epochs"], patience=state["epochs"])
    return {"history": history, "kept": kept}


# -------------------------------------------------------------------- work
def _ray_flops(model):
    return sum(RAY_FLOPS[p] for _, p in MODELS[model]) + RAY_OVERHEAD


def _flops(case):
    if case["kind"] == "training":  # forward and backward of the coupling layers' MLPs
        d = case["dims"]
        macs = 8 * ((d + 1) // 2 * 128 + 128 * 128 + 128 * 2 * ((d + 1) // 2))
        return 6.0 * macs * 0.8 * case["points"] * case["epochs"]
    ray = RULE_POINTS[case["rule"]] * _ray_flops(case["model"])
    if case["kind"] == "systems":
        return float(sum(n * w * w * (ray + 2 * p * p) for w, p, n in _counts(case)))
    evals = case["nlive"] + case["maxiter"] if case["kind"] == "sampler" else case["batch"]
    return float(evals) * case["width"] * case["height"] * (ray + 2 * case["psf_w"] * case["psf_h"])


def work(case):
    if case["kind"] == "training":
        return {"bytes": 8.0 * case["points"] * case["dims"] + 4.0 * case["epochs"], "flops": _flops(case)}
    if case["kind"] == "systems":
        data = sum(8.0 * w * w + 4.0 * p * p + 160.0 * n for w, p, n in _counts(case))
        return {"bytes": data, "flops": _flops(case)}
    npix = case["width"] * case["height"]
    data = 8.0 * npix + 4.0 * case["psf_w"] * case["psf_h"]
    if case["kind"] == "layers":
        data += 24.0 * npix
    elif case["kind"] == "sampler":
        data += 8.0 * 14 * (case["nlive"] + case["maxiter"])
    else:
        data += 8.0 * case["batch"] * (1 + len(_truth(case["model"], 64, 64, random.Random(0))[0]))
    return {"bytes": data, "flops": _flops(case)}


# ------------------------------------------------------- float64 restatement
def _rule64(rule):
    """Points (x, y, weight) on the unit pixel."""
    if rule.startswith("sub"):
        n = int(rule[3:])
        xs = [((i + 0.5) / n - 0.5, 1.0 / n) for i in range(n)]
    else:  # 7-point Kronrod rule (Kronrod 1965), tensor product
        node = [0.960491268708020283423507092629080, 0.774596669241483377035853079956480,
                0.434243749346802558002071502844628, 0.0]
        weig = [0.104656226026467265193823857192073, 0.268488089868333440728569280666710,
                0.401397414775962222905051818618432, 0.450916538658474142345110087255013]
        xs = [(s * a / 2, w / 2) for a, w in zip(node, weig) for s in ((-1, 1) if a else (1,))]
    return [(a, b, u * v) for a, u in xs for b, v in xs]


def _even(psf):
    """Half-pixel shift of the pixel coordinates for even PSF sides."""
    return (0.0, 0.0) if psf is None else (0.5 * (psf.shape[1] % 2 == 0), 0.5 * (psf.shape[0] % 2 == 0))


def _lens64(plugin, x, y, p):
    dx, dy = x - p[0], y - p[1]
    if plugin == "point_mass":
        k = p[2] ** 2 / (dx * dx + dy * dy)
        return k * dx, k * dy
    q, pa = {"sie": (3, 4), "sie_plus_shear": (3, 4), "nsie": (4, 5), "epl_plus_shear": (4, 5)}[plugin]
    q, c, s = p[q], torch.cos(p[pa] * (math.pi / 180)), torch.sin(p[pa] * (math.pi / 180))
    u, v = c * dx + s * dy, c * dy - s * dx
    if plugin == "epl_plus_shear":  # Tessore & Metcalf 2015, ten terms of the series
        t = p[3]
        z = torch.complex(q * u, v) / (p[2] * q.sqrt())
        r = z.abs()
        e = z / r
        e2 = e * e
        f = (1 - q) / (1 + q)
        term = total = e
        for k in range(1, 11):
            term = term * e2 * (-f * (2 * k - (2 - t)) / (2 * k + (2 - t)))
            total = total + term
        total = total * (2 * p[2] * q.sqrt() / (1 + q) * r ** (1 - t))
        a, b = total.real, total.imag
    else:  # (non-)singular isothermal ellipsoid, Schneider, Kochanek & Wambsganss 2006
        e = (1 - q * q).sqrt()
        core = p[3] if plugin == "nsie" else torch.zeros_like(q)
        w = (q * q * u * u + v * v).sqrt()
        d = p[2] * q.sqrt() / e
        a, b = d * torch.atan(u * e / (core + w)), d * torch.atanh(v * e / (core * q * q + w))
    ax, ay = c * a - s * b, s * a + c * b
    if plugin.endswith("_plus_shear"):
        g1, g2 = p[-2], p[-1]
        ax, ay = ax + g1 * dx + g2 * dy, ay + g2 * dx - g1 * dy
    return ax, ay


def _source64(plugin, x, y, p):
    dx, dy = x - p[0], y - p[1]
    mag, q, pa = p[3], p[-2], p[-1] * (math.pi / 180)
    c, s = torch.cos(pa), torch.sin(pa)
    r2 = (q * (c * dx + s * dy)) ** 2 + (c * dy - s * dx) ** 2
    flux = 10 ** (-0.4 * mag)
    if plugin == "sersic":  # b(n): Ciotti & Bertin 1999 as MacArthur, Courteau & Holtzman 2003 use it
        n = p[4]
        b = 2 * n - 1 / 3 + 4 / (405 * n) + 46 / (25515 * n ** 2) + 131 / (1148175 * n ** 3) - 2194697 / (30690717750 * n ** 4)
        log0 = -0.4 * mag * math.log(10) + 2 * n * b.log() - math.log(math.pi) - 2 * p[2].log() - torch.lgamma(2 * n + 1)
        return torch.exp(log0 - b * (r2 / (q * p[2] ** 2)) ** (0.5 / n))
    if plugin == "exponential":
        return flux / (2 * math.pi * p[2] ** 2 * q) * torch.exp(-r2.sqrt() / p[2])
    if plugin == "gauss":
        return flux / (2 * math.pi * p[2] ** 2 * q) * torch.exp(-0.5 * r2 / p[2] ** 2)
    b = 7.6692494425008039044
    return flux * b ** 8 / math.factorial(8) / (math.pi * p[2] ** 2 * q) * torch.exp(-b * (r2.sqrt() / p[2]) ** 0.25)


def _render64(model, width, height, params, points, even=(0.0, 0.0)):
    """Images (B, H, W) of B parameter vectors (object order, float64, GPU)."""
    dev, f8 = params.device, torch.float64
    px = torch.arange(width, device=dev, dtype=f8)[None, None, :] + (1 + even[0])
    py = torch.arange(height, device=dev, dtype=f8)[None, :, None] + (1 + even[1])
    cols = [params[:, i, None, None] for i in range(params.shape[1])]
    out = torch.zeros((params.shape[0], height, width), device=dev, dtype=f8)
    npar = {"sie": 5, "sie_plus_shear": 7, "epl_plus_shear": 8, "nsie": 6, "point_mass": 3, "sersic": 7,
            "exponential": 6, "devauc": 6, "gauss": 6, "sky": 3}
    for qx, qy, w in points:
        x, y = px + qx, py + qy
        ax = ay = 0.0
        f, k = 0.0, 0
        for _, plugin in MODELS[model]:
            p = cols[k: k + npar[plugin]]
            k += npar[plugin]
            if plugin in ("sersic", "exponential", "devauc", "gauss"):
                f = f + _source64(plugin, x - ax, y - ay, p)
            elif plugin == "sky":
                f = f + p[0] + p[1] * (x - 1) + p[2] * (y - 1)
            else:
                a, b = _lens64(plugin, x, y, p)
                ax, ay = ax + a, ay + b
        out += w * f
    return out


def _convolve64(images, psf):
    """Convolution with edge pixels repeated outside the image."""
    h, w = psf.shape
    oy, ox = h - 1 - h // 2, w - 1 - w // 2
    kernel = torch.from_numpy(psf.astype(np.float64)).to(images.device)
    kernel = kernel / kernel.sum()
    a = torch.nn.functional.pad(images[:, None], (w - 1 - ox, ox, h - 1 - oy, oy), mode="replicate")[:, 0]
    size = (a.shape[-2] + h - 1, a.shape[-1] + w - 1)
    r = torch.fft.irfft2(torch.fft.rfft2(a, s=size) * torch.fft.rfft2(kernel, s=size), s=size)
    return r[:, h - 1: h - 1 + images.shape[1], w - 1: w - 1 + images.shape[2]]


def _images64(s, width, height, rule, params):
    """(unconvolved, convolved) images of parameter vectors, a few at a time."""
    step = max(1, (1 << 23) // (width * height))
    for i in range(0, len(params), step):
        p = torch.from_numpy(np.float32(params[i: i + step]).astype(np.float64)).cuda()
        raw = _render64(s["model"], width, height, p, _rule64(rule), even=_even(s["psf"]))
        yield raw, raw if s["psf"] is None else _convolve64(raw, s["psf"])


def _logl64(s, width, height, rule, params):
    image = torch.from_numpy(s["image"]).cuda().double()
    weight = torch.from_numpy(s["weight"]).cuda().double()
    return torch.cat([-0.5 * (weight * (m - image) ** 2).sum((1, 2)) for _, m in _images64(s, width, height, rule, params)])


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sampler", "training"):
        return None  # random walks: no value but the program's own
    if kind == "systems":
        out = []
        for k, (s, n) in enumerate(_systems(case, seed)):
            h, w = s["image"].shape
            out.append(_logl64(s, w, h, case["rule"], _candidates(s, n, seed + 1 + k)))
        return {"logl": out}
    s = _inputs(case, seed)
    w, h = case["width"], case["height"]
    if kind == "layers":
        raw, img = (v[0] for v in next(_images64(s, w, h, case["rule"], s["params"])))
        image = torch.from_numpy(s["image"]).cuda().double()
        weight = torch.from_numpy(s["weight"]).cuda().double()
        chi = weight * (img - image) ** 2
        # (the quadrature error estimate is a difference of nearly equal sums: rounding alone)
        return {"IMG": img, "RES": image - img, "RAW": raw, "ERR": None, "WHT": weight, "PVL": torch.erfc((chi / 2).sqrt())}
    if kind in ("cube", "callback"):
        logl = _logl64(s, w, h, case["rule"], s["phys"])
        phys = s["phys"][:, _map_order(s)]
        return {"logl": float(logl[0]) if kind == "callback" else logl, "phys": phys[0] if kind == "callback" else phys}
    return {"logl": _logl64(s, w, h, case["rule"], s["params"])}
