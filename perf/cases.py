"""The work this engine does for its users, as cases that can be timed one by one.

A fit is a sequence of likelihood calls: the minimiser moves the parameters, `Engine.nll_grad` returns the NLL and
its analytic gradient, and a toy study does that for many data sets at once with `Engine.nll_batch`.  New data come
in through `Engine.upload`; per-event probabilities (plots, event weights) come out through `Engine.eval_events`.
The cases cover the model families of the package's workloads over the sizes its tests, configurations and benchmark
use, from a thousand events to tens of millions:

  decay      exponential, analytic normalisation (a lifetime fit)
  peak       extended sum of two Gaussians and a polynomial: every event's probability depends on x itself
  composite  smeared exponential (convolution table) plus a flat background
  new-data   the composite model's next data set: upload from ordinary host memory, then one call
  toys       many small composite data sets, one batched call
  dalitz     three-body amplitude model, resonance shapes fixed (the coefficients are fitted)
  dalitz-shapes, fourbody-shapes
             amplitude models whose masses and widths are fitted: every call rebuilds the amplitude caches and the
             normalisation integrals.  A pass makes two calls at two points, because a repeated point rebuilds nothing
  probs      per-event probabilities of the peak model, returned to the host
  fit        a whole minimisation in the FP64 engine (values, errors, minimum)

Gradients and toy NLLs of the mixed engine are given back as the FP32 numbers that its event arithmetic carries: the
engine chooses its event chunking by timing, so the last bits of its FP32 sums are not the same from process to
process.  FP64 results and per-event probabilities are given back as they come.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import goofit_gb300 as G
from goofit_gb300 import workloads as W

# ---------------------------------------------------------------- the cases


def listed():
    return [
        # the smallest fit: a thousand decay times, where the launch and the host round trip are everything
        {"name": "decay-1e3", "family": "decay", "n": 1003},
        # an ordinary mass spectrum
        {"name": "peak-2e4", "family": "peak", "n": 20011, "bins": 1000},
        # a large one: arithmetic per event
        {"name": "peak-5e6", "family": "peak", "n": 5000003, "bins": 1000},
        # the composite model at the benchmark's size
        {"name": "composite-2e6", "family": "composite", "n": 2000000},
        # ten times that, ragged: the events of one CTA no longer fit its shared memory
        {"name": "composite-2e7", "family": "composite", "n": 20000003},
        # the next data set of the composite model: host events to first likelihood value
        {"name": "new-data-2e6", "family": "new-data", "n": 2000000},
        # the benchmark's toy study: one lockstep round of 1024 data sets of about 20,000 events
        {"name": "toys-1024", "family": "toys", "toys": 1024, "mean": 20000},
        # the three-body amplitude model at the benchmark's size, coefficients fitted
        {"name": "dalitz-5e5", "family": "dalitz", "n": 500000, "res": 8, "bins": 1500},
        # the same model while masses and widths of four resonances are fitted
        {"name": "dalitz-shapes-1e5", "family": "dalitz-shapes", "n": 100003, "res": 8, "bins": 1500, "floated": 4},
        # the four-body amplitude model at the benchmark's size, all line shapes fitted
        {"name": "fourbody-shapes-3e5", "family": "fourbody-shapes", "n": 300000, "norm": 2000000},
        # per-event probabilities of a million events (a plot, event weights)
        {"name": "probs-1e6", "family": "probs", "n": 1000003, "bins": 1000},
        # a whole FP64 minimisation of a hundred thousand events
        {"name": "fit-fp64-1e5", "family": "fit", "n": 100003},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["decay", "peak", "peak", "composite", "composite", "new-data", "toys", "dalitz", "dalitz",
                         "dalitz-shapes", "fourbody-shapes", "probs", "fit"])
    case = {"family": family}
    if family == "decay":
        case["n"] = _log(rng, 500, 2000000)
    elif family == "peak":
        case.update(n=_log(rng, 2000, 5000000), bins=rng.choice([100, 1000, 2500]))
    elif family == "composite":
        case["n"] = _log(rng, 5000, 20000000)
    elif family == "new-data":
        case["n"] = _log(rng, 5000, 2000000)
    elif family == "toys":
        case.update(toys=_log(rng, 3, 1024), mean=_log(rng, 600, 20000))
    elif family == "dalitz":
        case.update(n=_log(rng, 5000, 2000000), res=rng.randint(2, 8), bins=rng.choice([300, 1500]))
    elif family == "dalitz-shapes":
        case.update(n=_log(rng, 2000, 100000), res=rng.randint(3, 8), bins=rng.choice([300, 600, 1500]),
                    floated=rng.randint(1, 3))
    elif family == "fourbody-shapes":
        case.update(n=_log(rng, 5000, 300000), norm=_log(rng, 50000, 1900000))
    elif family == "probs":
        case.update(n=_log(rng, 1000, 1000000), bins=rng.choice([100, 1000]))
    else:
        case["n"] = _log(rng, 2000, 100000)
    return case


# ---------------------------------------------------------------- inputs

PEAK_LO, PEAK_HI = 0.0, 10.0
PEAK_TRUTH = dict(mean=5.0, s1=0.3, s2=0.8, c1=-0.04, c2=0.002, f1=0.25, f2=0.15)
COMP = dict(alpha=-1 / 1.5, mu=0.0, sigma=0.3, fsig=0.7)
COMP_POINT = dict(alpha=-0.6, mu=0.05, sigma=0.35, c0=1.0, fsig=0.65)  # where the fits of the workload start
X_LO, X_HI, STEP, NM, NR, KMIN, NK, OFFSET = -5.0, 10.0, 0.01, 1000, 2500, -500, 1501, 1000


def _generator(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _rand(g, *n):
    return torch.rand(*n, generator=g, device="cuda", dtype=torch.float64)


def _host(x):
    return np.ascontiguousarray(x.cpu().numpy())


def _decay_events(n, seed):
    u = _rand(_generator(seed), n)
    return _host(-torch.log1p(-u * (1.0 - math.exp(-7.0))) / 0.7).reshape(1, -1)


def _peak_events(n, seed):
    g = _generator(seed)
    t = PEAK_TRUTH
    x = torch.empty(n, device="cuda", dtype=torch.float64)
    which = _rand(g, n)
    z = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    sig = which < t["f1"] + t["f2"]
    width = torch.where(which < t["f1"], t["s1"], t["s2"])
    # the background by inversion on a fine grid
    xs = torch.linspace(PEAK_LO, PEAK_HI, 4097, device="cuda", dtype=torch.float64)
    cdf = xs + t["c1"] * xs ** 2 / 2 + t["c2"] * xs ** 3 / 3
    cdf = cdf / cdf[-1]
    u = _rand(g, n)
    j = torch.searchsorted(cdf, u).clamp(1, 4096)
    bkg = xs[j - 1] + (u - cdf[j - 1]) / (cdf[j] - cdf[j - 1]) * (xs[j] - xs[j - 1])
    x = torch.where(sig, t["mean"] + width * z, bkg)
    return _host(x.clamp(PEAK_LO, PEAK_HI)).reshape(1, -1)


def _conv_table(alpha, mu, sigma, device="cuda"):
    """T[k] = sum_m exp(alpha t_m) gauss(t_{m + offset - k}) for the bin offsets k = KMIN .. KMIN + NK - 1."""
    f = dict(device=device, dtype=torch.float64)
    tm = 10.0 / NM * (torch.arange(NM, **f) + 0.5)
    tr = 25.0 / NR * (torch.arange(NR, **f) + 0.5) - 10.0
    m = torch.exp(alpha * tm)
    r = torch.exp(-0.5 * (tr - mu) ** 2 / sigma ** 2)
    full = r.unfold(0, NM, 1) @ m  # full[j] = sum_m M[m] R[m + j]
    ks = torch.arange(KMIN, KMIN + NK, device=device)
    return full[OFFSET - ks]


def _grid_counts(device="cuda"):
    """Normalisation bins (10,000 over the range) per bin offset."""
    c = (X_HI - X_LO) / 10000 * (torch.arange(10000, device=device, dtype=torch.float64) + 0.5) + X_LO
    return torch.bincount(torch.floor(c / STEP).long() - KMIN, minlength=NK).double()


def _composite_density(alpha, mu, sigma, fsig):
    """Probability density in every bin offset."""
    t = _conv_table(alpha, mu, sigma)
    norm = (X_HI - X_LO) / 10000 * (t * _grid_counts()).sum()
    return fsig * t / norm + (1 - fsig) / (X_HI - X_LO)


def _composite_sample(n, g, cdf):
    k = torch.searchsorted(cdf, _rand(g, n)).clamp(max=NK - 2)
    return ((k + KMIN + _rand(g, n)) * STEP).clamp(X_LO, X_HI)


def _composite_cdf(**truth):
    d = _composite_density(**{k: torch.tensor(v, device="cuda", dtype=torch.float64) for k, v in truth.items()})
    c = torch.cumsum(d[: NK - 1], 0)
    return c / c[-1]


def _composite_events(n, seed):
    return _host(_composite_sample(n, _generator(seed), _composite_cdf(**COMP))).reshape(1, -1)


def _toy_events(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    lo, hi = max(16, case["mean"] // 4), 3 * case["mean"]
    counts = np.clip(rng.poisson(case["mean"], case["toys"]), lo, hi)
    g = _generator(seed)
    cdfs = []
    for _ in range(min(16, case["toys"])):  # the toys' generation parameters: 16 points around the truth
        j = rng.uniform(-0.1, 0.1, 4)
        cdfs.append(_composite_cdf(alpha=COMP["alpha"] * (1 + j[0]), mu=0.3 * j[1], sigma=0.3 * (1 + j[2]),
                                   fsig=0.7 * (1 + j[3])))
    return [_host(_composite_sample(int(c), g, cdfs[t % len(cdfs)])).reshape(1, -1) for t, c in enumerate(counts)]


def _toy_points(case, seed, names):
    """Every toy's parameters (columns in the order of `names`): its own point near the start of the fits."""
    rng = np.random.Generator(np.random.PCG64(seed + 77))
    scale = 1 + 0.05 * rng.uniform(-1, 1, (case["toys"], len(names)))
    return np.array([COMP_POINT[k] for k in names]) * np.where([k == "c0" for k in names], 1.0, scale)


def _accept(n, g, propose, weigh, batch=2000000):
    """Accept-reject sample of the density weigh() over the points of propose() (columns first)."""
    out, have, top = [], 0, None
    while have < n:
        x = propose(g, batch)
        w = weigh(x)
        top = 1.1 * w.max() if top is None else torch.maximum(top, w.max())
        keep = x[:, _rand(g, x.shape[1]) * top < w]
        out.append(keep)
        have += keep.shape[1]
    return torch.cat(out, 1)[:, :n]


def _dalitz_points(g, n):
    return torch.stack([3.0 * _rand(g, n), 3.0 * _rand(g, n)])


def _with_number(x):
    """The columns with the event number as the last one."""
    return torch.cat([x, torch.arange(x.shape[1], device="cuda", dtype=torch.float64).reshape(1, -1)])


def _flat_four(g, n):
    """About n flat four-body phase-space points (m12, m34, cos12, cos34, phi)."""
    m1, m2, m3, m4 = W.C5_MASSES
    m12 = m1 + m2 + _rand(g, n) * (W.C5_M - sum(W.C5_MASSES))
    m34 = m3 + m4 + _rand(g, n) * (W.C5_M - sum(W.C5_MASSES))

    def mom(a, b, c):
        return torch.sqrt(((a - b - c) * (a + b + c) * (a - b + c) * (a + b - c)).clamp(min=0)) / (2 * a)

    w = torch.where(m12 + m34 < W.C5_M, mom(torch.full_like(m12, W.C5_M), m12, m34) * mom(m12, m1, m2)
                    * mom(m34, m3, m4), torch.zeros_like(m12))
    keep = _rand(g, n) * w.max() < w
    m = int(keep.sum())
    return torch.stack([m12[keep], m34[keep], 2 * _rand(g, m) - 1, 2 * _rand(g, m) - 1,
                        math.pi * (2 * _rand(g, m) - 1)])


def _norm_events(n, seed):
    g = _generator(seed, 5)
    out, have = [], 0
    while have < n:
        out.append(_flat_four(g, 3000000))
        have += out[-1].shape[1]
    return torch.cat(out, 1)[:, :n]


# ---------------------------------------------------------------- models and engines


def _peak_pdf(bins):
    x = G.Observable("x", PEAK_LO, PEAK_HI)
    x.setNumBins(bins)
    mean = G.Variable("mean", 5.0, 0.01, 4.0, 6.0)
    s1, s2 = G.Variable("s1", 0.3, 0.01, 0.05, 1.0), G.Variable("s2", 0.8, 0.01, 0.2, 3.0)
    g1, g2 = G.GaussianPdf("narrow", x, mean, s1), G.GaussianPdf("wide", x, mean, s2)
    bkg = G.PolynomialPdf("background", x, [G.Variable("c0", 1.0), G.Variable("c1", -0.04, 0.001, -0.1, 0.1),
                                            G.Variable("c2", 0.002, 0.0001, -0.01, 0.01)], 0)
    n1, n2, nb = (G.Variable(k, 1.0, 1.0, 0.0, 1e9) for k in ("n1", "n2", "nb"))
    return G.AddPdf("total", [n1, n2, nb], [g1, g2, bkg])


def _peak_point(n):
    """Parameters by name, a little away from the truth."""
    return dict(mean=5.02, s1=0.31, s2=0.77, c0=1.0, c1=-0.042, c2=0.0021, n1=0.24 * n, n2=0.16 * n, nb=0.61 * n)


def _composite_pdf():
    return W.make_c2(16, seed=0).pdf


def _dalitz_pdf(case):
    pdf = W.c3_model(case["bins"], case["res"])[0]
    for name, *_ in W.C3_RESONANCES[: case.get("floated", 0)]:
        for v in pdf.getParameters():
            if v.name in (f"{name}_mass", f"{name}_width"):
                v.setFixed(False)
    return pdf


def _fourbody_pdf():
    # its own normalisation events are replaced below (drawn on the GPU)
    return W.c5_model(1000, float_lineshapes=True)[0]


def _engine(pdf, precision="mixed"):
    """An engine with the tree of `pdf`, gradients with respect to its free parameters."""
    nodes, params, obs = pdf._flatten()
    fixed = pdf._nondiff_all()
    mask = [0 if (v.fixed or id(v) in fixed) else 1 for v in params]
    eng = G.Engine(precision)
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params),
                 mask)
    return eng, params


def _points_of(params, n_points, skip=()):
    """Parameter vectors a few per mille to a few per cent away from the values of `params`, as a fit visits them."""
    v0 = np.array([v.value for v in params])
    free = np.array([0.0 if v.fixed else 1.0 for v in params])
    return [v0 * (1 + free * (0.01 + 0.004 * k) * np.cos(1.7 * np.arange(len(v0)) + k)) for k in range(n_points)]


def _shape_values(params, value):
    return {v.name: value[i] for i, v in enumerate(params)}


def prepare(case, seed):
    family = case["family"]
    if family == "decay":
        eng, params = _engine(W.make_c1(16).pdf)
        eng.upload(_decay_events(case["n"], seed))
        return {"family": "call", "engine": eng, "points": [np.array([-0.3])]}
    if family in ("peak", "probs"):
        eng, params = _engine(_peak_pdf(case["bins"]))
        eng.upload(_peak_events(case["n"], seed))
        point = _peak_point(case["n"])
        p = np.array([point[v.name] for v in params])
        if family == "probs":
            eng.set_params(p)
        return {"family": "call" if family == "peak" else "probs", "engine": eng, "points": [p]}
    if family in ("composite", "new-data", "fit"):
        eng, params = _engine(_composite_pdf(), "fp64" if family == "fit" else "mixed")
        events = _composite_events(case["n"], seed)
        p = np.array([COMP_POINT[v.name] for v in params])
        if family != "new-data":
            eng.upload(events)
        if family == "composite":
            return {"family": "call", "engine": eng, "points": [p]}
        if family == "new-data":
            return {"family": family, "engine": eng, "points": [p], "events": events}
        return {"family": family, "engine": eng, "x0": p, "err": np.array([v.error for v in params]),
                "lo": np.array([v.lowerlimit for v in params]), "hi": np.array([v.upperlimit for v in params]),
                "fixed": np.array([int(v.fixed) for v in params], dtype=np.int32)}
    if family == "toys":
        eng, params = _engine(_composite_pdf())
        eng.set_num_toys(case["toys"])
        for t, events in enumerate(_toy_events(case, seed)):
            eng.upload(events, t)
        return {"family": family, "engine": eng, "points": _toy_points(case, seed, [v.name for v in params])}
    if family in ("dalitz", "dalitz-shapes"):
        pdf = _dalitz_pdf(case)
        eng, params = _engine(pdf)
        eng.upload(_dalitz_events(case, seed))
        return {"family": "call", "engine": eng, "points": _points_of(params, 1 if family == "dalitz" else 2)}
    pdf = _fourbody_pdf()
    eng, params = _engine(pdf)
    eng.set_norm_events(0, _host(_norm_events(case["norm"], seed)))
    eng.upload(_fourbody_events(case, seed))
    return {"family": "call", "engine": eng, "points": _points_of(params, 2)}


def _mixed(value, grad):
    return {"nll": value, "grad": grad.astype(np.float32)}


def run(state):
    family, eng = state["family"], state["engine"]
    if family == "call":
        return [_mixed(*eng.nll_grad(p)) for p in state["points"]]
    if family == "new-data":
        eng.upload(state["events"])
        return [_mixed(*eng.nll_grad(p)) for p in state["points"]]
    if family == "toys":
        nll, grad = eng.nll_batch(state["points"], grad=True)
        return {"nll": nll.astype(np.float32), "grad": grad.astype(np.float32)}
    if family == "probs":
        return eng.eval_events()
    fixed = state["fixed"]
    r = eng.fit(state["x0"], state["err"], state["lo"], state["hi"], 1 - fixed, fixed, tolerance=0.01)
    return {"values": r.values, "errors": r.errors, "fmin": np.array(r.fmin)}


# ---------------------------------------------------------------- what a pass cannot do without


def work(case):
    family = case["family"]
    n = case.get("n", 0)
    table = 2.0 * NM * NK * 4  # convolution table: the value and three derivatives
    if family == "decay":
        return {"bytes": 4 * n + 16, "flops": 12 * n}
    if family == "peak":
        return {"bytes": 4 * n + 80, "flops": 70 * n + 10 * case["bins"]}
    if family == "composite":
        return {"bytes": 4 * n + 48, "flops": table + 10 * n}
    if family == "new-data":  # host events in, the call's column out
        return {"bytes": 12 * n + 48, "flops": table + 15 * n}
    if family == "toys":
        events = case["toys"] * case["mean"]
        return {"bytes": 4 * events + 80 * case["toys"], "flops": case["toys"] * table + 40 * events}
    if family == "dalitz":
        return {"bytes": 8 * case["res"] * n, "flops": (20 * case["res"] + 20) * n}
    if family == "dalitz-shapes":
        # both calls: the events' two variables, the points' bin numbers; the shapes at every event and point, and
        # the integrals (the in-boundary share of the box is 0.353)
        points = 0.353 * case["bins"] ** 2
        cols = case["res"] + 2 * case["floated"]
        return {"bytes": 2 * (16 * n + 4 * points),
                "flops": 2 * ((100 * case["res"] + 300 * case["floated"]) * (n + points) + 8 * cols * case["res"] * points)}
    if family == "fourbody-shapes":
        # both calls: five variables of every event and normalisation event; six amplitudes and their thirty
        # derivative columns
        points = case["norm"]
        return {"bytes": 2 * 40 * (n + points), "flops": 2 * (3000 * (n + points) + 8 * 36 * 6 * points)}
    if family == "probs":
        return {"bytes": 12 * n, "flops": 40 * n}
    # a fit: about 40 calls over the FP64 model
    return {"bytes": 40 * 4 * n, "flops": 40 * (table + 40 * n)}


# ---------------------------------------------------------------- the same in 64 bits, plain torch


def _t(v, grad=False):
    return torch.tensor(v, device="cuda", dtype=torch.float64, requires_grad=grad)


def _value_grad(f, names, free, point):
    """NLL and gradient (free parameters in the order of `names`) of f(dict of scalars)."""
    p = {k: _t(float(point[k]), k in free) for k in names}
    nll = f(p)
    g = torch.autograd.grad(nll, [p[k] for k in names if k in free])
    return {"nll": float(nll.detach()), "grad": np.array([float(v) for v in g])}


def _peak_density(p, x):
    return [torch.exp(-0.5 * ((x - p["mean"]) / p[s]) ** 2) / (p[s] * math.sqrt(2 * math.pi)) for s in ("s1", "s2")]


def _peak_prob(p, x, bins):
    c = (PEAK_HI - PEAK_LO) / bins * (torch.arange(bins, device="cuda", dtype=torch.float64) + 0.5) + PEAK_LO
    poly = lambda t: p["c0"] + p["c1"] * t + p["c2"] * t * t  # noqa: E731
    norm = (PEAK_HI - PEAK_LO) / bins * poly(c).sum()
    total = p["n1"] + p["n2"] + p["nb"]
    g1, g2 = _peak_density(p, x)
    return (p["n1"] * g1 + p["n2"] * g2 + p["nb"] * poly(x) / norm) / total, total


def _exact_peak(case, seed):
    x = _t(_peak_events(case["n"], seed)[0])
    point = _peak_point(case["n"])
    names = [v.name for v in _peak_pdf(case["bins"]).getParameters()]
    if case["family"] == "probs":
        return _peak_prob({k: _t(v) for k, v in point.items()}, x, case["bins"])[0].cpu().numpy()

    def nll(p):
        prob, total = _peak_prob(p, x, case["bins"])
        return -torch.log(prob).sum() + (total - x.numel() * torch.log(total))

    return [_value_grad(nll, names, [k for k in names if k != "c0"], point)]


def _composite_nll(p, counts):
    return -(counts * torch.log(_composite_density(p["alpha"], p["mu"], p["sigma"], p["fsig"]))).sum()


def _counts(events):
    return torch.bincount(torch.floor(_t(events[0]) / STEP).long() - KMIN, minlength=NK).double()


def _composite_names():
    return [v.name for v in _composite_pdf().getParameters()]


def _exact_composite(case, seed):
    counts = _counts(_composite_events(case["n"], seed))
    names = _composite_names()
    free = [k for k in names if k != "c0"]
    if case["family"] != "fit":
        return [_value_grad(lambda p: _composite_nll(p, counts), names, free, COMP_POINT)]
    # the minimum by Newton's method from the generation parameters
    v = _t([COMP[k] for k in free])
    f = lambda u: _composite_nll(dict(zip(free, u)), counts)  # noqa: E731
    for _ in range(12):
        u = v.clone().requires_grad_()
        grad = torch.autograd.grad(f(u), u)[0]
        step = torch.linalg.solve(torch.autograd.functional.hessian(f, v), grad)
        v = v - step
    at = dict(zip(free, v.tolist()), c0=1.0)
    return {"values": np.array([at[k] for k in names]), "errors": None, "fmin": np.array(float(f(v)))}


def _exact_toys(case, seed):
    names = _composite_names()
    free = [k for k in names if k != "c0"]
    pts = _toy_points(case, seed, names)
    out = []
    for t, events in enumerate(_toy_events(case, seed)):
        counts = _counts(events)
        out.append(_value_grad(lambda p: _composite_nll(p, counts), names, free, dict(zip(names, pts[t]))))
    return {"nll": np.array([o["nll"] for o in out]), "grad": np.stack([o["grad"] for o in out])}


# three-body amplitudes: relativistic Breit-Wigner with Blatt-Weisskopf barrier factors and Zemach spin factors

D3 = (W.C3_M, W.C3_MK, W.C3_MPI, W.C3_MPI0)


def _momentum(s, a, b):
    k1, k2 = 1 - (a + b) ** 2 / s, 1 - (a - b) ** 2 / s
    one = torch.ones_like(s)
    return 0.5 * torch.sqrt(s) * torch.where(k1 >= 0, torch.sqrt(k1.clamp(min=1e-300)), one) \
        * torch.where(k2 >= 0, torch.sqrt(k2.clamp(min=1e-300)), one)


def _momentum_mother(s, m, c):
    k1, k2 = 1 - (m + c) ** 2 / s, 1 - (m - c) ** 2 / s
    one = torch.ones_like(s)
    return 0.5 * s / m * torch.where(k1 >= 0, torch.sqrt(k1.clamp(min=1e-300)), one) \
        * torch.where(k2 >= 0, torch.sqrt(k2.clamp(min=1e-300)), one)


def _barrier(p, spin, r):
    q = r * r * p * p
    return 1 + q if spin == 1 else 9 + 3 * q + q * q


def _resonance(m12, m13, mass, width, spin, pair):
    m, d1, d2, d3 = D3
    m23 = m * m + d1 * d1 + d2 * d2 + d3 * d3 - m12 - m13
    s, a, b, c = [(m12, d1, d2, d3), (m13, d1, d3, d2), (m23, d2, d3, d1)][pair]
    rs = mass * mass
    pm, pn = _momentum(s, a, b), _momentum(rs, a, b)
    fr = frm = torch.ones_like(s)
    if spin:
        fr = _barrier(pn, spin, 1.5) / _barrier(pm, spin, 1.5)
        frm = _barrier(_momentum_mother(rs, m, c), spin, 5.0) / _barrier(_momentum_mother(s, m, c), spin, 5.0)
    x = rs - s
    y = rs * width * (pm / pn) ** (2 * spin + 1) * fr / torch.sqrt(s)
    f = torch.sqrt(fr) * torch.sqrt(frm) / (x * x + y * y)
    if spin:
        ma, mb, mc = [(d1, d2, d3), (d3, d1, d2), (d2, d3, d1)][pair]
        sac, sbc, sab = [(m13, m23, m12), (m23, m12, m13), (m12, m13, m23)][pair]
        mm, ab = m * m - mc * mc, ma * ma - mb * mb
        z = -((sbc - sac) + mm * ab / sab)
        if spin == 2:
            z = z * z - (sab - 2 * m * m - 2 * mc * mc + mm * mm / sab) * (sab - 2 * ma * ma - 2 * mb * mb
                                                                         + ab * ab / sab) / 3
        f = f * z
    return torch.complex(x * f, y * f)


def _inside(m12, m13):
    m, d1, d2, d3 = D3
    m23 = m * m + d1 * d1 + d2 * d2 + d3 * d3 - m12 - m13
    rt = torch.sqrt(m12)
    e1, e3 = 0.5 * (m12 - d2 * d2 + d1 * d1) / rt, 0.5 * (m * m - m12 - d3 * d3) / rt
    p1, p3 = torch.sqrt((e1 * e1 - d1 * d1).clamp(min=0)), torch.sqrt((e3 * e3 - d3 * d3).clamp(min=0))
    lo, hi = (e1 + e3) ** 2 - (p1 + p3) ** 2, (e1 + e3) ** 2 - (p1 - p3) ** 2
    return (m23 >= 0) & (m23 <= (m - d1) ** 2) & (m12 >= (d1 + d2) ** 2) & (m12 <= (m - d3) ** 2) & (m13 >= lo) \
        & (m13 <= hi)


def _dalitz_amplitude(m12, m13, p, n_res):
    total = 0
    for name, mass, width, spin, pair in W.C3_RESONANCES[:n_res]:
        c = torch.complex(p[f"{name}_amp_real"], p[f"{name}_amp_imag"])
        total = total + c * _resonance(m12, m13, p[f"{name}_mass"], p[f"{name}_width"], spin, int(pair))
    return total


def _dalitz_events(case, seed):
    pdf = _dalitz_pdf(case)
    p = {v.name: _t(v.value) for v in pdf.getParameters()}

    def weigh(x):
        inside = _inside(x[0], x[1])
        w = torch.zeros_like(x[0])
        a = _dalitz_amplitude(x[0][inside], x[1][inside], p, case["res"])
        w[inside] = a.real ** 2 + a.imag ** 2
        return w

    return _host(_with_number(_accept(case["n"], _generator(seed), _dalitz_points, weigh)))


def _exact_dalitz(case, seed):
    params = _dalitz_pdf(case).getParameters()
    names = [v.name for v in params]
    free = [v.name for v in params if not v.fixed]
    ev = _t(_dalitz_events(case, seed))
    w = 3.0 / case["bins"]
    c = w * (torch.arange(case["bins"], device="cuda", dtype=torch.float64) + 0.5)
    g12, g13 = (t.reshape(-1) for t in torch.meshgrid(c, c, indexing="ij"))
    ok = _inside(g12, g13)
    g12, g13 = g12[ok], g13[ok]

    def nll(p):
        a, g = (_dalitz_amplitude(u, v, p, case["res"]) for u, v in ((ev[0], ev[1]), (g12, g13)))
        norm = (g.real ** 2 + g.imag ** 2).sum() * w * w
        return -(torch.log(a.real ** 2 + a.imag ** 2)).sum() + ev.shape[1] * torch.log(norm)

    return [_value_grad(nll, names, free, _shape_values(params, v))
            for v in _points_of(params, 1 if case["family"] == "dalitz" else 2)]


# four-body amplitudes: vectors are stacked as (x, y, z, E)


def _four_vectors(v):
    m12, m34, c12, c34, phi = v[:5]
    m1, m2, m3, m4 = W.C5_MASSES
    mm = W.C5_M

    def pos_sqrt(x):
        return torch.sqrt(x.clamp(min=0))

    e = [(m12 ** 2 + m1 ** 2 - m2 ** 2) / (2 * m12), (m12 ** 2 - m1 ** 2 + m2 ** 2) / (2 * m12),
         (m34 ** 2 + m3 ** 2 - m4 ** 2) / (2 * m34), (m34 ** 2 - m3 ** 2 + m4 ** 2) / (2 * m34)]
    p1, p3 = pos_sqrt(e[0] ** 2 - m1 ** 2), pos_sqrt(e[2] ** 2 - m3 ** 2)
    s12, s34 = pos_sqrt(1 - c12 ** 2), pos_sqrt(1 - c34 ** 2)
    ed1, ed2 = (mm ** 2 + m12 ** 2 - m34 ** 2) / (2 * m12), (mm ** 2 - m12 ** 2 + m34 ** 2) / (2 * m34)
    b1, b2 = pos_sqrt(ed1 ** 2 - mm ** 2) / ed1, -pos_sqrt(ed2 ** 2 - mm ** 2) / ed2
    x = [c12 * p1, -c12 * p1, -c34 * p3, c34 * p3]
    y = [s12 * p1, -s12 * p1, -s34 * p3, s34 * p3]
    out = []
    for k in range(4):
        b = b1 if k < 2 else b2
        g = 1 / torch.sqrt(1 - b * b)
        out.append(torch.stack([g * (x[k] + b * e[k]), torch.cos(phi) * y[k] if k < 2 else y[k],
                                torch.sin(phi) * y[k] if k < 2 else torch.zeros_like(y[k]), g * (e[k] + b * x[k])]))
    return out


def _dot(a, b):
    return a[3] * b[3] - a[0] * b[0] - a[1] * b[1] - a[2] * b[2]


def _spin1(q, p):
    """q projected orthogonal to p."""
    return q - _dot(q, p) / _dot(p, p) * p


def _spin2_on(q, p, v):
    """The spin-2 Zemach tensor of q in the frame of p, contracted with v."""
    t = _spin1(q, p)
    f = _dot(t, t) / 3
    return t * _dot(t, v) - f * (v - p * (_dot(p, v) / _dot(p, p)))


def _epsilon(a, b, c):
    """The fully antisymmetric product of three vectors, in the sign convention of the reference's helper."""
    ax, ay, az, ae = a
    bx, by, bz, be = b
    cx, cy, cz, ce = c
    e = -ax * (by * cz - bz * cy) - ay * (bz * cx - bx * cz) - az * (bx * cy - by * cx)
    z = ax * (be * cy - by * ce) + ay * (bx * ce - be * cx) + ae * (by * cx - bx * cy)
    y = ax * (bz * ce - be * cz) + az * (be * cx - bx * ce) + ae * (bx * cz - bz * cx)
    x = ay * (be * cz - bz * ce) + az * (by * ce - be * cy) + ae * (bz * cy - by * cz)
    return torch.stack([x, y, z, e])


def _spin_factor(kind, p1, p2, p3, p4):
    S = G.SF_4Body
    if kind == S.DtoV1V2_V1toP1P2_V2toP3P4_S:
        return _dot(_spin1(p1 - p2, p1 + p2), _spin1(p3 - p4, p3 + p4))
    if kind == S.DtoV1V2_V1toP1P2_V2toP3P4_P:
        v1, v2 = p1 + p2, p3 + p4
        return -_dot(_epsilon(v1 + v2, _spin1(v1 - v2, v1 + v2), _spin1(p2 - p1, v1)), _spin1(p4 - p3, v2))
    if kind == S.DtoV1V2_V1toP1P2_V2toP3P4_D:
        v1, v2 = p1 + p2, p3 + p4
        return _dot(_spin1(p1 - p2, v1), _spin2_on(v1 - v2, v1 + v2, _spin1(p3 - p4, v2)))
    if kind == S.DtoAP1_AtoVP2_VtoP3P4:
        v = p3 + p4
        a = p2 + v
        u = _spin1(p3 - p4, v)
        return -_dot(_spin1(a - p1, p1 + a), -_spin1(u, a))
    if kind == S.DtoVS_VtoP1P2_StoP3P4:
        v, s = p1 + p2, p3 + p4
        return _dot(_spin1(v - s, v + s), _spin1(p1 - p2, v))
    raise ValueError(kind)


# daughters of a combination: the pair (or the pair inside a triple) and the odd one
_PAIRS = {0: ((0,), (1,)), 1: ((2,), (3,)), 2: ((0,), (2,)), 5: ((1,), (3,)), 6: ((0, 1), (2,)), 9: ((0, 1), (3,)),
          10: ((0, 3), (1,)), 11: ((1, 3), (0,)), 16: ((1, 3), (2,))}


def _mass_of(p, which):
    if len(which) == 1:
        return torch.full_like(p[0][0], W.C5_MASSES[which[0]])
    q = sum(p[k] for k in which)
    return torch.sqrt(_dot(q, q))


def _line_shape(p, ls, mass, width):
    first, second = _PAIRS[ls._Mpair]
    m1, m2, m = _mass_of(p, first), _mass_of(p, second), _mass_of(p, first + second)
    s, s0 = m * m, mass * mass
    q2 = (s - (m1 + m2) ** 2) * (s - (m1 - m2) ** 2) / (4 * s)
    q02 = (s0 - (m1 + m2) ** 2) * (s0 - (m1 - m2) ** 2) / (4 * s0)
    r2, length = ls._radius ** 2, ls._L
    q02_form = torch.where(q02 < 0, torch.zeros_like(q02), q02)
    q02 = torch.abs(q02)

    def form(z, z0):
        return torch.ones_like(z) if length == 0 else (1 + z0) / (1 + z)

    fr = form(q2 * r2, q02_form * r2)
    if isinstance(ls, G.Lineshapes.SBW):
        gamma_m = width
        gamma = torch.sqrt(s0 * (s0 + width * width))
        k = mass * width * gamma / torch.sqrt(s0 + gamma)
    else:
        gamma_m = width * torch.sqrt(q2 / q02) ** (2 * length + 1) * (mass / m) * form(q2 * r2, q02 * r2)
        gamma = mass * torch.sqrt(s0 + width * width)
        k = 2 * math.sqrt(2.0) / math.pi * mass * width * gamma / torch.sqrt(s0 + gamma)
    x, y = s0 - s, mass * gamma_m
    f = torch.sqrt(k * fr) / (x * x + y * y)
    return torch.complex(f * x, f * y)


def _four_amplitudes(pdf, v, p):
    """A_a for every amplitude of the model at the points v (5 columns), parameters p by name."""
    vec = _four_vectors(v)
    shapes, spins, out = {}, {}, []
    for amp in pdf.decayInfo.amplitudes:
        step_l, step_s = len(amp._LS) // amp._nPerm, len(amp._SF) // amp._nPerm
        total = 0
        for k in range(amp._nPerm):
            r = 1
            for ls in amp._LS[k * step_l:(k + 1) * step_l]:
                mass, width = (q.name for q in ls.getParameters())
                key = (type(ls).__name__, mass, width, ls._L, ls._Mpair)
                if key not in shapes:
                    shapes[key] = _line_shape(vec, ls, p[mass], p[width])
                r = r * shapes[key]
            for sf in amp._SF[k * step_s:(k + 1) * step_s]:
                key = (sf._SF, sf._P)
                if key not in spins:
                    spins[key] = _spin_factor(sf._SF, *(vec[i] for i in sf._P))
                r = r * spins[key]
            total = total + r
        out.append(total / math.sqrt(amp._nPerm))
    return out


def _four_total(pdf, v, p):
    return sum(torch.complex(p[a._ar.name], p[a._ai.name]) * x
               for a, x in zip(pdf.decayInfo.amplitudes, _four_amplitudes(pdf, v, p)))


def _fourbody_events(case, seed):
    pdf = _fourbody_pdf()
    p = {v.name: _t(v.value) for v in pdf.getParameters()}

    def weigh(x):
        a = _four_total(pdf, x, p)
        return a.real ** 2 + a.imag ** 2

    return _host(_with_number(_accept(case["n"], _generator(seed), _flat_four, weigh)))


def _exact_fourbody(case, seed):
    pdf = _fourbody_pdf()
    fixed = pdf._nondiff_all()
    params = pdf.getParameters()
    names = [v.name for v in params]
    free = [v.name for v in params if not v.fixed and id(v) not in fixed]
    ev = _t(_fourbody_events(case, seed))
    ne = _norm_events(case["norm"], seed)
    parts = ne.split(250000, 1)

    def one(value):
        p = {k: _t(float(value[k]), k in free) for k in names}
        leaf = [p[k] for k in names if k in free]
        a = _four_total(pdf, ev, p)
        nll = -(torch.log(a.real ** 2 + a.imag ** 2)).sum()
        g = [x.detach() for x in torch.autograd.grad(nll, leaf)]
        norm, dn = 0.0, [torch.zeros_like(x) for x in g]
        for part in parts:
            a = _four_total(pdf, part, p)
            s = (a.real ** 2 + a.imag ** 2).sum()
            dn = [x + y.detach() for x, y in zip(dn, torch.autograd.grad(s, leaf))]
            norm = norm + s.detach()
        n = ev.shape[1]
        value = nll.detach() + n * torch.log(norm / ne.shape[1])
        return {"nll": float(value), "grad": np.array([float(x + n * y / norm) for x, y in zip(g, dn)])}

    return [one(_shape_values(params, v)) for v in _points_of(params, 2)]


def exact(case, seed):
    family = case["family"]
    if family == "decay":
        x = _t(_decay_events(case["n"], seed)[0])

        def nll(p):
            return -(p["alpha"] * x).sum() + x.numel() * torch.log((torch.exp(10 * p["alpha"]) - 1) / p["alpha"])

        return [_value_grad(nll, ["alpha"], ["alpha"], {"alpha": -0.3})]
    if family in ("peak", "probs"):
        return _exact_peak(case, seed)
    if family in ("composite", "new-data", "fit"):
        return _exact_composite(case, seed)
    if family == "toys":
        return _exact_toys(case, seed)
    if family in ("dalitz", "dalitz-shapes"):
        return _exact_dalitz(case, seed)
    return _exact_fourbody(case, seed)
