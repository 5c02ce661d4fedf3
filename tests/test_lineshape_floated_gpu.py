"""Four-body line shapes of the mixed engine (floated ones: gf_lineshape_k, and the dual numbers of shapes whose thresholds
move with the event) against the FP64 engine: at and just above the thresholds, and over orbital
angular momenta, form factors, constant widths, poles below threshold and daughter combinations.  Amplitudes of one line
shape and no spin factor, so that the cached wave is the line shape itself."""
import numpy as np
import pytest

import goofit_gb300 as G
from goofit_gb300 import phasespace
from goofit_gb300 import workloads as W

pytestmark = pytest.mark.gpu

P, FF, RBW, SBW = G.DP4Pair, G.FF, G.Lineshapes.RBW, G.Lineshapes.SBW
M = W.C5_MASSES


def _model(shapes, floated=True):
    """One amplitude per (kind, mass, width, L, pair, form factor), the first one's coefficient fixed."""
    obs = [G.Observable("m12", 0, 3), G.Observable("m34", 0, 3), G.Observable("cos12", -1, 1), G.Observable("cos34", -1, 1),
           G.Observable("phi", -3.5, 3.5), G.EventNumber("eventNumber")]
    d = G.DecayInfo4()
    d.particle_masses = [W.C5_M] + M
    d.meson_radius = 1.5
    for k, (kind, mass, width, L, pair, ff) in enumerate(shapes):
        m, w = G.Variable(f"m{k}", mass, 0.01, 0, 0), G.Variable(f"w{k}", width, 0.01, 0, 0)
        m.setFixed(not floated)
        w.setFixed(not floated)
        re, im = G.Variable(f"re{k}", 1.0 - 0.1 * k, 0.01, 0, 0), G.Variable(f"im{k}", 0.3 * k, 0.01, 0, 0)
        re.setFixed(k == 0)
        im.setFixed(k == 0)
        one = G.SpinFactor("one", G.SF_4Body.ONE, W.C5_M, 0, 1, 2, 3)
        d.amplitudes.append(G.Amplitude(f"a{k}", re, im, [kind(f"ls{k}", m, w, L, pair, ff)], [one], 1))
    eff = G.PolynomialPdf("eff", obs[:2], [G.Variable("one", 1)], [G.Variable("z0", 0), G.Variable("z1", 0)], 0)
    return G.Amp4Body("p", obs, d, eff, 1000, 5)


def _engine(precision, pdf, events, norm):
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    mask = [0 if (v.fixed or id(v) in nd) else 1 for v in params]
    eng = G.Engine(precision)
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params), mask)
    eng.set_norm_events(0, norm)
    eng.upload(np.vstack([events, np.arange(events.shape[1])]))
    p = np.array([v.value for v in params])
    eng.set_params(p)
    return eng, p, [v.name for v in params]


def _events(n, seed):
    return np.ascontiguousarray(phasespace.norm_events(W.C5_M, M, n, seed))


DISTANCES = np.array([0.0, 1e-9, 5e-9, 1e-8, 2e-8, 3e-8, 4e-8, 6e-8, 1e-7, 1e-6])


def _threshold_events():
    """Events whose m12, then whose m34, lies at DISTANCES above its threshold, before ordinary ones."""
    x = _events(400, 3)
    k = len(DISTANCES)
    x[0, :k] = (M[0] + M[1]) + DISTANCES
    x[1, :k] = np.minimum(x[1, :k], 1.2)
    x[1, k:2 * k] = (M[2] + M[3]) + DISTANCES
    x[0, k:2 * k] = np.minimum(x[0, k:2 * k], 0.9)
    return x


def test_at_and_just_above_the_threshold():
    shapes = [(RBW, 0.775, 0.149, 0, P.M_12, FF.BL_Prime), (RBW, 0.892, 0.1, 1, P.M_34, FF.BL_Prime),
              (RBW, 0.6, 0.3, 1, P.M_12, FF.BL), (RBW, 0.8, 0.3, 2, P.M_34, FF.BL2)]
    x = _threshold_events()
    ref, p, _ = _engine("fp64", _model(shapes, floated=False), x, x[:, 20:])
    eng, _, _ = _engine("mixed", _model(shapes), x, x)
    for a in range(len(shapes)):
        want, got = ref.amp3_cached_wave(0, a), eng.amp3_cached_wave(0, a)
        # value: some 20 FP32 operations of relative 2^-24 on differences formed in pairs
        assert np.all(np.abs(got - want) <= 2e-6 * np.abs(want)), a
        # the imaginary part falls as q^(2L+1): pairs hold s to 2^-45, 2e-15 of a difference of 5e-10 at 1e-9 GeV above
        # threshold, and L = 2 takes its 2.5th power; below 1e-9 the difference itself is rounding
        at = (np.arange(x.shape[1]) % len(DISTANCES) != 0) | (np.arange(x.shape[1]) >= 2 * len(DISTANCES))
        assert np.all(np.abs(got.imag - want.imag)[at] <= 5e-5 * np.abs(want.imag)[at] + 1e-30), a
    nll, grad = eng.nll_grad(p)
    assert np.isfinite(nll) and np.all(np.isfinite(grad))
    # the same without the 20 threshold events (a dropped event would change the difference by its own -log P, of order one)
    some, _, _ = _engine("mixed", _model(shapes), x[:, 20:], x)
    r64, _, _ = _engine("fp64", _model(shapes, floated=False), x[:, :20], x[:, 20:])
    probs = r64.eval_events()  # normalised by r64's own integral
    assert np.all(probs > 0)
    want = -np.log(probs).sum() + 20 * (np.log(r64.normalize()[1][0]) - np.log(eng.normalize()[1][0]))
    # per event: FP32 log of a density of relative error 1e-6
    assert abs((nll - some.nll(p)) - want) <= 20 * 1e-5


def test_fixed_shapes_at_and_just_above_the_threshold():
    shapes = [(RBW, 0.775, 0.149, 0, P.M_12, FF.BL_Prime), (RBW, 0.892, 0.1, 1, P.M_34, FF.BL_Prime),
              (RBW, 0.6, 0.3, 1, P.M_12, FF.BL2), (RBW, 0.8, 0.3, 2, P.M_34, FF.BL2)]
    x = _threshold_events()
    ref, p, _ = _engine("fp64", _model(shapes, floated=False), x, x[:, 20:])
    eng, _, _ = _engine("mixed", _model(shapes, floated=False), x, x)
    for a in range(len(shapes)):
        want, got = ref.amp3_cached_wave(0, a), eng.amp3_cached_wave(0, a)
        # these shapes subtract in FP32: q^2 is off by 2^-23 s at most, 1e-4 GeV of q at the threshold, against a pole term
        # of 0.5 GeV^2 and a width term of m Gamma q / q0 < 0.4 GeV q
        assert np.all(np.abs(got - want) <= 5e-4 * np.abs(want).max()), a
    nll, grad = eng.nll_grad(p)
    assert np.isfinite(nll) and np.all(np.isfinite(grad))


def _triple_events(cos34):
    """Events in which daughter 3 moves with the pair (1,2), so that m123 = m12 + m3; where it moves against it, for the
    other sign of cos34."""
    m12 = np.linspace(M[0] + M[1] + 0.01, W.C5_M - M[2] - M[3] - 0.2, 200)
    cl = m12 + M[2]
    p = np.sqrt((W.C5_M ** 2 - (cl + M[3]) ** 2) * (W.C5_M ** 2 - (cl - M[3]) ** 2)) / (2 * W.C5_M)
    e3, e4 = M[2] * np.sqrt(1 + (p / cl) ** 2), np.sqrt(M[3] ** 2 + p ** 2)
    m34 = np.sqrt((e3 + e4) ** 2 - (p * m12 / cl) ** 2)
    return np.vstack([m12, m34, np.full(200, 0.3), np.full(200, cos34), np.linspace(-3, 3, 200)])


@pytest.mark.parametrize("floated", [True, False])
def test_triples_at_their_threshold(floated):
    # poles above every event's mass (1.53 GeV): the width vanishes at the threshold, and a pole there would diverge
    shapes = [(RBW, 1.8, 0.3, 0, P.M_12_3, FF.BL_Prime), (RBW, 1.75, 0.3, 1, P.M_12_3, FF.BL2), (SBW, 1.8, 0.3, 1, P.M_12_3, FF.BL)]
    x = np.hstack([_triple_events(c) for c in (1.0, -1.0)])
    near = np.hstack([_triple_events(c) for c in (1 - 1e-9, -1 + 1e-9)])
    ref, p, _ = _engine("fp64", _model(shapes, floated=False), near, _events(400, 3))
    eng, _, _ = _engine("mixed", _model(shapes, floated), x, np.hstack([x, _events(400, 3)]))
    for a in range(len(shapes)):
        want, got = ref.amp3_cached_wave(0, a), eng.amp3_cached_wave(0, a)
        # the squared mass from FP32 four-vectors: a few units of 2^-24 M^2, 1e-6 GeV^2, so q is off by up to 1e-3 GeV
        # there, and the wave by m Gamma q / q0 (the last shape's form factor: q r) over a pole term of 0.7 GeV^2
        assert np.all(np.isfinite(got)) and np.all(np.abs(got - want) <= 5e-3 * np.abs(want).max()), a
    nll, grad = eng.nll_grad(p)
    assert np.isfinite(nll) and np.all(np.isfinite(grad))


FORMS = [
    [(RBW, 0.775, 0.149, 2, P.M_12, FF.BL_Prime), (RBW, 0.892, 0.1, 1, P.M_34, FF.BL)],
    [(RBW, 0.775, 0.149, 1, P.M_12, FF.BL2), (RBW, 1.0, 0.2, 2, P.M_34, FF.BL)],
    [(RBW, 0.775, 0.149, 1, P.M_12, FF.One), (RBW, 1.0, 0.2, 2, P.M_34, FF.BL2)],
    [(SBW, 0.775, 0.149, 1, P.M_12, FF.BL_Prime), (SBW, 0.892, 0.1, 2, P.M_34, FF.BL)],
    [(SBW, 0.775, 0.149, 2, P.M_12, FF.BL2), (SBW, 0.892, 0.1, 1, P.M_34, FF.One)],
    [(RBW, 0.2, 0.3, 1, P.M_12, FF.BL_Prime), (RBW, 0.5, 0.3, 2, P.M_34, FF.BL_Prime)],  # poles below threshold
    [(RBW, 0.2, 0.3, 0, P.M_12, FF.BL_Prime), (SBW, 0.5, 0.3, 1, P.M_34, FF.BL_Prime)],
    [(RBW, 0.9, 0.2, 2, P.M_13, FF.BL_Prime), (RBW, 0.7, 0.2, 1, P.M_24, FF.BL)],
    [(RBW, 0.7, 0.2, 1, P.M_14, FF.BL2), (SBW, 0.9, 0.2, 2, P.M_23, FF.BL_Prime)],
    [(SBW, 1.2, 0.3, 1, P.M_12_3, FF.BL), (SBW, 1.1, 0.3, 2, P.M_24_1, FF.BL2)],
    [(SBW, 1.2, 0.3, 1, P.M_12_3, FF.BL_Prime), (RBW, 1.1, 0.3, 1, P.M_23_4, FF.BL_Prime)],  # dual numbers
]


@pytest.mark.parametrize("shapes", FORMS)
def test_every_form_matches_the_fp64_engine(shapes):
    # a reference shape first, so that neither of the two is the overall scale
    shapes = [(RBW, 0.85, 0.25, 0, P.M_12, FF.BL_Prime)] + shapes
    x, norm = _events(64, 4), _events(4096, 5)
    ref, p, names = _engine("fp64", _model(shapes), x, norm)
    eng, _, _ = _engine("mixed", _model(shapes), x, norm)
    # pairs (1,2) and (3,4): FP32 arithmetic on the event's own masses.  Others: s from FP32 four-vectors, a few units of
    # 2^-24 E^2 = 2e-7 GeV^2 each, against a pole term of m Gamma >= 0.14 GeV^2
    tol = 3e-6 if all(s[4] in (P.M_12, P.M_34) for s in shapes) else 2e-5
    for a in range(len(shapes)):
        want, got = ref.amp3_cached_wave(0, a), eng.amp3_cached_wave(0, a)
        assert np.all(np.isfinite(want)) and np.all(np.abs(got - want) <= tol * np.abs(want).max()), a
    n0, g0 = ref.nll_grad(p)
    n1, g1 = eng.nll_grad(p)
    assert abs(n1 - n0) <= 64 * 5 * tol
    # an event's logarithmic derivative by a mass or width is at most about 2 / width, and the same tolerance applies to it
    scale = 2 / min(s[2] for s in shapes)
    assert eng.grad_params == ref.grad_params
    assert np.all(np.abs(g1 - g0) <= 64 * 5 * tol * scale), [names[i] for i in eng.grad_params]
