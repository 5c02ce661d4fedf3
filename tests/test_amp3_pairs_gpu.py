"""The floated resonances of Amp3Body (point parts and chain rule in pairs of FP32 values, or FP64) against the FP64
engine's fixed-resonance formula, over spins, daughter pairs, normalisation, symmetrisation and a pole below threshold,
at points that include the kinematic boundary."""
import numpy as np
import pytest

import goofit_gb300 as G
from goofit_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _model(spin, pair, norm, sym, mass, floated):
    m12, m13 = G.Observable("m12", 0.0, 3.0), G.Observable("m13", 0.0, 3.0)
    m12.setNumBins(97)
    m13.setNumBins(97)
    d = G.DecayInfo3()
    d.motherMass, d.daug1Mass, d.daug2Mass, d.daug3Mass = W.C3_M, W.C3_MK, W.C3_MPI, W.C3_MPI0
    d.meson_radius, d.mother_meson_radius = 1.5, 5.0
    d.add_resonance(G.RBW("ref", G.Variable("ref_re", 1.0), G.Variable("ref_im", 0.0), G.Variable("ref_m", 0.892),
                          G.Variable("ref_w", 0.05), 1, int(G.PAIR_12)))
    m, w = G.Variable("m", mass), G.Variable("w", 0.12)
    m.setFixed(not floated)
    w.setFixed(not floated)
    d.add_resonance(G.RBW("res", G.Variable("re", 0.6), G.Variable("im", -0.4), m, w, spin, int(pair), norm, sym))
    return G.Amp3Body("p", m12, m13, G.EventNumber("eventNumber"), d)


def _events(n=4099):
    rng = np.random.Generator(np.random.PCG64(5))
    x, y = rng.uniform(0.0, 3.0, (2, n))
    # a third of the points within 1e-3 of the upper limit of m13, on both sides
    k = n // 3
    e1 = 0.5 * (x[:k] - W.C3_MPI ** 2 + W.C3_MK ** 2) / np.sqrt(x[:k])
    e3 = 0.5 * (W.C3_M ** 2 - x[:k] - W.C3_MPI0 ** 2) / np.sqrt(x[:k])
    p1, p3 = (np.sqrt(np.maximum(e * e - q * q, 0)) for e, q in ((e1, W.C3_MK), (e3, W.C3_MPI0)))
    y[:k] = np.clip((e1 + e3) ** 2 - (p1 - p3) ** 2 + rng.uniform(-1e-3, 1e-3, k), 0, 3)
    return np.vstack([x, y, np.arange(n, dtype=np.float64)])


def _engine(precision, *model, floated):
    pdf = _model(*model, floated)
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    eng = G.Engine(precision)
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params),
                 [0 if (v.fixed or id(v) in nd) else 1 for v in params])
    eng.upload(_events())
    return eng, params


@pytest.mark.parametrize("spin,pair,norm,sym,mass", [
    (0, G.PAIR_12, True, False, 1.2), (1, G.PAIR_13, True, False, 0.8), (2, G.PAIR_23, True, False, 1.275),
    (1, G.PAIR_23, False, False, 0.775), (2, G.PAIR_12, False, True, 1.3), (1, G.PAIR_12, True, True, 0.9),
    (0, G.PAIR_13, True, False, 0.55),  # the pole lies below the pair's threshold
])
def test_floated_resonance_matches_the_fixed_formula(spin, pair, norm, sym, mass):
    model = (spin, pair, norm, sym, mass)
    ref, params = _engine("fp64", *model, floated=False)
    p0 = np.array([v.value for v in params])
    ref.set_params(p0)
    want = ref.amp3_cached_wave(0, 1)
    im, iw = ([v.name for v in params].index(k) for k in ("m", "w"))

    def nll(q, i, h):
        q = q.copy()
        q[i] += h
        return ref.nll(q)

    inside = want != 0
    assert 0 < inside.sum() < len(want)
    # central differences of the fixed FP64 formula: truncation ~h^2, rounding ~1e-15 |NLL| / h
    h = 1e-5
    fd = np.array([(nll(p0, i, h) - nll(p0, i, -h)) / (2 * h) for i in (im, iw)])
    scale = np.abs(fd).max() + np.abs(ref.nll(p0))
    # FP64: the same numbers in another order of operations.  Mixed: pairs carry 2^-44 per operation, some 60
    # operations, amplified by up to ~1e3 at the momentum thresholds; the stored wave rounds to FP32 (2^-24)
    for precision, tol, gtol in (("fp64", 1e-11, 1e-6), ("mixed", 1.5e-7, 2e-5)):
        eng, _ = _engine(precision, *model, floated=True)
        eng.set_params(p0)
        got = eng.amp3_cached_wave(0, 1)
        assert np.array_equal(got != 0, inside)  # the same side of the boundary for every point
        assert np.all(np.abs(got - want) <= tol * np.abs(want) + tol * 1e-3 * np.abs(want).max())
        g = eng.nll_grad(p0)[1]
        g = np.array([g[eng.grad_params.index(i)] for i in (im, iw)])
        assert np.all(np.abs(g - fd) <= gtol * scale)
