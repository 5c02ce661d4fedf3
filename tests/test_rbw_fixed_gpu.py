"""A resonance with fixed mass and width beside a floated one (gf_rbw_k, the mixed engine) and in a tree without floated
shapes (gf_rbw) against the FP64 engine, over spins, daughter pairs, normalisation, symmetrisation and a pole below
threshold, and the gradient by the coefficients."""
import numpy as np
import pytest

import goofit_gb300 as G
from goofit_gb300 import workloads as W

pytestmark = pytest.mark.gpu

N = 4099


def _engine(precision, floated, spin, pair, norm, sym, mass):
    m12, m13 = G.Observable("m12", 0.0, 3.0), G.Observable("m13", 0.0, 3.0)
    m12.setNumBins(97)
    m13.setNumBins(97)
    d = G.DecayInfo3()
    d.motherMass, d.daug1Mass, d.daug2Mass, d.daug3Mass = W.C3_M, W.C3_MK, W.C3_MPI, W.C3_MPI0
    # the unnormalised spin-2 barrier 13 q / (q - 3)^2 + 9 q^2, q = (r p)^2, has a pole that radii of 1.5 and 5 would put among
    # the events; q < 0.2 with these, and the barrier leaves a tenth of the width, which is therefore ten times larger
    barrier = spin == 2 and not norm
    d.meson_radius, d.mother_meson_radius = (0.4, 0.4) if barrier else (1.5, 5.0)
    m, w = G.Variable("m", 0.892), G.Variable("w", 0.05)
    m.setFixed(not floated)
    w.setFixed(not floated)
    d.add_resonance(G.RBW("beside", G.Variable("re0", 1.0), G.Variable("im0", 0.0), m, w, 1, int(G.PAIR_12)))
    re, im = G.Variable("re1", 0.6, 0.01, 0, 0), G.Variable("im1", -0.4, 0.01, 0, 0)
    fm, fw = G.Variable("fm", mass), G.Variable("fw", 1.2 if barrier else 0.12)
    fm.setFixed(True)
    fw.setFixed(True)
    d.add_resonance(G.RBW("fixed", re, im, fm, fw, spin, int(pair), norm, sym))
    pdf = G.Amp3Body("p", m12, m13, G.EventNumber("eventNumber"), d)
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    eng = G.Engine(precision)
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params),
                 [0 if (v.fixed or id(v) in nd) else 1 for v in params])
    x, y = np.random.Generator(np.random.PCG64(5)).uniform(0.0, 3.0, (2, N))
    eng.upload(np.vstack([x, y, np.arange(N, dtype=np.float64)]))
    p = np.array([v.value for v in params])
    eng.set_params(p)
    return eng, p, [v.name for v in params]


@pytest.mark.parametrize("floated", [True, False])
@pytest.mark.parametrize("spin,pair,norm,sym,mass", [
    (0, G.PAIR_12, True, False, 1.2), (1, G.PAIR_13, True, False, 0.8), (2, G.PAIR_23, True, False, 1.275),
    (0, G.PAIR_23, False, False, 0.9), (1, G.PAIR_23, False, False, 0.775), (2, G.PAIR_12, False, True, 1.3),
    (2, G.PAIR_13, False, False, 1.1), (1, G.PAIR_12, True, True, 0.9), (0, G.PAIR_13, True, False, 0.55),
])
def test_fixed_resonance_matches_the_fp64_engine(spin, pair, norm, sym, mass, floated):
    ref, p, names = _engine("fp64", floated, spin, pair, norm, sym, mass)
    eng, _, _ = _engine("mixed", floated, spin, pair, norm, sym, mass)
    want, got = ref.amp3_cached_wave(0, 1), eng.amp3_cached_wave(0, 1)
    assert 0 < (want != 0).sum() < N and np.array_equal(got != 0, want != 0)
    # some 40 FP32 operations of 2^-24 in products and quotients, and the cancellation of the spin factor's terms against
    # its largest values
    med = np.median(np.abs(want[want != 0]))
    assert np.all(np.abs(got - want) <= 5e-6 * np.maximum(np.abs(want), med))
    # a misplaced value moves an event by more than all FP32 roundings of the sums together
    n0, g0 = ref.nll_grad(p)
    n1, g1 = eng.nll_grad(p)
    assert abs(n1 - n0) <= 1e-6 * abs(n0)
    for i, a, b in zip(eng.grad_params, g1, g0):
        if names[i] in ("re1", "im1"):
            # per event at most 2 |A_1| / |T| by the coefficient, with events of small |T| at most ten times the median
            assert abs(a - b) <= 5e-6 * N * 10 / abs(0.6 - 0.4j)
