"""The derivative rows of the one-pass integrals (H_ab = sum dA_a conj(A_b) e) against the CUDA-core integrals, through the
gradient of a few events, in which the normalisation's derivative is not scaled up: each entry within the bound of its own
row."""
import numpy as np
import pytest

import goofit_gb300 as G
from goofit_gb300 import phasespace
from goofit_gb300 import workloads as W

pytestmark = pytest.mark.gpu

N = 8


def _three(n_res, floated, bins):
    m12, m13 = G.Observable("m12", 0.0, 3.0), G.Observable("m13", 0.0, 3.0)
    m12.setNumBins(bins)
    m13.setNumBins(bins)
    d = G.DecayInfo3()
    d.motherMass, d.daug1Mass, d.daug2Mass, d.daug3Mass = W.C3_M, W.C3_MK, W.C3_MPI, W.C3_MPI0
    d.meson_radius, d.mother_meson_radius = 1.5, 5.0
    for k in range(n_res):
        m, w = G.Variable(f"m{k}", 0.7 + 0.03 * k), G.Variable(f"w{k}", 0.1)
        m.setFixed(k >= floated)
        w.setFixed(k >= floated)
        # the later ones a thousand times smaller: a lost row would be small as well
        d.add_resonance(G.RBW(f"r{k}", G.Variable(f"re{k}", 1.0 if k < 2 else 1e-3, 0.01, 0, 0),
                              G.Variable(f"im{k}", 0.1 * (k % 5) * (1.0 if k < 2 else 1e-3), 0.01, 0, 0), m, w, k % 2,
                              int((G.PAIR_12, G.PAIR_13, G.PAIR_23)[k % 3])))
    x = np.random.Generator(np.random.PCG64(3)).uniform(0.3, 2.8, (2, 8000))
    s = W.C3_M ** 2 + W.C3_MK ** 2 + W.C3_MPI ** 2 + W.C3_MPI0 ** 2
    x = x[:, (s - x.sum(0) > 0.2) & (x.sum(0) > 1.2)][:, :N]
    return G.Amp3Body("p", m12, m13, G.EventNumber("eventNumber"), d), np.vstack([x, np.arange(N)]), None, n_res


def _four(points):
    pdf = W.c5_model(1000, float_lineshapes=True)[0]
    ev = phasespace.norm_events(W.C5_M, W.C5_MASSES, N + points, 11)
    return pdf, np.vstack([ev[:, :N], np.arange(N)]), np.ascontiguousarray(ev[:, N:]), 6


def _evaluate(make, args):
    pdf, events, norm, n = make(*args)
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    eng = G.Engine("mixed")
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params),
                 [0 if (v.fixed or id(v) in nd) else 1 for v in params])
    if norm is not None:
        eng.set_norm_events(0, norm)
    eng.upload(events)
    p = np.array([v.value for v in params])
    grad = eng.nll_grad(p)[1]
    coef = np.array([p[nodes[0]["params"][2 * a]] + 1j * p[nodes[0]["params"][2 * a + 1]] for a in range(n)])
    out = dict(zip([params[i].name for i in eng.grad_params], grad)), eng.amp3_integrals(0, n), coef, {v.name: v.value for v in params}
    eng.close()
    return out


@pytest.mark.parametrize("make,args", [
    (_three, (3, 3, 61)), (_three, (8, 4, 61)), (_three, (10, 10, 40)), (_three, (16, 8, 40)), (_three, (28, 2, 40)),
    (_four, (1001,)), (_four, (60001,)),
])
def test_every_derivative_row(make, args, monkeypatch):
    monkeypatch.delenv("GF_GRAM", raising=False)
    grad, integrals, coef, value = _evaluate(make, args)
    monkeypatch.setenv("GF_GRAM", "cuda")
    grad0, ref, _, _ = _evaluate(make, args)
    # the events' part is the same; d log Q = 2 Re sum_ab c_a conj(c_b) H_ab / Q.  Each H_ab within 2e-6 sqrt(H_aa I_bb) (split
    # TF32 products 2^-21, truncated accumulations, FP32 sums of the other kernel), with |dA_a| <= 2 / width |A_a| on average;
    # Q within 2e-6 of the same sum of I alone
    size = np.abs(coef) * np.sqrt(np.abs(np.diag(ref)))
    Q = (coef[:, None] * coef.conj()[None, :] * ref).sum().real
    common = 2e-6 * size.sum() ** 2 / Q
    assert grad.keys() == grad0.keys()
    seen = 0
    for name, g in grad.items():
        if make is _three and name[0] in "mw":
            own, width = size[int(name[1:])], 0.1
        elif make is _four and name.endswith(("_mass", "_width")):
            own, width = size.sum(), value[name.rsplit("_", 1)[0] + "_width"]
        else:
            continue
        seen += 1
        # two permutations of a four-body amplitude carry the shape twice
        rows = 2 * own * size.sum() / Q * (2 / width) * (1 if make is _three else 2)
        assert abs(g - grad0[name]) <= N * rows * (2e-6 + common), name
    assert seen == (2 * args[1] if make is _three else 10)
