"""gf_ampng (amplitudes and tensor-core contraction in one pass) against the CUDA-core integrals of the same engine, over
its layouts: slices of 32 and 64 real columns, weighted (Amp3Body) and unweighted (Amp4Body), 1 to 31 amplitudes, with
and without derivative columns, and point counts around one tile of 128."""
import numpy as np
import pytest

import goofit_gb300 as G
from goofit_gb300 import phasespace
from goofit_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _three(n_res, floated, bins):
    pdf = W.c3_model(bins, n_res)[0]
    for name, *_ in W.C3_RESONANCES[:floated]:
        for v in pdf.getParameters():
            if v.name in (f"{name}_mass", f"{name}_width"):
                v.setFixed(False)
    rng = np.random.Generator(np.random.PCG64(3))
    x = rng.uniform(0.3, 2.8, (2, 8000))
    s = W.C3_M ** 2 + W.C3_MK ** 2 + W.C3_MPI ** 2 + W.C3_MPI0 ** 2
    x = x[:, (s - x.sum(0) > 0.2) & (x.sum(0) > 1.2)][:, :1500]
    return pdf, np.vstack([x, np.arange(x.shape[1])]), None


def _many(n_res, floated, bins):
    """n_res resonances: value columns up to the widest that one slice holds."""
    m12, m13 = G.Observable("m12", 0.0, 3.0), G.Observable("m13", 0.0, 3.0)
    m12.setNumBins(bins)
    m13.setNumBins(bins)
    d = G.DecayInfo3()
    d.motherMass, d.daug1Mass, d.daug2Mass, d.daug3Mass = W.C3_M, W.C3_MK, W.C3_MPI, W.C3_MPI0
    d.meson_radius, d.mother_meson_radius = 1.5, 5.0
    for k in range(n_res):
        m, w = G.Variable(f"m{k}", 0.7 + 0.03 * k), G.Variable(f"w{k}", 0.1)
        m.setFixed(k >= floated)
        d.add_resonance(G.RBW(f"r{k}", G.Variable(f"re{k}", 1.0, 0.01, 0, 0), G.Variable(f"im{k}", 0.1 * (k % 5), 0.01, 0, 0), m, w,
                              k % 2, int((G.PAIR_12, G.PAIR_13, G.PAIR_23)[k % 3])))
    pdf = G.Amp3Body("p", m12, m13, G.EventNumber("eventNumber"), d)
    return pdf, _three(2, 0, 40)[1], None


def _four(floated, points):
    pdf = W.c5_model(1000, float_lineshapes=floated)[0]
    ev = phasespace.norm_events(W.C5_M, W.C5_MASSES, 1500 + points, 11)
    return pdf, np.vstack([ev[:, :1500], np.arange(1500)]), np.ascontiguousarray(ev[:, 1500:])


def _evaluate(make, args):
    pdf, events, norm = make(*args)
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    mask = [0 if (v.fixed or id(v) in nd) else 1 for v in params]
    eng = G.Engine("mixed")
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params), mask)
    if norm is not None:
        eng.set_norm_events(0, norm)
    eng.upload(events)
    p = np.array([v.value for v in params]) * (1 + 0.01 * np.cos(np.arange(len(params))) * np.array(mask))
    nll, grad = eng.nll_grad(p)
    n = 6 if make is _four else args[0]
    out = nll, grad, eng.amp3_integrals(0, n), n
    eng.close()
    return out


@pytest.mark.parametrize("make,args", [
    (_three, (8, 0, 61)), (_three, (8, 4, 61)), (_three, (8, 8, 40)), (_three, (1, 1, 40)), (_three, (3, 2, 19)),
    (_four, (False, 1000)), (_four, (True, 1)), (_four, (True, 127)), (_four, (True, 128)), (_four, (True, 129)),
    (_four, (True, 60001)), (_many, (9, 0, 40)), (_many, (16, 0, 40)), (_many, (17, 2, 40)), (_many, (31, 1, 40)),
])
def test_one_pass_integrals_match_the_cuda_core_integrals(make, args, monkeypatch):
    monkeypatch.delenv("GF_GRAM", raising=False)
    nll, grad, integrals, n = _evaluate(make, args)
    monkeypatch.setenv("GF_GRAM", "cuda")
    nll0, grad0, ref, _ = _evaluate(make, args)
    # products of split-TF32 pairs carry 2^-21, four accumulations that round towards zero 4 x 2^-23, the other
    # kernel's FP32 products and per-thread sums at most as much again: 2e-6 of sqrt(I_ii I_jj)
    d = np.sqrt(np.abs(np.diag(ref)))
    assert np.all(np.abs(integrals - ref) <= 2e-6 * np.outer(d, d))
    np.testing.assert_array_equal(integrals, integrals.conj().T)
    # the same errors in N and dN/dp: N is a sum of n^2 such terms, and a line shape's logarithmic derivative is at
    # most 2 / width < 40 in these models; 1500 events
    assert abs(nll - nll0) <= 1500 * 2e-6 * n
    np.testing.assert_allclose(grad, grad0, rtol=2e-6, atol=1500 * 2e-6 * n * 40)
