"""Normalisation grids of at most 4096 bins are summed by every CTA of the one-launch evaluation; larger ones, and the
separate launches (GF_FUSED=0), spread the bins over CTAs.  Both sides of the limit and of the CTA's 256 threads, one
and two grids, against the separate launches: the factors agree to about 1e-14, so the NLL differs by the last bits of a
few events' FP32 logarithms (1e-9 relative allows every event one more rounding of 2^-24 in a hundred), and so do the
gradient sums, here within 1e-6 of the events' root sum of squares or of their value."""
import numpy as np
import pytest

import goofit_gb300 as gf

pytestmark = pytest.mark.gpu


def _pdf(bins, two):
    x = gf.Observable("x", 0.0, 10.0)
    x.setNumBins(bins)
    g = gf.GaussianPdf("g", x, gf.Variable("m", 5.0, 0.01, 4, 6), gf.Variable("s", 0.5, 0.01, 0.1, 2))

    def poly(name, c):
        return gf.PolynomialPdf(name, x, [gf.Variable(name + "0", 1.0), gf.Variable(name + "1", c, 0.001, -0.05, 0.2),
                                          gf.Variable(name + "2", 0.002, 0.0001, -0.01, 0.01)], 0)

    parts = [g, poly("p", -0.04)] + ([poly("r", 0.1)] if two else [])
    return gf.AddPdf("sum", [gf.Variable(f"n{k}", 3000.0 + 500 * k, 10, 0, 1e6) for k in range(len(parts))], parts)


def _evaluate(bins, two):
    pdf = _pdf(bins, two)
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    eng = gf.Engine("mixed")
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params),
                 [0 if (v.fixed or id(v) in nd) else 1 for v in params])
    rng = np.random.Generator(np.random.PCG64(4))
    eng.upload(np.clip(np.where(rng.random(7001) < 0.4, rng.normal(5, 0.5, 7001), rng.uniform(0, 10, 7001)), 0, 10).reshape(1, -1))
    out = []
    for step in range(3):
        p = np.array([v.value * (1 + 0.02 * np.cos(step + i)) for i, v in enumerate(params)])
        out.append((eng.nll(p), *eng.nll_grad(p)))
    eng.close()
    return out


@pytest.mark.parametrize("bins,two", [(1, False), (255, False), (256, True), (257, False), (2048, True), (2049, True),
                                      (4096, False), (4097, False)])
def test_every_cta_sums_a_small_grid(bins, two, monkeypatch):
    monkeypatch.delenv("GF_FUSED", raising=False)
    one = _evaluate(bins, two)
    monkeypatch.setenv("GF_FUSED", "0")
    for (n0, n1, g), (r0, r1, rg) in zip(one, _evaluate(bins, two)):
        assert n0 == pytest.approx(r0, rel=1e-9) and n1 == pytest.approx(r1, rel=1e-9)
        assert np.all(np.abs(g - rg) <= 1e-6 * np.abs(rg) + 1e-6 * np.sqrt(7001) * np.maximum(1.0, np.abs(rg)))
