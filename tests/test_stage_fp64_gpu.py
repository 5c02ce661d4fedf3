"""FP64, one launch: the convolutions' model and resolution values are evaluated once per launch and read back by the
table CTAs, whose tiles depend on the table's size.  Against the separate launches, which evaluate them in every table
CTA: the same values summed in another partition, 1e-13 of the NLL (a thousand terms of 2^-53 each, at random)."""
import numpy as np
import pytest

import goofit_gb300 as gf

pytestmark = pytest.mark.gpu


def _evaluate(step, two, n):
    x = gf.Observable("x", -5.0, 10.0)
    x.setNumBins(1000)

    def conv(k, mu, sigma):
        c = gf.ConvolutionPdf(f"conv{k}", x, gf.ExpPdf(f"e{k}", x, gf.Variable(f"a{k}", -0.6 - 0.2 * k, 0.05, -2.0, -0.1)),
                              gf.GaussianPdf(f"g{k}", x, gf.Variable(f"mu{k}", mu, 0.02, -1, 1), gf.Variable(f"s{k}", sigma, 0.02, 0.05, 1)))
        c.setIntegrationConstants(0.0, 10.0, step)
        return c

    parts = [conv(0, 0.05, 0.35)] + ([conv(1, -0.1, 0.6)] if two else [])
    parts.append(gf.PolynomialPdf("flat", x, [gf.Variable("c0", 1.0)], 0))
    pdf = gf.AddPdf("sum", [gf.Variable(f"f{k}", 0.3, 0.01, 0, 1) for k in range(len(parts) - 1)], parts)
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    eng = gf.Engine("fp64")
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params),
                 [0 if (v.fixed or id(v) in nd) else 1 for v in params])
    rng = np.random.Generator(np.random.PCG64(n))
    eng.upload(np.clip(rng.exponential(1.5, n) + rng.normal(0, 0.3, n), -4.9, 9.9).reshape(1, -1))
    out = []
    for k in range(3):
        p = np.array([v.value * (1 + 0.02 * np.cos(k + i)) for i, v in enumerate(params)])
        out.append((eng.nll(p), *eng.nll_grad(p)))
    eng.close()
    return out


@pytest.mark.parametrize("step,two,n", [(0.01, False, 5000), (0.01, True, 5000), (0.5, False, 1), (0.1, True, 70001), (0.037, False, 300)])
def test_staged_tables_match_the_separate_launches(step, two, n, monkeypatch):
    monkeypatch.delenv("GF_FUSED", raising=False)
    one = _evaluate(step, two, n)
    monkeypatch.setenv("GF_FUSED", "0")
    for (n0, n1, g), (r0, r1, rg) in zip(one, _evaluate(step, two, n)):
        assert n0 == pytest.approx(r0, rel=1e-13) and n1 == pytest.approx(r1, rel=1e-13)
        # gradient terms below 100 per event, a thousand roundings each at random
        np.testing.assert_allclose(g, rg, rtol=1e-11, atol=1e-12 * 100 * n)
