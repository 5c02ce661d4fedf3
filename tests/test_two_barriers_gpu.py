"""A product that shares its observable with a convolution is normalised on a grid that reads the convolution's table,
so its one-launch evaluation has two grid barriers: table, grid, events.  Both variants (with and without gradient) are
evaluated in turn at points that move every factor, against FP64 numpy: a barrier that let a CTA past early would mix
one point's table or normalisation with the next point's."""
import numpy as np
import pytest

import goofit_gb300 as gf
from goofit_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _nll(v, x):
    ks, table, lbo = W._conv_table(v["alpha"], v["mu"], v["sigma"])

    def density(t):
        return table[np.floor(t / 0.01 - lbo).astype(np.int64) - ks[0]] * (v["a0"] + v["a1"] * t)

    centres = 15.0 / 3000 * (np.arange(3000) + 0.5) - 5.0
    return -np.log(density(x) / (15.0 / 3000 * density(centres).sum())).sum()


@pytest.mark.parametrize("prec,rtol", [("mixed", 1e-6), ("fp64", 1e-10)])
def test_grid_that_reads_a_convolution_table(prec, rtol):
    x = gf.Observable("x", -5.0, 10.0)
    x.setNumBins(3000)
    model = gf.ExpPdf("decay", x, gf.Variable("alpha", -0.6, 0.05, -2.0, -0.1))
    resolution = gf.GaussianPdf("res", x, gf.Variable("mu", 0.05, 0.02, -1.0, 1.0), gf.Variable("sigma", 0.35, 0.02, 0.05, 1.0))
    conv = gf.ConvolutionPdf("conv", x, model, resolution)
    conv.setIntegrationConstants(0.0, 10.0, 0.01)
    poly = gf.PolynomialPdf("acc", x, [gf.Variable("a0", 1.0), gf.Variable("a1", 0.03, 0.001, -0.05, 0.09)], 0)
    pdf = gf.ProdPdf("prod", [conv, poly])
    nodes, params, obs = pdf._flatten()
    olist = [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs]
    nd = pdf._nondiff_all()
    mask = [0 if (v.fixed or id(v) in nd) else 1 for v in params]
    rng = np.random.Generator(np.random.PCG64(9))
    cols = np.clip(rng.exponential(1.5, 20_000) + rng.normal(0, 0.3, 20_000), -4.9, 9.9).reshape(1, -1)
    eng = gf.Engine(prec)
    eng.set_tree(nodes, olist, len(params), mask)
    eng.upload(cols)
    free = [i for i, m in enumerate(mask) if m]
    for step in range(12):
        p = np.array([v.value for v in params])
        p[free] *= 1 + 0.04 * np.cos(step + np.arange(len(free)))
        at = {v.name: p[i] for i, v in enumerate(params)}
        ref = _nll(at, cols[0])
        assert eng.nll(p) == pytest.approx(ref, rel=rtol)
        got, grad = eng.nll_grad(p)
        assert got == pytest.approx(ref, rel=rtol)
        if step == 0:
            fd = [(_nll({**at, k: at[k] + 1e-6}, cols[0]) - _nll({**at, k: at[k] - 1e-6}, cols[0])) / 2e-6
                  for k in (params[i].name for i in free)]
            np.testing.assert_allclose(grad, fd, rtol=2e-4, atol=2e-3 * np.sqrt(cols.shape[1]))
    eng.close()
