"""A root AddPdf without convolution tables takes the event loop of factored sums: fractions and yields, weights of zero
and one, analytic, numeric and unit normalisations, parameters shared between children (more sums than the general form
has: it is kept), and fixed parameters.  NLL and gradient against the oracle: 1e-6 relative, and 2e-4 relative plus
2e-3 sqrt(n) of its central differences, the mixed engine's tolerances for every tree."""
import math

import numpy as np
import pytest

import goofit_gb300 as gf
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _parts(x, shared):
    v = gf.Variable
    m = v("m", 5.0, 0.01, 4, 6)
    s = v("s", 0.6, 0.01, 0.1, 2)
    out = [gf.GaussianPdf("g", x, m, s), gf.ExpPdf("e", x, v("a", -0.3, 0.01, -2, 2)),
           gf.PolynomialPdf("p", x, [v("p0", 1.0), v("p1", -0.03, 0.001, -0.05, 0.2)], 0)]
    if shared:
        out += [gf.GaussianPdf(f"g{k}", x, m, s) for k in range(4)]
    return out


@pytest.mark.parametrize("kind,weights,shared,fixed", [
    ("fractions", (0.4, 0.3), False, ()), ("fractions", (0.0, 0.3), False, ()), ("fractions", (0.0, 1.0), False, ()),
    ("fractions", (0.4, 0.3), False, ("m", "a", "f1")), ("fractions", (0.2, 0.2, 0.1, 0.1, 0.1, 0.1), True, ()),
    ("yields", (900.0, 700.0, 400.0), False, ()), ("yields", (0.0, 700.0, 400.0), False, ()),
    ("yields", (900.0, 700.0, 400.0), False, ("s", "p1", "f0")),
])
def test_root_add_matches_the_oracle(kind, weights, shared, fixed):
    x = gf.Observable("x", 0.0, 10.0)
    x.setNumBins(500)
    parts = _parts(x, shared)
    hi = 1.0 if kind == "fractions" else 1e6
    w = [gf.Variable(f"f{k}", q, 0.01, 0.0, hi) for k, q in enumerate(weights)]
    assert len(w) == len(parts) - (kind == "fractions")
    pdf = gf.AddPdf("sum", w, parts)
    nodes, params, obs = pdf._flatten()
    olist = [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs]
    nd = pdf._nondiff_all()
    mask = [0 if (v.fixed or id(v) in nd or v.name in fixed) else 1 for v in params]
    rng = np.random.Generator(np.random.PCG64(8))
    n = 3001
    cols = np.clip(np.where(rng.random(n) < 0.4, rng.normal(5, 0.6, n), rng.uniform(0, 10, n)), 0.01, 9.99).reshape(1, -1)
    eng = gf.Engine("mixed")
    eng.set_tree(nodes, olist, len(params), mask)
    eng.upload(cols)
    p = np.array([v.value for v in params])
    free = [i for i, k in enumerate(mask) if k]
    ref = O.nll(nodes, olist, p, cols)
    got, g = eng.nll_grad(p)
    assert got == pytest.approx(ref, rel=1e-6) and eng.nll(p) == pytest.approx(ref, rel=1e-6)
    fd = O.fd_grad(nodes, olist, p, cols, free, h=1e-6)
    np.testing.assert_allclose(g, fd, rtol=2e-4, atol=2e-3 * math.sqrt(n))
    eng.close()
