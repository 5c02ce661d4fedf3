"""Which grids every CTA of the one-launch evaluation sums itself also depends on the components they are summed in: both
sides of the limits of bins x components and of components, with and without derivatives (the value alone may take the
other way), against the separate launches (GF_FUSED=0).  Tolerances as for the limit of bins: the factors agree to about
1e-14, NLL within 1e-9 relative, gradient within 1e-6 of its value or of the events' root sum of squares."""
import numpy as np
import pytest

import goofit_gb300 as gf

pytestmark = pytest.mark.gpu

N = 5003


def _pdf(bins, degree, nodes):
    x, y = gf.Observable("x", 0.0, 10.0), gf.Observable("y", 0.0, 10.0)
    x.setNumBins(bins)
    y.setNumBins(bins)
    parts = []
    for k in range(nodes):
        count = (degree + 1) * (degree + 2) // 2
        c = [gf.Variable(f"c{k}_{i}", 1.0 if i == 0 else 0.3 / (1 + i) * 0.1 ** (i % (degree + 1)), 0.01, -1, 2) for i in range(count)]
        parts.append(gf.MultiPolynomialPdf(f"m{k}", [x, y], c, [gf.Variable(f"a{k}", 5.0), gf.Variable(f"b{k}", 5.0)], degree))
    if nodes == 1:
        return parts[0]
    return gf.AddPdf("sum", [gf.Variable(f"f{k}", 0.8 / nodes, 0.01, 0, 1) for k in range(nodes - 1)], parts)


def _evaluate(shape):
    pdf = _pdf(*shape)
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    eng = gf.Engine("mixed")
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params),
                 [0 if (v.fixed or id(v) in nd) else 1 for v in params])
    eng.upload(np.random.Generator(np.random.PCG64(6)).uniform(0, 10, (2, N)))
    out = []
    for step in range(2):
        p = np.array([v.value * (1 + 0.01 * np.cos(step + i)) for i, v in enumerate(params)])
        out.append((eng.nll(p), *eng.nll_grad(p), eng.nll(p)))
    eng.close()
    return out


# 29 components of 41^2 and 42^2 bins (48,749 and 51,156 products), two and three polynomials of 16 and 11 (32 and 33
# components), 7 of 64^2 bins, 46 of 5^2
@pytest.mark.parametrize("shape", [(41, 6, 1), (42, 6, 1), (32, 4, 2), (32, 3, 3), (64, 2, 1), (5, 8, 1)])
def test_grids_of_many_components(shape, monkeypatch):
    monkeypatch.delenv("GF_FUSED", raising=False)
    one = _evaluate(shape)
    monkeypatch.setenv("GF_FUSED", "0")
    for (n0, n1, g, n2), (r0, r1, rg, _) in zip(one, _evaluate(shape)):
        assert np.isfinite(r0) and n0 == n2
        assert n0 == pytest.approx(r0, rel=1e-9) and n1 == pytest.approx(r1, rel=1e-9)
        assert np.all(np.abs(g - rg) <= 1e-6 * np.abs(rg) + 1e-6 * np.sqrt(N) * np.maximum(1.0, np.abs(rg)))
