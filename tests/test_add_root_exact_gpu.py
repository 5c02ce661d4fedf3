"""The extended root AddPdf of the mixed engine (the event loop of factored sums) against the FP64 engine's general form,
gradient entry by entry: yields near and far from the number of events, zero, fixed, a normalisation whose ratio to the
yields is below the range of FP32, one child, and fractions (the general form) beside them.

Every parameter is an FP32 number, so both engines evaluate the same function.  An event's term of a gradient entry is a
few FP32 operations (2^-24 each) on exponentials of relative error 2e-6 at most (5e-6 where the exponent reaches 85), its
cancelling parts at most ten times the term: 1e-5 (2e-5) of the sum of the events' absolute terms.  A yield's term is
1 / (summed yields) less the child's share over its yield, which cancel wholly where one child alone contributes: there the
parts themselves are summed."""
import numpy as np
import pytest

import goofit_gb300 as gf

pytestmark = pytest.mark.gpu


def _pdf(kind, weights, alpha, parts):
    x = gf.Observable("x", 0.0, 10.0)
    x.setNumBins(500)
    v = lambda name, value, e, lo, hi: gf.Variable(name, float(np.float32(value)), e, lo, hi)  # noqa: E731
    comps = [gf.GaussianPdf("g", x, v("m", 5.1, 0.01, 4, 6), v("s", 0.6, 0.01, 0.1, 2)),
             gf.ExpPdf("e", x, v("a", alpha, 0.01, -9, 9)),
             gf.PolynomialPdf("p", x, [v("p0", 1.0, 0.01, 0.5, 2), v("p1", -0.03, 0.001, -0.05, 0.2)], 0)][:parts]
    w = [v(f"w{k}", q, 1, 0, 1e9) for k, q in enumerate(weights)]
    return gf.AddPdf("sum", w, comps)


def _engine(precision, pdf, fixed):
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    eng = gf.Engine(precision)
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params),
                 [0 if (id(v) in nd or v.name in fixed) else 1 for v in params])
    return eng, np.array([v.value for v in params]), [v.name for v in params]


@pytest.mark.parametrize("kind,weights,alpha,parts,fixed", [
    ("yields", (128, 96, 77), -0.3, 3, ()), ("yields", (900, 700, 400), -0.3, 3, ()), ("yields", (9, 7, 4), 0.7, 3, ()),
    ("yields", (0, 700, 400), -0.3, 3, ()), ("yields", (900, 0, 0), -0.3, 3, ()), ("yields", (2e7, 1e6, 3e5), -0.3, 3, ()),
    ("yields", (900, 700, 400), -0.3, 3, ("s", "p1", "w0")), ("yields", (900, 700, 400), -0.3, 3, ("m", "s", "a", "p0", "p1")),
    ("yields", (300,), -0.3, 1, ()), ("yields", (300, 100), -0.3, 2, ()),
    ("yields", (1e7, 8e6, 7e6), 8.5, 3, ()), ("fractions", (0.5, 0.25), -0.3, 3, ()),
])
def test_root_add_gradient_entry_by_entry(kind, weights, alpha, parts, fixed):
    assert len(weights) == parts - (kind == "fractions")
    pdf = _pdf(kind, weights, alpha, parts)
    rng = np.random.Generator(np.random.PCG64(9))
    n = 301
    x = np.concatenate([rng.normal(5, 0.6, 120), rng.uniform(0, 10, 90), rng.uniform(9, 10, 91)])
    x = np.clip(x, 0.01, 9.99).reshape(1, -1)
    eng, p, names = _engine("mixed", pdf, fixed)
    eng.upload(x)
    ref, _, _ = _engine("fp64", pdf, fixed)
    ref.upload(x)
    want, g64 = ref.nll_grad(p)
    got, g = eng.nll_grad(p)
    rel = 2e-5 if alpha > 8 else 1e-5
    assert abs(got - want) <= rel * n and abs(eng.nll(p) - want) <= rel * n
    # the absolute terms: single events, without the extended term
    terms = np.zeros(len(g))
    extended = np.array([1 - 1 / sum(weights) if kind == "yields" and names[i].startswith("w") else 0.0 for i in eng.grad_params])
    one, _, _ = _engine("fp64", pdf, fixed)
    for i in range(n):
        one.upload(x[:, i:i + 1])
        terms += np.abs(one.nll_grad(p)[1] - extended) + np.where(extended != 0, 1 / sum(weights), 0)
    assert np.all(np.abs(g - g64) <= rel * terms + 1e-12), dict(zip([names[i] for i in eng.grad_params], (g - g64) / terms))
