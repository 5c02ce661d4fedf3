"""gf_amp_store_bytes counts the memory that the store mode keeps: derivative columns of the events, and scratch columns of
the normalisation points only where the integrals are formed from columns.  The automatic mode stores at a budget of the
size of both and recomputes one byte below it."""
import numpy as np
import pytest

import goofit_gb300 as gf
from goofit_gb300 import workloads as W

pytestmark = pytest.mark.gpu

N, RES, FLOATED = 5001, 8, 4


def _engine(precision, mode="auto", budget=0):
    pdf = W.c3_model(120)[0]
    for name, *_ in W.C3_RESONANCES[:FLOATED]:
        for v in pdf.getParameters():
            if v.name in (f"{name}_mass", f"{name}_width"):
                v.setFixed(False)
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    eng = gf.Engine(precision)
    eng.set_amp_mode(mode, budget)
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params),
                 [0 if (v.fixed or id(v) in nd) else 1 for v in params])
    rng = np.random.Generator(np.random.PCG64(3))
    x = rng.uniform(0.3, 2.8, (2, 4 * N))
    x = x[:, x.sum(0) > 1.2][:, :N]
    assert x.shape[1] == N
    eng.upload(np.vstack([x, np.arange(N)]))
    return eng, np.array([v.value for v in params])


@pytest.mark.parametrize("precision,gram,item,scratch", [("mixed", None, 8, False), ("mixed", "cuda", 8, True), ("fp64", None, 16, True)])
def test_store_bytes_are_what_the_store_mode_keeps(precision, gram, item, scratch, monkeypatch):
    if gram:
        monkeypatch.setenv("GF_GRAM", gram)
    else:
        monkeypatch.delenv("GF_GRAM", raising=False)
    eng, p = _engine(precision, "store")
    got = eng.amp_store_bytes()
    columns = (N + 7) // 8 * 8 * 2 * FLOATED * item
    # 120^2 bins, of which about a third lie inside the boundary, each with value and derivative columns and an efficiency
    per_point = (RES + 2 * FLOATED) * item + item // 2
    monkeypatch.setenv("GF_GRAM", "cuda")  # its integrals take the columns in the mixed engine too
    other, _ = _engine(precision, "store")
    both = other.amp_store_bytes()
    other.close()
    assert (both - columns) % (4 * per_point) == 0 and 0.2 < (both - columns) / per_point / 120 ** 2 < 0.5
    assert got == (both if scratch else columns)
    if not gram:
        monkeypatch.delenv("GF_GRAM")
    want = eng.nll_grad(p)
    eng.close()
    for budget, recomputes in ((both, False), (both - 1, True)):
        eng, _ = _engine(precision, "auto", budget)
        assert eng.amp_recomputing() is recomputes
        nll, grad = eng.nll_grad(p)
        assert nll == pytest.approx(want[0], rel=1e-6)
        if not recomputes:
            assert nll == want[0] and np.array_equal(grad, want[1])
        eng.close()
