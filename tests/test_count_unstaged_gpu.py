"""The tabulated event pass counts sorted bin offsets from shared memory or, when a CTA's events do not fit there, from
global memory: the same runs, so the same sums bit for bit.  Sizes around a thread's group of 8, a warp's and a CTA's
step, and many events per CTA; at 6e6 events one CTA's share does not fit its shared memory."""
import numpy as np
import pytest

import goofit_gb300 as gf
from goofit_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _evaluate(x):
    pdf = W.make_c2(16, seed=0).pdf
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    eng = gf.Engine("mixed")
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params),
                 [0 if (v.fixed or id(v) in nd) else 1 for v in params])
    eng.upload(x.reshape(1, -1))
    p = np.array([v.value for v in params]).astype(np.float32).astype(np.float64)
    out = [eng.nll(p), *eng.nll_grad(p)]
    eng.close()
    return out


def _events(n):
    rng = np.random.Generator(np.random.PCG64(n))
    return np.clip(rng.exponential(1.5, n) + rng.normal(0, 0.3, n), -4.99, 9.99)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 255, 2049, 77777, 700001])
def test_counts_from_global_memory(n, monkeypatch):
    x = _events(n)
    monkeypatch.setenv("GF_CHUNK", "512")
    staged = _evaluate(x)
    monkeypatch.setenv("GF_STAGE", "0")
    for a, b in zip(staged, _evaluate(x)):
        np.testing.assert_array_equal(a, b)


def test_events_that_do_not_fit_shared_memory(monkeypatch):
    """Against the per-event loop over unsorted offsets: its iterations of 8 events round in FP32 (three sums of up to
    8 terms, 2^-24 each), at random over the iterations: 1e-10 of the NLL, 2e-6 sqrt(n) of gradient terms below 10."""
    x = _events(6_000_001)
    nll, nll_g, grad = _evaluate(x)
    monkeypatch.setenv("GF_KSORT", "0")
    ref, ref_g, rgrad = _evaluate(x)
    assert nll == pytest.approx(ref, rel=1e-9) and nll_g == pytest.approx(ref_g, rel=1e-9)
    np.testing.assert_allclose(grad, rgrad, rtol=1e-6, atol=2e-6 * 6e6 ** 0.5 * 10)
