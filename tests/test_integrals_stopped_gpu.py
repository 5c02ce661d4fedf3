"""A wait of the one-pass integrals that runs out in some CTAs only: every evaluation that needed them reports it, also
where the integrals are read behind the event launch without a synchronisation, and nothing of the failed sums is kept."""
import numpy as np
import pytest

import goofit_gb300 as G
from goofit_gb300 import _abi as A
from goofit_gb300 import phasespace
from goofit_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _three():
    # 173,000 points in tiles of 128: the last of three rounds of tiles reaches a quarter of the CTAs
    pdf = W.c3_model(700)[0]
    for v in pdf.getParameters():
        if v.name in ("rho770_mass", "rho770_width"):
            v.setFixed(False)
    rng = np.random.Generator(np.random.PCG64(3))
    x = rng.uniform(0.3, 2.8, (2, 8000))
    x = x[:, x.sum(0) > 1.2][:, :1500]
    return pdf, np.vstack([x, np.arange(x.shape[1])]), None


def _four():
    # three CTAs per SM of 152 take 58,368 points a round
    pdf = W.c5_model(1000, float_lineshapes=True)[0]
    ev = phasespace.norm_events(W.C5_M, W.C5_MASSES, 1500 + 130_000, 11)
    return pdf, np.vstack([ev[:, :1500], np.arange(1500)]), np.ascontiguousarray(ev[:, 1500:])


def _engine(make):
    pdf, events, norm = make()
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    mask = np.array([0 if (v.fixed or id(v) in nd) else 1 for v in params])
    eng = G.Engine("mixed")
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params), mask)
    if norm is not None:
        eng.set_norm_events(0, norm)
    eng.upload(events)
    p = np.array([v.value for v in params])
    return eng, [p * (1 + 0.01 * k * mask) for k in range(4)]


@pytest.mark.parametrize("make", [_three, _four])
def test_a_stop_in_some_ctas_is_reported_and_not_kept(make, monkeypatch):
    monkeypatch.delenv("GF_GRAM", raising=False)
    eng, points = _engine(make)
    want = [eng.nll_grad(p) for p in points]
    for k in (1, 2, 3, 1):
        monkeypatch.setenv("GF_GRAM_TEST_STALL_STAGE", "2")
        eng.set_gram_wait_limit(1_000_000)
        for _ in range(2):  # the failed rebuild is not taken for a finished one
            with pytest.raises(A.EngineError) as e:
                eng.nll_grad(points[k])
            assert e.value.code == A.GF_ERR_CUDA
        monkeypatch.delenv("GF_GRAM_TEST_STALL_STAGE")
        eng.set_gram_wait_limit(0)
        for q in (k, 0):
            nll, grad = eng.nll_grad(points[q])
            assert nll == want[q][0]
            np.testing.assert_array_equal(grad, want[q][1])
    eng.close()
