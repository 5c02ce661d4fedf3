"""Sums of squares of the one-pass integrals against the FP64 engine, for floated Dalitz resonances, whose columns are the
FP64 values rounded to FP32 (so that their own error averages out over the points: 1e-9).  What is left is the tensor
core's truncation of each of four accumulations, half a unit of 2^-23 to 2^-24 on sums of a quarter, half, three quarters and
all of a tile: 2.5 x 0.5 x 0.75 x 2^-23 = 1.1e-7 on average.  A product part left out (lo lo, 4e-8 of a square) shows."""
import numpy as np
import pytest

import goofit_gb300 as G
from goofit_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _integrals(precision, bins):
    pdf = W.c3_model(bins)[0]
    for name, *_ in W.C3_RESONANCES:
        for v in pdf.getParameters():
            if v.name in (f"{name}_mass", f"{name}_width"):
                v.setFixed(False)
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    eng = G.Engine(precision)
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params),
                 [0 if (v.fixed or id(v) in nd) else 1 for v in params])
    eng.upload(np.array([[1.0], [1.2], [0.0]]))
    eng.set_params([v.value for v in params])
    out = eng.amp3_integrals(0, 8)
    eng.close()
    return out


@pytest.mark.parametrize("bins", [701, 1500])
def test_sums_of_squares_are_short_of_truncation_only(bins, monkeypatch):
    monkeypatch.delenv("GF_GRAM", raising=False)
    got, want = (np.diag(_integrals(p, bins)).real for p in ("mixed", "fp64"))
    err = got / want - 1
    assert np.all(err < 0) and -err.mean() <= 1.1e-7, err
