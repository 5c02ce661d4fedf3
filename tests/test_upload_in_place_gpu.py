"""Events of 4 MB and more are read in place from ordinary host memory; smaller uploads, and GF_UPLOAD_STAGE=1, go
through the staging buffer.  Both sides of the limit, an address that is only 8-byte aligned, a memory-mapped file whose
pages are not resident, and a buffer that is changed right after the upload: the same NLL bit for bit, and an event
outside the convolution's range is still refused."""
import numpy as np
import pytest

import goofit_gb300 as gf
from goofit_gb300 import _abi as A
from goofit_gb300 import workloads as W

pytestmark = pytest.mark.gpu

LIMIT = (4 << 20) // 8


def _engine(prec="mixed"):
    pdf = W.make_c2(16, seed=0).pdf
    nodes, params, obs = pdf._flatten()
    nd = pdf._nondiff_all()
    eng = gf.Engine(prec)
    eng.set_tree(nodes, [(o.lowerlimit, o.upperlimit, o.numbins, int(o.is_event_number)) for o in obs], len(params),
                 [0 if (v.fixed or id(v) in nd) else 1 for v in params])
    return eng, np.array([v.value for v in params])


def _events(n):
    rng = np.random.Generator(np.random.PCG64(n))
    return np.clip(rng.exponential(1.5, n) + rng.normal(0, 0.3, n), -4.99, 9.99)


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [LIMIT - 1, LIMIT, LIMIT + 77])
def test_in_place_and_staged_uploads_agree(n, prec, monkeypatch, tmp_path):
    x = _events(n)
    eng, p = _engine(prec)
    monkeypatch.setenv("GF_UPLOAD_STAGE", "1")
    eng.upload(x)
    nll, grad = eng.nll_grad(p)
    monkeypatch.delenv("GF_UPLOAD_STAGE")
    shifted = np.empty(n + 1)
    shifted[1:] = x
    x.tofile(tmp_path / "x.bin")
    for y in (x, shifted[1:], np.memmap(tmp_path / "x.bin", dtype=np.float64, mode="r")):
        eng.upload(y)
        if y.flags.writeable:
            y[:] = 0.0  # the call has read the events
        a, b = eng.nll_grad(p)
        assert a == nll
        np.testing.assert_array_equal(b, grad)
        if y.flags.writeable:
            y[:] = np.fromfile(tmp_path / "x.bin")
    x[n // 2] = 11.0
    with pytest.raises(A.EngineError):
        eng.upload(x)
    eng.close()
