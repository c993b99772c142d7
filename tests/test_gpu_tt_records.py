"""Records that leave nothing to measure: the synthetic and the data of a source share a transform, which must not
carry rounding of one into the other where the other is zero or the two are equal."""
import numpy as np
import pytest
import torch

from oracle import tt_oracle as TO
from sparc_flows_gb300 import ttadjoint as TT

pytestmark = pytest.mark.gpu
CAD, X00, NX = 30.0, [-4.0, 9.0], 64
XL = NX * 0.78125e8
MODES = {1: (2.0, 20.0, 4.0), 8: (1.0, 18.0, 6.0)}


def _records(nt):
    rng = np.random.default_rng(nt)
    s = rng.standard_normal((2, nt, NX))
    return s, np.roll(s, 1, axis=1) + 0.1 * rng.standard_normal(s.shape)


def _run(s, d):
    nt = s.shape[1]
    t_min = -(CAD * (np.arange(nt) + 1.0))[::-1] / 60.0
    tt = TT.TTAdjoint(NX, nt, 2, XL, CAD)
    dev = [torch.as_tensor(v, device="cuda") for v in (s, d)]
    res, bands = tt.run(*dev, X00, t_min, MODES), tt.misfit_all(*dev, X00, t_min, MODES)
    tt.close()
    return t_min, res, bands


def _same(res, good, b):
    assert torch.equal(res["adj"][b], good["adj"][b]) and res["misfit"][b] == good["misfit"][b]
    assert all(res["rows"][p][b] == good["rows"][p][b] for p in MODES)


@pytest.mark.parametrize("nt", [128, 141])
def test_no_synthetic_is_no_travel_time(nt):
    s, d = _records(nt)
    good = _run(s, d)
    s[0] = 0.0
    _, res, bands = _run(s, d)
    _same(res, good[1], 1)
    for pord in MODES:
        rows = res["rows"][pord][0]
        assert rows and all(np.isnan(r[1]) for r in rows)
        assert all(r[4] == max(r[5], 1) for r in rows)  # the first of equal values
    assert np.isnan(res["misfit"][0]) and torch.isnan(res["adj"][0]).all()
    for fb in range(3):
        assert bands[fb]["nmeas"][0].sum() == 0 and bands[fb]["misfit"][0].sum() == 0.0
        assert np.array_equal(bands[fb]["misfit"][1], good[2][fb]["misfit"][1])


@pytest.mark.parametrize("nt", [128, 141])
def test_no_data(nt):
    s, d = _records(nt)
    good = _run(s, d)
    d[1] = 0.0
    t_min, res, bands = _run(s, d)
    _same(res, good[1], 0)
    ref = TO.adjoint_source(s[1], d[1], X00[1], XL, t_min, CAD, MODES)
    for pord in MODES:
        got, want = res["rows"][pord][1], ref["rows"][pord]
        assert [g[2:7] for g in got] == [w[2:7] for w in want]
        assert np.allclose([g[1] for g in got], [w[1] for w in want], rtol=1e-9, atol=1e-12)
    for fb in range(3):  # no correlation: no peak inside the lag range
        assert bands[fb]["nmeas"][1].sum() == 0


@pytest.mark.parametrize("nt", [128, 141])
def test_equal_records_have_no_shift(nt):
    s, d = _records(nt)
    good = _run(s, d)
    d[0] = s[0]
    _, res, bands = _run(s, d)
    _same(res, good[1], 1)
    for pord in MODES:
        assert res["rows"][pord][0] and all(r[1] == 0.0 for r in res["rows"][pord][0])
    assert res["misfit"][0] == 0.0 and (res["adj"][0] == 0.0).all()
    for fb in range(3):
        assert bands[fb]["nmeas"][0].sum() > 0 and bands[fb]["misfit"][0].sum() == 0.0
