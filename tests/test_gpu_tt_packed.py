"""The shared transforms of the travel-time stage: record counts around the lengths of Bluestein's convolution
(odd and even, which split the derivatives differently), row lengths, data much larger and smaller than the
synthetic, and data that are not finite."""
import numpy as np
import pytest
import torch

from oracle import tt_oracle as TO
from sparc_flows_gb300 import ttadjoint as TT

pytestmark = pytest.mark.gpu
CAD, X00 = 30.0, [-4.0, 9.0]
MODES = {1: (2.0, 20.0, 4.0), 8: (1.0, 18.0, 6.0)}


def _records(nx, nt, size):
    rng = np.random.default_rng(nt)
    s = rng.standard_normal((2, nt, nx))
    return s, size * (np.roll(s, 1, axis=1) + 0.1 * rng.standard_normal(s.shape))


def _run(nx, nt, s, d):
    xl, t_min = nx * 0.78125e8, -(CAD * (np.arange(nt) + 1.0))[::-1] / 60.0
    tt = TT.TTAdjoint(nx, nt, 2, xl, CAD)
    res = tt.run(torch.as_tensor(s, device="cuda"), torch.as_tensor(d, device="cuda"), X00, t_min, MODES)
    tt.close()
    return xl, t_min, res


@pytest.mark.parametrize("nx,nt,size", [(64, 128, 1.0), (128, 129, 1e-9), (192, 200, 1e12), (384, 256, 1.0),
                                        (64, 257, 1.0), (128, 258, 1e-9), (512, 121, 1.0), (768, 90, 1.0),
                                        (1024, 127, 1.0), (64, 514, 1.0)])
def test_matches_oracle(nx, nt, size):
    s, d = _records(nx, nt, size)
    xl, t_min, res = _run(nx, nt, s, d)
    for b in range(2):
        ref = TO.adjoint_source(s[b], d[b], X00[b], xl, t_min, CAD, MODES)
        assert res["nmeas"][b] == ref["nmeas"] > 0
        for pord in MODES:
            got, want = res["rows"][pord].get(b, []), ref["rows"][pord]
            assert [g[2:7] for g in got] == [w[2:7] for w in want]
            assert np.allclose([g[1] for g in got], [w[1] for w in want], rtol=1e-9, atol=1e-12)
        adj = res["adj"][b].cpu().numpy()
        assert np.linalg.norm(adj - ref["adj"]) <= 1e-10 * np.linalg.norm(ref["adj"])


def test_data_that_are_not_finite_leave_the_windows():
    s, d = _records(128, 141, 1.0)
    good = _run(128, 141, s, d)[2]
    d[1, 3, 5] = np.nan
    res = _run(128, 141, s, d)[2]
    assert res["windows"] == good["windows"]
    assert np.isfinite(res["misfit"][0]) and np.isnan(res["misfit"][1])
    assert torch.equal(res["adj"][0], good["adj"][0]) and torch.isnan(res["adj"][1]).all()
