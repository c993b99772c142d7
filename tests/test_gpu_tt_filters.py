"""Filters that are not even, filter(-f, -k) != filter(f, k): the filtered records are complex, and the picks and travel
times see their real parts (driver.f90:1990-2100)."""
import numpy as np
import pytest
import torch

from oracle import tt_oracle as TO
from sparc_flows_gb300 import ttadjoint as TT

pytestmark = pytest.mark.gpu
CAD, X00, NX = 30.0, [-4.0, 9.0], 64
XL = NX * 0.78125e8
MODES = {1: (2.0, 20.0, 4.0), 8: (1.0, 18.0, 6.0)}


def _filters(nt, shape):
    """(9, nt, NX): the ridges of one direction of travel, or no symmetry at all."""
    rng = np.random.default_rng(nt)
    if shape == "one-sided":
        f = TO.distmat(nt)[None, :, None] * TO.distmat(NX)[None, None, :] > 0
        return np.stack([TO.ridge_filter(p, NX, nt, XL, CAD) for p in range(9)]) * f
    return rng.uniform(0.0, 1.0, (9, nt, NX))


@pytest.mark.parametrize("nt", [128, 141, 514, 515])  # the two derivatives' transforms, and both t transforms
@pytest.mark.parametrize("shape", ["one-sided", "any"])
def test_matches_oracle(monkeypatch, nt, shape):
    filt = _filters(nt, shape)
    monkeypatch.setattr(TO, "ridge_filter", lambda p, *a: filt[p])
    monkeypatch.setattr(TT, "_ridge_filters", lambda *a: torch.as_tensor(filt, device="cuda"))
    rng = np.random.default_rng(nt)
    s = rng.standard_normal((2, nt, NX))
    d = np.roll(s, 1, axis=1) + 0.1 * rng.standard_normal(s.shape)
    t_min = -(CAD * (np.arange(nt) + 1.0))[::-1] / 60.0
    tt = TT.TTAdjoint(NX, nt, 2, XL, CAD)
    dev = [torch.as_tensor(v, device="cuda") for v in (s, d)]
    res, bands = tt.run(*dev, X00, t_min, MODES), tt.misfit_all(*dev, X00, t_min, MODES)
    tt.close()
    for b in range(2):
        ref = TO.adjoint_source(s[b], d[b], X00[b], XL, t_min, CAD, MODES)
        for pord in MODES:
            got, want = res["rows"][pord].get(b, []), ref["rows"][pord]
            assert want and [g[2:7] for g in got] == [w[2:7] for w in want]
            assert np.allclose([g[1] for g in got], [w[1] for w in want], rtol=1e-9, atol=1e-12)
        adj = res["adj"][b].cpu().numpy()
        assert np.linalg.norm(adj - ref["adj"]) <= 1e-10 * np.linalg.norm(ref["adj"])
        ref = TO.misfit_all(s[b], d[b], X00[b], XL, t_min, CAD, MODES)
        for fb in range(3):
            assert np.array_equal(bands[fb]["nmeas"][b], ref[fb]["nmeas"])
            assert np.allclose(bands[fb]["misfit"][b], ref[fb]["misfit"], rtol=1e-9, atol=0)
