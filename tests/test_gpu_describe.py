"""What sparc_plan_describe says of a plan is what its steps do: the stage overlap where the column pass has a partial
last wave behind a full one, with the same bits as without it, and the bulk-copied inputs of the banded pass."""
import numpy as np
import pytest

from sparc_flows_gb300 import model as M
from sparc_flows_gb300.config import RunConfig

pytestmark = pytest.mark.gpu


def _solver(nx, nz, nb, nsteps=16):
    from sparc_flows_gb300.solver import WaveSolver
    run = RunConfig(nx=nx, nz=nz, xlength_cm=nx * 0.78125e8, nsteps=nsteps, flows=True, npmlbot=20)
    ws = WaveSolver(run, M.polytrope(nz), nbatch=nb, precision=32, psi=np.zeros((nz, nx)))
    ws.set_forward_sources([M.SourceSpec(3.0 * b, spatial=M.SPATIAL_REFERENCE, temporal=M.TEMPORAL_REFERENCE)
                            for b in range(nb)])
    return ws


@pytest.mark.parametrize("nb,taken", [(1, "0"), (9, "0"), (10, "1"), (19, "0"), (20, "1")])  # 16 tiles a solve, 152 SMs
def test_overlap_of_the_default_rule(monkeypatch, nb, taken):
    monkeypatch.delenv("SPARC_STAGE_OVERLAP", raising=False)
    ws = _solver(512, 100, nb)
    d = ws.describe()
    ws.close()
    assert (d["stage_overlap"], d["overlap_taken"]) == ("1", taken), d
    for env, want in (("0", "0"), ("1", "1")):
        monkeypatch.setenv("SPARC_STAGE_OVERLAP", env)
        ws = _solver(512, 100, nb)
        assert ws.describe()["overlap_taken"] == want
        ws.close()


def test_default_rule_has_the_bits_of_no_overlap(monkeypatch):
    monkeypatch.delenv("SPARC_STAGE_OVERLAP", raising=False)
    out = []
    for env in (None, "0"):
        if env:
            monkeypatch.setenv("SPARC_STAGE_OVERLAP", env)
        ws = _solver(512, 300, 10, nsteps=46)
        assert ws.describe()["overlap_taken"] == ("0" if env else "1")
        out.append((ws.forward().cpu().numpy(), ws.state().cpu().numpy()))
        ws.check()
        ws.close()
    for a, b in zip(*out):
        assert np.abs(b).max() > 0 and np.array_equal(a, b)


@pytest.mark.parametrize("nx,nz,nb", [(64, 89, 1), (128, 157, 3), (192, 217, 2), (512, 256, 1), (256, 271, 2),
                                      (512, 301, 2), (768, 300, 1), (1024, 101, 2), (512, 300, 1)])
def test_staged_grids(nx, nz, nb):
    ws = _solver(nx, nz, nb)
    d = ws.describe()
    ws.close()
    assert d["column"].startswith("col_band_kernel<32,") and d["staged"] == "1", d
