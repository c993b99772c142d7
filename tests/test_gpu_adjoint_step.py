"""The fused reverse step (sparc_adjoint_step) against the transposed operators applied one at a time
(StepOperators.step, step_T) on random states and adjoints, over transform lengths, odd depths, one and two
solves, a depth-only and a 2-D sound speed, and both filter coverages."""
import numpy as np
import pytest
import torch

from sparc_flows_gb300 import model as M
from sparc_flows_gb300.config import RunConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,nb,bump,wide", [(64, 150, 1, False, False), (128, 217, 2, True, False),
                                                (192, 301, 1, True, True), (256, 300, 3, False, False),
                                                (384, 199, 2, True, False), (512, 160, 1, False, True),
                                                (768, 151, 1, True, False), (1024, 150, 2, False, False)])
def test_matches_operators(nx, nz, nb, bump, wide):
    from sparc_flows_gb300.discrete_adjoint import ExactGradient
    from sparc_flows_gb300.solver import WaveSolver
    run = RunConfig(nx=nx, nz=nz, xlength_cm=nx * 0.78125e8, nsteps=20, flows=True, npmlbot=12, filter_all_x=wide,
                    filter_kst=4 if wide else 6)
    model = M.polytrope(nz)
    psi = M.gaussian_psi(run, model, M.psi_amplitude_for_peak(run, model, 240.0))
    ws = WaveSolver(run, model, nbatch=nb, precision=64, psi=psi, cmul=M.c_bump(run, model) if bump else None)
    ws.set_forward_sources([M.SourceSpec(3.0 * i) for i in range(nb)])
    eg = ExactGradient(ws, receivers=[nx // 2], segment=10, use_graph=False)
    ops, S = eg.ops, eg._static()
    g = torch.Generator(device="cpu").manual_seed(nx + nz)
    for k in ("a", "Pz", "Px", "la", "lZ", "lW", "f"):
        S[k].copy_(torch.randn(S[k].shape, generator=g, dtype=torch.float64))
    v0x, v0z = ws.bg["v0x"][0], ws.bg["v0z"][0]
    caches = ops.step(S["a"], S["Pz"], S["Px"], v0x, v0z, S["f"])[3]
    want = ops.step_T(S["la"].clone(), S["lZ"].clone(), S["lW"].clone(), v0x, v0z, caches)
    before = S["a"].clone()
    eg._reverse_step()
    got = (S["la"], S["lZ"], S["lW"], S["gx"].sum(0), S["gz"].sum(0), S["gc"].sum(0))
    assert torch.equal(before, S["a"])
    # five stages of solves of condition below 20 on values that differ by 1e3 between the fields: 1e-16 rounds to
    # less than 1e-11 of each result's norm
    for name, x, y in zip(("state", "z auxiliaries", "x auxiliaries", "v0x", "v0z", "c2rho0"), got, want):
        err = float((x - y).norm() / y.norm())
        assert np.isfinite(err) and err <= 1e-11, (name, err)
    ws.close()


@pytest.mark.parametrize("graph", [True, False])
def test_kept_caches_equal_recomputed_stages(monkeypatch, graph):
    """A segment's stage caches kept by its replay, or the states kept and every reverse step's stages recomputed:
    the same kernels on values that differ by the rounding of the forcing (its two products in another order, 2 ulp),
    which 37 steps carry on: far below 1e-12 of the norm."""
    from sparc_flows_gb300 import discrete_adjoint as D
    from sparc_flows_gb300.solver import WaveSolver
    run = RunConfig(nx=128, nz=157, xlength_cm=100e8, nsteps=37, flows=True)
    model = M.polytrope(157)
    psi = torch.as_tensor(M.gaussian_psi(run, model, M.psi_amplitude_for_peak(run, model, 240.0)), device="cuda")
    out = []
    for limit in (1 << 40, 0):
        monkeypatch.setattr(D, "CACHE_BYTES", limit)
        ws = WaveSolver(run, model, nbatch=2, precision=64, psi=psi.cpu().numpy())
        ws.set_forward_sources([M.SourceSpec(-5.0), M.SourceSpec(8.0)])
        eg = D.ExactGradient(ws, receivers=[30, 64, 90], segment=10, use_graph=graph)
        assert eg._keep_caches == (limit > 0)
        rec = eg.forward(psi).clone()
        g = eg.gradient(psi, rec)
        out.append([rec, g] + [eg.last[k] for k in ("v0x", "v0z", "c2rho0")])
        ws.close()
    for a, b in zip(*out):
        assert torch.isfinite(a).all() and float((a - b).norm()) <= 1e-12 * float(b.norm()) and float(b.norm()) > 0
