"""A device too full for the exact gradient's stage caches and the buffers of its reverse step together: the caches go
(the first allocation of the step's buffers is refused here; no memory is taken)."""
import pytest
import torch

from sparc_flows_gb300 import discrete_adjoint as D
from sparc_flows_gb300 import model as M
from sparc_flows_gb300.config import RunConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("refuse", ["work", "adjoints"])
def test_caches_make_room_for_the_step(monkeypatch, refuse):
    from sparc_flows_gb300.solver import WaveSolver
    run = RunConfig(nx=128, nz=157, xlength_cm=100e8, nsteps=37, flows=True)
    model = M.polytrope(157)
    psi = torch.as_tensor(M.gaussian_psi(run, model, M.psi_amplitude_for_peak(run, model, 240.0)), device="cuda")

    def gradient():
        ws = WaveSolver(run, model, precision=64, psi=psi.cpu().numpy())
        ws.set_forward_sources([M.SourceSpec(-5.0)])
        eg = D.ExactGradient(ws, receivers=[30, 64, 90], segment=10)
        assert eg._keep_caches
        rec = eg.forward(psi).clone()
        refused = []
        if refuse:
            size = int(ws.L.sparc_adjoint_step_bytes(ws.plan))
            name = "empty" if refuse == "work" else "zeros"
            real = getattr(torch, name)

            def full(*a, **kw):
                if not refused and (refuse != "work" or a[0] == size):
                    refused.append(a)
                    raise torch.cuda.OutOfMemoryError("refused")
                return real(*a, **kw)

            monkeypatch.setattr(D.torch, name, full)
        g = eg.gradient(psi, rec)
        monkeypatch.undo()
        out = [rec, g] + [eg.last[k].clone() for k in ("v0x", "v0z", "c2rho0")]
        assert eg._keep_caches != bool(refused)
        if refuse:
            assert refused and eg.segbuf.shape == (10, eg.row)
        ws.close()
        return out

    got = gradient()
    refuse = None
    # the same steps with their stages run again: 2 ulp in the forcing, carried on by 37 steps
    for a, b in zip(got, gradient()):
        assert float(b.norm()) > 0 and float((a - b).norm()) <= 1e-12 * float(b.norm())
