"""The top row's value of d xi_z/dz is set from d xi_x/dx without the horizontal PML's auxiliary (physics2d.f90:954-955):
a checkpoint that holds nothing but psi_vx of the top row, stepped on the FP32 512-column row pass and on the generic one
against FP64."""
import numpy as np
import pytest
import torch

from sparc_flows_gb300 import model as M
from sparc_flows_gb300.config import RunConfig

pytestmark = pytest.mark.gpu
NZ = 300


def _step(nx, precision, psi):
    from sparc_flows_gb300.solver import WaveSolver
    run = RunConfig(nx=nx, nz=NZ, xlength_cm=nx * 0.78125e8, nsteps=16, flows=True, npmlbot=20)
    ws = WaveSolver(run, M.polytrope(NZ), precision=precision, psi=np.zeros((NZ, nx)))
    ws.set_forward_sources([M.SourceSpec(0.0)])
    ws.reset(0)
    buf = torch.empty(-(-ws.checkpoint_bytes() // 256) * 256, dtype=torch.uint8, device="cuda")
    ws.checkpoint_save(buf)
    size, nzpml, nhx = ws.dtype.itemsize, run.npmlbot + run.npmltop, 2 * run.npmlhor
    first = 16 + size * (4 * NZ * nx + 2 * nzpml * nx)
    px = buf[first:first + size * 2 * NZ * nhx].view(ws.dtype).view(2, NZ, nhx)
    assert not px.any()
    px[0, NZ - 1] = torch.as_tensor(psi, dtype=ws.dtype, device="cuda")
    ws.checkpoint_load(buf)
    ws.run_steps(1)
    out = ws.state().double().cpu().numpy()[0]
    ws.close()
    return out


@pytest.mark.parametrize("nx", [384, 512])
def test_auxiliary_of_the_top_row(nx):
    psi = np.random.default_rng(nx).uniform(1.0, 2.0, 18)  # x-PML columns of both sides
    got, want = _step(nx, 32, psi), _step(nx, 64, psi)
    for f, name in enumerate(("xi_x", "xi_z", "v_x", "v_z")):  # FP32's bound on every field
        a, b = got[f, -8:], want[f, -8:]
        assert np.abs(b).max() > 0 and np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b), name
