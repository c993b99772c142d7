"""The banded FP32 column pass with its inputs staged by bulk copies on grids without a compiled specialisation:
odd and even depths (an odd one takes a copy of one row besides the two boxes), row groups that end short, per-solve
backgrounds; against the FP64 plan."""
import numpy as np
import pytest

from sparc_flows_gb300 import model as M
from sparc_flows_gb300.config import RunConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,nb,per_solve", [(64, 89, 1, False), (128, 157, 3, True), (192, 217, 2, False),
                                                (512, 256, 1, False), (256, 271, 2, True), (512, 301, 2, False),
                                                (768, 300, 1, False), (1024, 101, 2, False)])
def test_tracks_fp64(nx, nz, nb, per_solve):
    from sparc_flows_gb300.solver import WaveSolver
    run = RunConfig(nx=nx, nz=nz, xlength_cm=nx * 0.78125e8, nsteps=46, flows=True, npmlbot=20)
    model = M.polytrope(nz)
    amp = M.psi_amplitude_for_peak(run, model, 200.0)
    psi, cmul = M.gaussian_psi(run, model, amp), M.c_bump(run, model)
    if per_solve:
        psi = [M.gaussian_psi(run, model, amp * (1 + 0.1 * b)) for b in range(nb)]
        cmul = [M.c_bump(run, model, 0.02 * (1 + b)) for b in range(nb)]
    out = {}
    for precision in (32, 64):
        ws = WaveSolver(run, model, nbatch=nb, precision=precision, psi=psi, cmul=cmul)
        if precision == 32:
            name = ws.column_kernel_name()
            assert name.startswith("col_band_kernel<32,"), name
        ws.set_forward_sources([M.SourceSpec(3.0 * b, spatial=M.SPATIAL_REFERENCE, temporal=M.TEMPORAL_REFERENCE)
                                for b in range(nb)])
        out[precision] = (ws.forward().double().cpu().numpy(), ws.state().double().cpu().numpy())
        ws.check()  # no wait gave up
        ws.close()
    for a, b in zip(out[32], out[64]):
        assert np.abs(b).max() > 0 and np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b)
