"""The y passes of 384 and 512 rows with flow, field by field, and the records: against the 3-D CPU oracle."""
import numpy as np
import pytest

from oracle.oracle3d import Sim3D
from sparc_flows_gb300 import model as M
from sparc_flows_gb300.solver3d import WaveSolver3D

pytestmark = pytest.mark.gpu
XL, YL, NSTEPS, NX = 200e8, 150e8, 4, 64


# FP32's bound on every field and on the records, FP64's; 512 rows in FP32 only (an FP64 block has not the shared memory)
@pytest.mark.parametrize("ny,nz,precision,tol", [(512, 30, 32, 1e-4), (512, 41, 32, 1e-4), (384, 31, 32, 1e-4),
                                                 (384, 30, 64, 1e-10)])
def test_fields_match_oracle(ny, nz, precision, tol):
    X, Y = np.meshgrid(np.arange(NX) / NX - 0.5, np.arange(ny) / ny - 0.5)
    pats = np.stack([np.exp(-((X - 0.1 * b) ** 2 + (Y + 0.05 * b) ** 2) / 0.003) for b in range(2)])
    amp = np.sin(np.arange(NSTEPS + 5) * 0.4 + 0.3) * 1e-6
    env = np.exp(-(np.linspace(-1, 1, nz)[:, None, None] / 0.3) ** 2)
    v0 = (0.02 * env * np.sin(2 * np.pi * X) * np.cos(2 * np.pi * Y),
          -0.015 * env * np.cos(2 * np.pi * X) * np.sin(4 * np.pi * Y), 0.01 * env * np.cos(2 * np.pi * (X + Y)))
    model = M.polytrope(nz)
    ws = WaveSolver3D(NX, ny, model, XL, YL, nbatch=2, precision=precision, steps_out=1, flows=True, obsheight_cm=-100e5)
    ws.set_flow(*v0)
    ws.set_source(pats, amp)
    ws.reset(0)
    seis = ws.forward(NSTEPS).double().cpu().numpy()
    st = ws.state().double().cpu().numpy()
    ws.close()
    for b in range(2):
        s = Sim3D(NX, ny, nz, model, XL, YL, steps_out=1, obsheight_cm=-100e5)
        s.set_flow(*v0)
        s.set_source(pats[b], amp)
        rec = s.run(NSTEPS)
        want = s.state()
        s.close()
        for f in range(6):
            assert np.linalg.norm(want[f]) > 0 and np.linalg.norm(st[f, :, b] - want[f]) <= tol * np.linalg.norm(want[f]), f
        assert np.linalg.norm(seis[:, b] - rec) <= tol * np.linalg.norm(rec)
