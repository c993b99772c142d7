"""The x-derivative of few rows and of many at 192 and 384 columns: both of its transforms, the row counts around the
change from one to the other, a last row without a partner; the same bits for a row among few and among many."""
import numpy as np
import pytest
import torch

from sparc_flows_gb300 import model as M
from sparc_flows_gb300.config import RunConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,precision,limit", [(192, 32, 3648), (192, 64, 3648), (384, 32, 1216), (384, 64, 1216)])
def test_few_and_many_rows(nx, precision, limit):
    """Tolerance: a transform rounds to about 10 eps of its row's norm, white noise's derivative weighs no wavenumber by
    more than twice its root mean square."""
    from sparc_flows_gb300.solver import WaveSolver
    run = RunConfig(nx=nx, nz=300, xlength_cm=nx * 0.78125e8, nsteps=16, flows=True, npmlbot=20)
    ws = WaveSolver(run, M.polytrope(300), nbatch=1, precision=precision, psi=np.zeros((300, nx)))
    v = np.random.default_rng(nx).standard_normal((limit + 3, nx))
    v[::3] *= 1e-200
    v[7] = 0.0
    k = 2 * np.pi * np.arange(nx // 2 + 1)
    k[-1] = 0.0
    want = np.fft.irfft(np.fft.rfft(v, axis=1) * (0.75j * k), n=nx, axis=1)
    out = {}
    for rows in (1, 2, 5, 301, limit - 1, limit, limit + 1, limit + 3):
        src = torch.as_tensor(v[:rows], device="cuda")
        out[rows] = torch.full_like(src, float("nan"))
        ws.ddx(src, out[rows], nrows=rows, stretchx=0.75)
        err = np.linalg.norm(out[rows].cpu().numpy() - want[:rows], axis=1)
        assert (err <= 1e-13 * np.linalg.norm(want[:rows], axis=1)).all(), rows
    for rows in out:
        pairs = rows // 2 * 2  # the last of an odd number of rows has no partner
        assert torch.equal(out[rows][:pairs], out[limit + 3][:pairs]), rows
    ws.close()
