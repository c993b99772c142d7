"""The fused x, y and z passes of the 3-D step at every transform length and at odd depths: FP64 plans with
flow and two solves against the 3-D CPU oracle, FP32 plans against FP64."""
import numpy as np
import pytest

from oracle.oracle3d import Sim3D
from sparc_flows_gb300 import model as M

pytestmark = pytest.mark.gpu
XL, YL, NSTEPS = 200e8, 150e8, 3


def _inputs(nx, ny, nz):
    x, y = np.arange(nx) / nx - 0.5, np.arange(ny) / ny - 0.5
    X, Y = np.meshgrid(x, y)
    pats = np.stack([np.exp(-((X - 0.1 * b) ** 2 + (Y + 0.05 * b) ** 2) / 0.003) for b in range(2)])
    amp = np.sin(np.arange(NSTEPS + 5) * 0.4 + 0.3) * 1e-6
    env = np.exp(-(np.linspace(-1, 1, nz)[:, None, None] / 0.3) ** 2)
    v0 = (0.02 * env * np.sin(2 * np.pi * X) * np.cos(2 * np.pi * Y),
          -0.015 * env * np.cos(2 * np.pi * X) * np.sin(4 * np.pi * Y), 0.01 * env * np.cos(2 * np.pi * (X + Y)))
    return M.polytrope(nz), pats, amp, v0


def _gpu(nx, ny, nz, precision, flows):
    from sparc_flows_gb300.solver3d import WaveSolver3D
    model, pats, amp, v0 = _inputs(nx, ny, nz)
    ws = WaveSolver3D(nx, ny, model, XL, YL, nbatch=2, precision=precision, steps_out=1, flows=flows,
                      obsheight_cm=-100e5)
    if flows:
        ws.set_flow(*v0)
    ws.set_source(pats, amp)
    ws.reset(0)
    seis = ws.forward(NSTEPS).double().cpu().numpy()
    st = ws.state().double().cpu().numpy()
    ws.close()
    return st, seis


@pytest.mark.parametrize("nx,ny,nz,flows", [(64, 64, 40, True), (128, 192, 41, True), (192, 128, 35, True),
                                            (256, 64, 49, True), (64, 256, 33, True), (384, 64, 30, True),
                                            (64, 384, 31, False), (512, 64, 30, True), (768, 64, 32, True),
                                            (1024, 64, 31, True)])
def test_passes_match_oracle(nx, ny, nz, flows):
    st, seis = _gpu(nx, ny, nz, 64, flows)
    model, pats, amp, v0 = _inputs(nx, ny, nz)
    for b in range(2):
        s = Sim3D(nx, ny, nz, model, XL, YL, steps_out=1, obsheight_cm=-100e5)
        if flows:
            s.set_flow(*v0)
        s.set_source(pats[b], amp)
        s.run(NSTEPS)
        want = s.state()
        s.close()
        assert np.linalg.norm(st[:, :, b] - want) <= 1e-10 * np.linalg.norm(want)
    st32, seis32 = _gpu(nx, ny, nz, 32, flows)
    assert np.linalg.norm(st32 - st) <= 1e-4 * np.linalg.norm(st)
    assert np.linalg.norm(seis32 - seis) <= 1e-4 * np.linalg.norm(seis) and seis.shape[0] == NSTEPS


def test_five_hundred_and_twelve_columns_along_y():
    """FP32 only: an FP64 block has not the shared memory."""
    a, b = _gpu(64, 512, 30, 32, True), _gpu(512, 64, 30, 64, True)
    assert np.isfinite(a[0]).all() and np.abs(a[0]).max() > 0 and b[0].shape[1] == a[0].shape[1]
