"""The fused x and z passes and the end of step of the velocity formulation (options 5, 6, 12) over transform
lengths, odd depths and block widths: FP64 plans against the CPU oracle, FP32 plans against FP64."""
import numpy as np
import pytest

from oracle.oracle_sponge import SimSponge
from sparc_flows_gb300 import model as M
from sparc_flows_gb300.solver_sponge import WaveSolverSponge

pytestmark = pytest.mark.gpu
NSTEPS = 7


def _inputs(nx, nz, nb):
    x = np.arange(nx) / nx - 0.5
    pats = np.stack([np.exp(-((x - 0.02 * b) ** 2) / 0.002) for b in range(nb)])
    return M.polytrope(nz), nx * 0.78125e8, pats, np.sin(np.arange(NSTEPS + 5) * 0.3 + 0.2) * 1e-6


def _gpu(nx, nz, nb, option, precision):
    model, xl, pats, amp = _inputs(nx, nz, nb)
    box, boz = M.potential_field(nx, model, xl, 80.0) if option == 12 else (None, None)
    ws = WaveSolverSponge(nx, model, xl, nbatch=nb, precision=precision, steps_out=2, obsheight_cm=-100e5,
                          option=option, box=box, boz=boz)
    ws.set_source(pats, amp)
    ws.reset(0)
    seis = ws.forward(NSTEPS).double().cpu().numpy()
    st = ws.state().double().cpu().numpy()
    ws.close()
    return st, seis


@pytest.mark.parametrize("option", [5, 6, 12])
@pytest.mark.parametrize("nx,nz,nb", [(64, 100, 1), (128, 217, 9), (192, 151, 2), (256, 300, 20), (384, 131, 1),
                                      (768, 90, 7), (1024, 100, 2)])
def test_passes_match_oracle(option, nx, nz, nb):
    st, seis = _gpu(nx, nz, nb, option, 64)
    model, xl, pats, amp = _inputs(nx, nz, nb)
    for b in {0, nb - 1}:
        s = SimSponge(nx, model, xl, steps_out=2, obsheight_cm=-100e5, option=option)
        if option == 12:
            s.set_magnetic(*M.potential_field(nx, model, xl, 80.0))
        s.set_source(pats[b], amp)
        rec = s.run(NSTEPS)
        want = s.state()
        s.close()
        for v in range(st.shape[0]):
            assert np.linalg.norm(st[v, :, b] - want[v]) <= 1e-10 * np.linalg.norm(want[v]), v
        assert np.linalg.norm(seis[:, b] - rec) <= 1e-10 * np.linalg.norm(rec) and rec.shape[0] == 4
    st32, seis32 = _gpu(nx, nz, nb, option, 32)
    for v in range(st.shape[0]):
        assert np.linalg.norm(st32[v] - st[v]) <= 1e-4 * np.linalg.norm(st[v]), v
    assert np.linalg.norm(seis32 - seis) <= 1e-4 * np.linalg.norm(seis)
