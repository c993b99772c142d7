"""FP32 row pass of 192, 384 and 768 columns at the batch sizes where its stages 2 to 5 run with fewer registers a thread: a
solve of such a batch has the bits it has alone, and tracks FP64."""
import numpy as np
import pytest

from sparc_flows_gb300 import model as M
from sparc_flows_gb300.config import RunConfig

pytestmark = pytest.mark.gpu


# rows (solves x levels) just inside both ends of (4864, 7296] at 192, (2432, 3648] at 384 and (1216, 2432] at 768, and
# outside
@pytest.mark.parametrize("nx,nz,nb", [(192, 271, 18), (192, 256, 28), (192, 271, 17), (384, 271, 9), (384, 256, 14),
                                      (384, 157, 24), (768, 246, 5), (768, 300, 8), (768, 174, 14)])
def test_bits_of_a_solve(nx, nz, nb):
    from sparc_flows_gb300.solver import WaveSolver
    run = RunConfig(nx=nx, nz=nz, xlength_cm=nx * 0.78125e8, nsteps=31, flows=True, npmlbot=20)
    model = M.polytrope(nz)
    psi = M.gaussian_psi(run, model, M.psi_amplitude_for_peak(run, model, 200.0))

    def forward(precision, solves):
        ws = WaveSolver(run, model, nbatch=len(solves), precision=precision, psi=psi)
        ws.set_forward_sources([M.SourceSpec(2.0 * b - nb, spatial=M.SPATIAL_REFERENCE, temporal=M.TEMPORAL_REFERENCE)
                                for b in solves])
        out = ws.forward().cpu().numpy(), ws.state().cpu().numpy()
        ws.check()
        ws.close()
        return out

    many = forward(32, range(nb))
    for b in (0, nb // 2, nb - 1):
        one, exact = forward(32, [b]), forward(64, [b])
        for m, o, e in zip(many, one, exact):
            assert np.abs(e).max() > 0 and np.array_equal(m[b], o[0])
            assert np.linalg.norm(o[0] - e[0]) <= 1e-4 * np.linalg.norm(e[0])
