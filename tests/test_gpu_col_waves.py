"""FP64 column pass with fewer registers a thread, taken where that saves a wave of blocks: a solve of such a batch has
the bits it has alone (narrower blocks, more registers) and matches the CPU oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from sparc_flows_gb300 import model as M
from sparc_flows_gb300.config import RunConfig

pytestmark = pytest.mark.gpu


# chunks of 8 and of 10 rows; 7, 6, 5 and 8 warps a block; the first and the last batch of a wave, and one beyond
@pytest.mark.parametrize("nx,nz,nb", [(512, 217, 5), (512, 217, 7), (256, 240, 12), (768, 158, 6), (256, 300, 10),
                                      (256, 300, 14), (256, 300, 15)])
def test_bits_of_a_solve(nx, nz, nb):
    from sparc_flows_gb300.solver import WaveSolver
    run = RunConfig(nx=nx, nz=nz, xlength_cm=nx * 0.78125e8, nsteps=16, flows=True, npmlbot=20)
    model = M.polytrope(nz)
    psi = M.gaussian_psi(run, model, M.psi_amplitude_for_peak(run, model, 200.0))
    specs = [M.SourceSpec(2.0 * b - nb, spatial=M.SPATIAL_REFERENCE, temporal=M.TEMPORAL_REFERENCE) for b in range(nb)]

    def forward(s):
        ws = WaveSolver(run, model, nbatch=len(s), precision=64, psi=psi)
        ws.set_forward_sources(s)
        out = ws.forward().cpu().numpy(), ws.state().cpu().numpy()
        ws.close()
        return out

    many = forward(specs)
    for b in (0, nb - 1):
        for m, o in zip(many, forward([specs[b]])):
            assert np.abs(o).max() > 0 and np.array_equal(m[b], o[0])
    spec = specs[-1]
    sim = O.OracleSim(run, model)
    sim.set_psi(psi)
    sim.set_forward_source(spec.xloc, spec.spatial, spec.sigma, spec.temporal, spec.nu0, run.nsteps + 8)
    seis = sim.run_steps(run.nsteps)
    want = sim.get("a").reshape(6, nz, nx)[[0, 2, 3, 5]]
    sim.close()
    # set-up by differences of neighbouring levels: 1.7e-10 between the two at 90 levels, where the cancellation is
    # the same; 1e-9 of each field
    assert np.linalg.norm(many[0][-1] - seis) <= 1e-9 * np.linalg.norm(seis)
    for f in range(4):
        assert np.linalg.norm(many[1][-1, f] - want[f]) <= 1e-9 * np.linalg.norm(want[f]), f
