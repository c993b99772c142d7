"""Chunk lengths, block widths and coupling windows of the partitioned column solve: the host form at
short chunks against the oracle's dbyd2, and FP64 plans whose geometry differs (odd depths, one to
twelve solves) against the oracle's step."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from sparc_flows_gb300 import capi
from sparc_flows_gb300 import model as M
from sparc_flows_gb300.config import RunConfig

DP = ctypes.POINTER(ctypes.c_double)


@pytest.mark.parametrize("ibc", [0, 1])
@pytest.mark.parametrize("nz,lmax", [(16, 8), (34, 8), (99, 8), (160, 8), (199, 10), (250, 13), (320, 16)])
def test_windowed_coupling_matches_dbyd2(nz, lmax, ibc):
    b = np.random.default_rng(nz).standard_normal((nz, 4)) * np.exp(-np.linspace(0.0, 16.0, nz))[:, None]
    out = np.zeros_like(b)
    assert capi.lib().sparc_zsolve_host(nz, ibc, lmax, b.ctypes.data_as(DP), out.ctypes.data_as(DP), None, 4) == 0
    ref = O.dbyd2(b, ibc)
    # row by row: the values fall by 1e7 over the depth, as pressure does
    scale = np.maximum.accumulate(np.abs(ref).max(1)[::-1])[::-1]
    assert (np.abs(out - ref).max(1) <= 1e-12 * scale).all()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,nz,nb", [(64, 90, 1), (128, 151, 2), (192, 217, 3), (256, 320, 12)])
def test_fp64_geometry_matches_sixteen_row_chunks(nx, nz, nb):
    """The chosen chunk length and width against 8-column blocks of 16-row chunks (column_block = 8) on the
    same inputs.  Both solve the same systems; 31 steps x 5 stages x 4 solves of condition below 20 round
    to 31 * 5 * 4 * 20 * 1.1e-16 = 1.4e-12 at most."""
    from sparc_flows_gb300.solver import WaveSolver
    run = RunConfig(nx=nx, nz=nz, xlength_cm=nx * 0.78125e8, nsteps=31, flows=True)
    model = M.polytrope(nz)
    psi = M.gaussian_psi(run, model, M.psi_amplitude_for_peak(run, model, 240.0))
    out = []
    for block in (0, 8):
        ws = WaveSolver(run, model, nbatch=nb, precision=64, psi=psi, column_block=block)
        ws.set_forward_sources([M.SourceSpec(4.0 * i - 8.0) for i in range(nb)])
        out.append([ws.forward().cpu().numpy(), ws.state().cpu().numpy()])
        ws.close()
    for a, b in zip(*out):
        assert np.abs(b).max() > 0 and np.linalg.norm(a - b) <= 1.4e-12 * np.linalg.norm(b)
