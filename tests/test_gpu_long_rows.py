"""Rows of 768 (FP64) and 1024 columns, whose transforms are shared by two warps: x-derivatives of few and many rows whose
largest value lies in either warp's part, the 2-D row pass and the kernel integral against the CPU oracle, FP32 against
FP64."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from sparc_flows_gb300 import model as M
from sparc_flows_gb300.config import RunConfig

pytestmark = pytest.mark.gpu
SIZES = [768, 1024]


def _run(nx, nsteps=31):
    return RunConfig(nx=nx, nz=300, xlength_cm=nx * 0.78125e8, nsteps=nsteps, flows=True, npmlbot=20)


def _spec(x):
    return M.SourceSpec(x, spatial=M.SPATIAL_REFERENCE, temporal=M.TEMPORAL_REFERENCE)


def rel_l2(a, b):
    a, b = np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("precision", [32, 64])  # of the plan: its set-up's transform and its step's
@pytest.mark.parametrize("nx", SIZES)
def test_derivative_of_each_row(nx, precision):
    """A transform of N points rounds to about 10 eps of its row's norm, and the derivative of white noise weighs
    no wavenumber by more than 2 of its root mean square: 1e-14.  Rows share a transform, not its scale."""
    from sparc_flows_gb300.solver import WaveSolver
    ws = WaveSolver(_run(nx), M.polytrope(300), nbatch=1, precision=precision,
                    psi=np.zeros((300, nx)))
    rng = np.random.default_rng(nx)
    k = 2 * np.pi * np.arange(nx // 2 + 1)
    k[-1] = 0.0
    for rows in (1, 2, 3, 305, 2433):
        v = rng.standard_normal((rows, nx))
        v[::3] *= 1e-200
        v[1::7, nx - 1] *= 1e9
        v[2::7, 0] *= 1e9
        if rows > 4:
            v[4] = 0.0
        src = torch.as_tensor(v, device="cuda")
        out = torch.empty_like(src)
        ws.ddx(src, out, nrows=rows, stretchx=0.75)
        want = np.fft.irfft(np.fft.rfft(v, axis=1) * (0.75j * k), n=nx, axis=1)
        err = np.linalg.norm(out.cpu().numpy() - want, axis=1)
        assert (err <= 1e-13 * np.linalg.norm(want, axis=1)).all(), rows
    ws.close()


@pytest.mark.parametrize("nx", SIZES)
def test_step_and_kernels_match_oracle(nx):
    from sparc_flows_gb300.pipeline import FwdAdjKernels, receiver_columns
    from sparc_flows_gb300.solver import WaveSolver
    run, model = _run(nx), M.polytrope(300)
    psi = M.gaussian_psi(run, model, M.psi_amplitude_for_peak(run, model, 240.0))
    cmul, specs = M.c_bump(run, model), [_spec(4.0 * b) for b in range(3)]
    out = {}
    for precision in (64, 32):
        ws = WaveSolver(run, model, nbatch=3, precision=precision, psi=psi, cmul=cmul)
        ws.set_forward_sources(specs)
        out[precision] = ws.forward().cpu().numpy(), ws.state().cpu().numpy()
        ws.close()
    spec = specs[2]
    fw = O.OracleSim(run, model, cmul=cmul)
    fw.set_psi(psi)
    fw.set_forward_source(spec.xloc, spec.spatial, spec.sigma, spec.temporal, spec.nu0, run.nsteps + 8)
    seis, fsn = fw.run_steps(run.nsteps, snapshots=True)
    want = fw.get("a").reshape(6, 300, nx)[[0, 2, 3, 5]]
    assert rel_l2(out[64][0][2], seis) < 1e-10
    for f in range(4):
        assert rel_l2(out[64][1][2, f], want[f]) < 1e-10, f
        assert rel_l2(out[32][1][:, f], out[64][1][:, f]) < 1e-4, f
    assert rel_l2(out[32][0], out[64][0]) < 1e-4
    rcv = receiver_columns(run, n=32, x0=-62.0, dx=4.0)
    src = np.zeros_like(seis)
    src[:, rcv] = seis[::-1][:, rcv]
    ad = O.OracleSim(run.replace(adjoint=True), model, cmul=cmul)
    ad.set_psi(psi)
    ad.set_adjoint_source(src, run.replace(adjoint=True).num_steps)
    ker = fw.kernels(fsn, ad.run_steps(run.nsteps, snapshots=True)[1])
    fw.close()
    ad.close()
    pipe = FwdAdjKernels(run, model, [spec], psi=psi, cmul=cmul, precision=64, receivers=rcv)
    pipe.run_all()
    got = {k: v.cpu().numpy()[0] for k, v in pipe.final_kernels(summed=False).items()}
    pipe.close()
    for name in ("kernel_c", "kernel_vx", "kernel_vz", "hessian"):
        assert np.abs(ker[name]).max() > 0 and rel_l2(got[name], ker[name]) < 1e-9, name
