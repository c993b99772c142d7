"""Performance cases of the wave solver: the calls its users make, over the sizes they make them at.

Every case goes through a public entry point: ``WaveSolver`` and ``FwdAdjKernels`` (2-D option 17),
``WaveSolver3D`` and ``FwdAdjKernels3D`` (option 16), ``WaveSolverSponge`` (options 5, 6, 12),
``autograd.exact_records`` (exact discrete adjoint), ``TTAdjoint`` (travel-time adjoint source)
and ``gradient`` (grad.py).  Runs are the first steps of the runs that a user makes: a production
run has 1800 to 3600 steps that all cost the same, so 16 to 61 of them stand for it.

``exact`` states what each pass computes in plain FP64 torch: derivatives along z as dense
matrices (the compact scheme's tridiagonal solve), along x and y by torch.fft, every right-hand
side as whole-field arithmetic, and gradients by torch.autograd through those steps.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from sparc_flows_gb300 import model as M
from sparc_flows_gb300.config import RunConfig

DEV = "cuda"
F64 = torch.float64
MM = 1e8                                    # cm
RSUN, DIMC, DIMRHO = 6.95989467700e10, 1.0e6, 1.0e-3
PI = 3.141592653589793
CELL_MM = 0.78125                           # horizontal spacing of every 2-D grid of the repository
FFT_SIZES = (64, 128, 192, 256, 384, 512, 768, 1024)


def f32(v):
    """A single-precision literal of the reference."""
    return float(np.float32(v))


# ------------------------------------------------------------------------------------------------
# cases
# ------------------------------------------------------------------------------------------------
def listed():
    return [
        # one source on the plain FP64 grid, no flow: the reference's own use, one small solve, all latency
        dict(name="forward64_one_256", kind="forward", precision=64, nx=256, nz=300, nb=1, steps=31, flows=False,
             cbump=False, per_solve=False, npmlbot=10),
        # one source through a supergranule in FP32: a single interactive forward run
        dict(name="forward32_one_512", kind="forward", precision=32, nx=512, nz=300, nb=1, steps=61, flows=True,
             cbump=False, per_solve=False, npmlbot=20),
        # line search: seven trial models of a smaller, odd-depth box in FP32, a background per solve
        dict(name="forward32_trials_192", kind="forward", precision=32, nx=192, nz=217, nb=7, steps=31, flows=True,
             cbump=True, per_solve=True, npmlbot=20),
        # the batch of an inversion iteration: forward, adjoint and kernels of 32 sources
        dict(name="kernels32_batch32_512", kind="kernels", precision=32, nx=512, nz=300, nb=32, steps=46, flows=True,
             cbump=True, per_solve=False, npmlbot=20, checkpoint=0),
        # a group of the uneven batch, forward field checkpointed and recomputed
        dict(name="kernels32_uneven_384", kind="kernels", precision=32, nx=384, nz=300, nb=5, steps=46, flows=True,
             cbump=True, per_solve=True, npmlbot=20, checkpoint=2),
        # the same kernels in FP64, as accuracy reports run them
        dict(name="kernels64_batch4_256", kind="kernels", precision=64, nx=256, nz=300, nb=4, steps=31, flows=True,
             cbump=True, per_solve=False, npmlbot=20, checkpoint=0),
        # the 3-D configuration: four sources on 256 x 256 x 300 with the outflow
        dict(name="forward3d32_batch4_256", kind="forward3d", precision=32, nx=256, ny=256, nz=300, nb=4, steps=4,
             flows=True),
        # a small 3-D forward + adjoint + kernel run in FP64 with checkpoints
        dict(name="kernels3d64_64", kind="kernels3d", precision=64, nx=64, ny=64, nz=100, nb=2, steps=31, flows=True,
             checkpoint=15),
        # velocity formulation with the sponge, a batch of sources in FP32
        dict(name="velocity32_sponge_512", kind="velocity", precision=32, option=5, nx=512, nz=300, nb=8, steps=31),
        # the magnetic velocity formulation, one source in FP64
        dict(name="velocity64_mhd_128", kind="velocity", precision=64, option=12, nx=128, nz=300, nb=1, steps=16),
        # exact gradient of a waveform misfit by the discrete adjoint, one source
        dict(name="exact_gradient64_256", kind="gradient", precision=64, nx=256, nz=300, nb=1, steps=31, npmlbot=10),
        # one iteration's travel-time adjoint sources, all nine ridges, and the gradient post-processing
        dict(name="traveltime64_8_512", kind="traveltime", nx=512, nt=241, nb=8, nz=300),
    ]


def depth(rng, lo, hi):
    """A number of levels in [lo, hi] that the plans take: the last of the equal chunks of at most 16
    levels must hold two."""
    while True:
        nz = rng.randint(lo, hi)
        n = -(-nz // 16)
        if nz - (n - 1) * (-(-nz // n)) >= 2:
            return nz


def spread(rng, lo, hi):
    """A whole number in [lo, hi], uniform in its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "kernels", "kernels", "forward3d", "kernels3d", "velocity", "velocity",
                       "gradient", "traveltime"])
    precision = rng.choice([32, 64])
    if kind in ("forward", "kernels"):
        nx = rng.choice(FFT_SIZES)
        nb = spread(rng, 1, 32 if precision == 32 else 6)
        case = dict(kind=kind, precision=precision, nx=nx, nz=depth(rng, 150, 320), nb=nb, steps=rng.randint(31, 46),
                    flows=rng.random() < 0.8, cbump=rng.random() < 0.6, per_solve=rng.random() < 0.3,
                    npmlbot=rng.choice([10, 15, 20]))
        if kind == "kernels":
            case["checkpoint"] = rng.choice([0, 0, 1, 2])
        while case["nb"] * nx > 32 * 512:
            case["nb"] = max(1, case["nb"] // 2)
        return case
    if kind in ("forward3d", "kernels3d"):
        nx, ny = rng.choice([64, 128, 192, 256]), rng.choice([64, 128, 192])
        case = dict(kind=kind, precision=precision, nx=nx, ny=ny, nz=depth(rng, 60, 200), nb=rng.randint(1, 2),
                    steps=rng.randint(3, 6), flows=rng.random() < 0.7)
        if kind == "kernels3d":
            case.update(precision=64, nx=min(nx, 128), ny=64, steps=rng.randint(31, 33), checkpoint=rng.randint(5, 20))
            case["nz"] = min(case["nz"], 100)
        return case
    if kind == "velocity":
        return dict(kind=kind, precision=64 if (opt := rng.choice([5, 6, 12])) == 12 else precision, option=opt,
                    nx=rng.choice(FFT_SIZES), nz=depth(rng, 90, 320), nb=spread(rng, 1, 12), steps=rng.randint(11, 31))
    if kind == "gradient":
        return dict(kind=kind, precision=64, nx=rng.choice([128, 192, 256, 384, 512]), nz=depth(rng, 200, 320),
                    nb=rng.randint(1, 2), steps=rng.randint(31, 36), npmlbot=rng.choice([10, 20]))
    return dict(kind="traveltime", nx=rng.choice([128, 192, 256, 384, 512]), nt=rng.randint(180, 300),
                nb=spread(rng, 1, 16), nz=depth(rng, 90, 320))


# ------------------------------------------------------------------------------------------------
# inputs, from the case and the seed alone
# ------------------------------------------------------------------------------------------------
def run_config(c):
    return RunConfig(nx=c["nx"], nz=c["nz"], xlength_cm=c["nx"] * CELL_MM * MM, nsteps=c["steps"],
                     flows=bool(c.get("flows", True)), npmlbot=c["npmlbot"])


@functools.lru_cache(maxsize=None)
def flow_amplitude(nx, nz):
    run = RunConfig(nx=nx, nz=nz, xlength_cm=nx * CELL_MM * MM)
    return M.psi_amplitude_for_peak(run, M.polytrope(nz), 1.0)


def inputs_2d(c, seed):
    """RunConfig, model, source positions, psi and cmul ((nz, nx), a list of nb of them, or None)."""
    run, model = run_config(c), M.polytrope(c["nz"])
    rng = np.random.default_rng(seed)
    box = c["nx"] * CELL_MM
    xs = [float(v) for v in box * rng.uniform(-0.35, 0.35, c["nb"])]
    n = c["nb"] if c.get("per_solve") else 1
    psi = [M.gaussian_psi(run, model, flow_amplitude(c["nx"], c["nz"]) * float(rng.uniform(60.0, 300.0)),
                          x0=float(rng.uniform(-0.1, 0.1)) * box) for _ in range(n)] if run.flows else None
    cmul = [M.c_bump(run, model, float(rng.uniform(0.01, 0.05)), x0=float(rng.uniform(-0.1, 0.1)) * box)
            for _ in range(n)] if c.get("cbump") else None
    if not c.get("per_solve"):
        psi, cmul = (v[0] if v else None for v in (psi, cmul))
    return run, model, xs, psi, cmul


# Sources: the reference's own profile and time function, whose first steps already carry signal
def source_specs(xs):
    return [M.SourceSpec(x, spatial=M.SPATIAL_REFERENCE, temporal=M.TEMPORAL_REFERENCE) for x in xs]


@functools.lru_cache(maxsize=2)
def outflow(nx, ny, nz):
    return M.outflow_3d(nx, ny, M.polytrope(nz), nx * CELL_MM * MM)


def inputs_3d(c, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nb, xl = c["nx"], c["ny"], c["nb"], c["nx"] * CELL_MM
    half = 0.35 * xl
    pats = np.stack([M.point_source_pattern(nx, ny, xl * MM, *rng.uniform(-half, half, 2)) for _ in range(nb)])
    amp = 1e-6 * np.sin(0.35 * np.arange(c["steps"] + 8) + rng.uniform(0.2, 1.2))
    flow = [float(rng.uniform(0.5, 1.0)) * v for v in outflow(nx, ny, c["nz"])] if c["flows"] else None
    return M.polytrope(c["nz"]), xl * MM, pats, amp, flow


def inputs_velocity(c, seed):
    rng = np.random.default_rng(seed)
    nx, nb = c["nx"], c["nb"]
    x = np.arange(nx) / nx - 0.5
    pats = np.stack([np.exp(-((x - x0) * nx * CELL_MM) ** 2 / 8.0) for x0 in rng.uniform(-0.35, 0.35, nb)])
    amp = 1e-6 * np.sin(0.3 * np.arange(c["steps"] + 8) + rng.uniform(0.2, 1.2))
    model = M.polytrope(c["nz"])
    field = M.potential_field(nx, model, nx * CELL_MM * MM, float(rng.uniform(50.0, 100.0))) if c["option"] == 12 else (None, None)
    return model, nx * CELL_MM * MM, pats, amp, field


def inputs_traveltime(c, seed):
    """Records of a travelling, dispersing packet with noise, data arriving a little later; kernels
    and hessians of every source; the measured modes."""
    rng = np.random.default_rng(seed)
    nb, nt, nx = c["nb"], c["nt"], c["nx"]
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    x0 = rng.uniform(-0.2, 0.2, nb) * nx * CELL_MM
    x = torch.as_tensor((np.arange(nx) / nx - 0.5) * nx * CELL_MM, device=DEV)
    d = (x[None, :] - torch.as_tensor(x0, device=DEV)[:, None]).abs()[:, None, :]
    t = (torch.arange(nt, dtype=F64, device=DEV) * 0.5)[None, :, None]  # minutes

    def packet(delay):
        out = 0.0
        for vel, f in ((0.5, 0.18), (0.8, 0.2), (1.2, 0.22), (1.7, 0.24)):
            a = t - d / vel - 6.0 - delay
            out = out + torch.exp(-(a / 8.0) ** 2) * torch.cos(2 * PI * f * a)
        return out

    noise = lambda: 1e-2 * torch.randn((nb, nt, nx), generator=g, dtype=F64, device=DEV)  # noqa: E731
    synth, data = packet(0.0) + noise(), packet(float(rng.uniform(0.05, 0.3))) + noise()
    kern = torch.randn((nb, c["nz"], nx), generator=g, dtype=F64, device=DEV)
    hess = torch.randn((nb, c["nz"], nx), generator=g, dtype=F64, device=DEV) ** 2
    far = min(60.0, 0.25 * nx * CELL_MM)
    modes = {p: (5.0, far, 10.0 + p) for p in range(9)}
    return synth, data, [float(v) for v in x0], np.arange(nt) * 0.5, modes, kern, hess


def misfit_weights(c, seed, nrec, nrcv):
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
    return torch.randn((c["nb"], nrec, nrcv), generator=g, dtype=F64, device=DEV)


RECEIVERS = 32


def receivers(nx):
    return np.linspace(0.1 * nx, 0.9 * nx, RECEIVERS).astype(int)


def record_height(nz):
    """Height (cm) of the 3-D records: the default where the grid reaches above it, else near the sources."""
    return 200e5 if nz >= 200 else -100e5


# ------------------------------------------------------------------------------------------------
# prepare, run
# ------------------------------------------------------------------------------------------------
class State(dict):
    """What the program holds; its plans are closed with it."""

    def __del__(self):
        for v in self.values():
            if hasattr(v, "close"):
                v.close()


def prepare(case, seed):
    kind = case["kind"]
    s = State(case=dict(case))
    if kind == "forward":
        from sparc_flows_gb300.solver import WaveSolver
        run, model, xs, psi, cmul = inputs_2d(case, seed)
        s["solver"] = WaveSolver(run, model, nbatch=case["nb"], precision=case["precision"], psi=psi, cmul=cmul)
        s["solver"].set_forward_sources(source_specs(xs))
    elif kind == "kernels":
        from sparc_flows_gb300.pipeline import FwdAdjKernels
        run, model, xs, psi, cmul = inputs_2d(case, seed)
        s["pipe"] = FwdAdjKernels(run, model, source_specs(xs), psi=psi, cmul=cmul, precision=case["precision"],
                                  receivers=receivers(case["nx"]), checkpoint_every=case["checkpoint"] or None)
    elif kind == "forward3d":
        from sparc_flows_gb300.solver3d import WaveSolver3D
        model, xl, pats, amp, flow = inputs_3d(case, seed)
        w = s["solver"] = WaveSolver3D(case["nx"], case["ny"], model, xl, nbatch=case["nb"], precision=case["precision"],
                                       steps_out=2, flows=flow is not None, obsheight_cm=record_height(case["nz"]))
        if flow is not None:
            w.set_flow(*flow)
        w.set_source(pats, amp)
    elif kind == "kernels3d":
        from sparc_flows_gb300.pipeline3d import FwdAdjKernels3D
        model, xl, pats, amp, flow = inputs_3d(case, seed)
        s["pipe"] = FwdAdjKernels3D(case["nx"], case["ny"], model, xl, pats, amp, case["steps"], flow=flow,
                                    precision=case["precision"], steps_out=5, checkpoint_every=case["checkpoint"],
                                    obsheight_cm=record_height(case["nz"]))
    elif kind == "velocity":
        from sparc_flows_gb300.solver_sponge import WaveSolverSponge
        model, xl, pats, amp, (box, boz) = inputs_velocity(case, seed)
        s["solver"] = WaveSolverSponge(case["nx"], model, xl, nbatch=case["nb"], precision=case["precision"],
                                       steps_out=5, option=case["option"], box=box, boz=boz)
        s["solver"].set_source(pats, amp)
    elif kind == "gradient":
        from sparc_flows_gb300.discrete_adjoint import ExactGradient
        from sparc_flows_gb300.solver import WaveSolver
        run, model, xs, psi, _ = inputs_2d(case, seed)
        s["solver"] = WaveSolver(run, model, nbatch=case["nb"], precision=64, psi=psi)
        s["solver"].set_forward_sources(source_specs(xs))
        s["exact"] = ExactGradient(s["solver"], receivers(case["nx"]), segment=10)
        s["psi"] = torch.as_tensor(psi, dtype=F64, device=DEV)
        s["weights"] = misfit_weights(case, seed, run.nrec, RECEIVERS)
    else:
        from sparc_flows_gb300 import gradient as G
        from sparc_flows_gb300.ttadjoint import TTAdjoint
        nx = case["nx"]
        s["inputs"] = inputs_traveltime(case, seed)
        s["tt"] = TTAdjoint(nx, case["nt"], case["nb"], nx * CELL_MM * MM, 30.0)
        s["rho"] = torch.as_tensor(np.ascontiguousarray(M.polytrope(case["nz"])[:, 2]), device=DEV)
        s["work"] = G.Workspace(nx, case["nz"])
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "forward":
        return {"seis": s["solver"].forward(c["steps"]), "state": s["solver"].state()}
    if kind in ("kernels", "kernels3d"):
        # the integrands of an FP32 run are accumulated in FP64 and kept, as its records, in its own precision
        seis, kacc = s["pipe"].run_all()
        parts = kacc.to(seis.dtype).unbind(1 if kind == "kernels" else 0)
        return {"seis": seis, "kernels": list(parts)}
    if kind in ("forward3d", "velocity"):
        s["solver"].reset(0)
        return {"seis": s["solver"].forward(c["steps"]), "state": s["solver"].state()}
    if kind == "gradient":
        from sparc_flows_gb300.autograd import exact_records
        psi = s["psi"].detach().requires_grad_(True)
        rec = exact_records(psi, s["exact"])
        (grad,) = torch.autograd.grad((rec,), (psi,), (s["weights"],))
        last = s["exact"].last
        return {"records": rec.detach(), "psi": grad, "v0x": last["v0x"], "v0z": last["v0z"], "c2rho0": last["c2rho0"]}
    from sparc_flows_gb300 import gradient as G
    synth, data, x0, t, modes, kern, hess = s["inputs"]
    res = s["tt"].run(synth, data, x0, t, modes, {"allmodes": (1.5, 6.0)})
    g = G.gradient_psi(kern, hess, s["rho"], ws=s["work"])
    u, beta = G.update_direction("cg", g, kern[0], hess[0], ws=s["work"])
    trial = G.linesearch_models(g, u, [0.01, 0.02, 0.03], ws=s["work"])
    windows = np.zeros((9, c["nb"], c["nx"], 2), dtype=np.int64)
    for p, sources in res["rows"].items():
        for b, rows in sources.items():
            for i, _, left, right, *_ in rows:
                windows[p, b, i - 1] = left, right
    return {"adjoint": res["adj"], "misfit": res["misfit"], "measured": res["nmeas"], "windows": windows, "gradient": g,
            "update": u, "beta": beta, "trial": trial}


# ------------------------------------------------------------------------------------------------
# work: a time step couples every point of a row and of a column in each of its five stages, so the
# live fields cross memory once a stage.  Words of one step of one point: 15 per live field (state and
# right-hand side in and out), 5 per background field that varies over the grid, 10 for the filter.
# ------------------------------------------------------------------------------------------------
def point_flops(nx, ny, ndx, ndy, ndz):
    """One stage of one point: spectral derivatives (two real transforms each), compact ones, the rest."""
    return ndx * 5 * math.log2(nx) + ndy * 5 * math.log2(max(ny, 2)) + 12 * ndz + 30


def work(case):
    c, kind = case, case["kind"]
    w = c.get("precision", 64) // 8
    if kind in ("forward", "kernels", "gradient"):
        n = c["nx"] * c["nz"] * c["nb"]
        flows = 2 if c.get("flows", True) else 0
        shared = 1.0 if c.get("per_solve") else 1.0 / c["nb"]
        words = 15 * 4 + 10 + 5 * (flows + (1 if c.get("cbump") else 0)) * shared
        nd = 4 if flows else 2
        step = {"bytes": n * w * words, "flops": n * 5 * point_flops(c["nx"], 1, nd, 0, nd)}
        # forward and adjoint; with checkpoints the forward run again; the exact gradient recomputes and transposes
        solves = {"forward": 1, "kernels": 3 if c.get("checkpoint") else 2, "gradient": 5}[kind]
        records = c["steps"] // 15 + 1 if kind == "kernels" else 0
        return {"bytes": step["bytes"] * c["steps"] * solves + records * n * (12 * w + 64),
                "flops": step["flops"] * c["steps"] * solves}
    if kind in ("forward3d", "kernels3d"):
        n = c["nx"] * c["ny"] * c["nz"] * c["nb"]
        flows = 3 if c["flows"] else 0
        words = 15 * 6 + 10 + 5 * flows / c["nb"]
        nd = 2 + flows
        solves = 3 if kind == "kernels3d" else 1
        records = (c["steps"] - 1) // 5 + 1 if kind == "kernels3d" else 0
        return {"bytes": n * w * words * c["steps"] * solves + records * n * (10 * w + 80),
                "flops": n * 5 * point_flops(c["nx"], c["ny"], nd, nd, nd) * c["steps"] * solves}
    if kind == "velocity":
        n = c["nx"] * c["nz"] * c["nb"]
        live, back, nd = (6, 3, 4) if c["option"] == 12 else (4, 0, 2)
        return {"bytes": n * w * (15 * live + 10 + 5 * back / c["nb"]) * c["steps"],
                "flops": n * 5 * point_flops(c["nx"], 1, nd, 0, nd) * c["steps"]}
    n, m = c["nx"] * c["nt"] * c["nb"], c["nx"] * c["nz"]
    return {"bytes": 8.0 * (3 * n + 2 * c["nb"] * m + 7 * m),
            "flops": 9.0 * n * 4 * 5 * math.log2(c["nx"] * c["nt"]) + 12.0 * c["nb"] * m}


# ------------------------------------------------------------------------------------------------
# exact: the same passes in plain FP64 torch
# ------------------------------------------------------------------------------------------------
def t64(v):
    return torch.as_tensor(np.ascontiguousarray(v), dtype=F64, device=DEV)


def compact_matrix(n, ibc):
    """The compact z-derivative (dbyd2.f) as a dense matrix, and its response to a given top value
    (ibc 3).  ibc 0: zero at both ends, 1: one-sided closures, 2: zero at the bottom, 3: given at the top.
    The reference's coefficients are single precision."""
    s = np.float32
    d = s(n - 1)
    c1, c2 = d * s(7) / s(9), d / s(36)
    b = [-(s(43) / s(96) * d), -(s(5) / s(6) * d), s(9) / s(8) * d, s(1) / s(6) * d, -(s(1) / s(96) * d)]
    f = [-(s(10) / s(3) * d), -(s(3) * d), s(6) * d, s(1) / s(3) * d, s(0)]
    alpha, alpha2, gamma2 = s(1) / s(3), s(0.75), s(0.125)
    cn = s(1) / (alpha2 - s(3) * gamma2)
    up = (s(6) * alpha2 - s(3)) * cn
    b, f = np.array(b, dtype=np.float64), np.array(f, dtype=np.float64)
    end = (float(alpha2) * f - 3.0 * b) * float(cn)
    rhs, tri = np.zeros((n, n)), np.eye(n)
    for k in range(2, n - 2):
        rhs[k, k - 2:k + 3] = [-float(c2), -float(c1), 0.0, float(c1), float(c2)]
        tri[k, k - 1] = tri[k, k + 1] = float(alpha)
    rhs[1, :5], rhs[n - 2, n - 5:] = b, -b[::-1]
    tri[1, 0], tri[1, 2] = float(gamma2), float(alpha2)
    tri[n - 2, n - 1], tri[n - 2, n - 3] = float(gamma2), float(alpha2)
    if ibc in (1, 3):
        rhs[0, :5], tri[0, 1] = end, float(up)
    if ibc in (1, 2):
        rhs[n - 1, n - 5:], tri[n - 1, n - 2] = -end[::-1], float(up)
    inv = np.linalg.inv(tri)
    return inv @ rhs, inv[:, n - 1]


TAPS = np.array([0.001953125, -0.01953125, 0.087890625, -0.234375, 0.41015625]) / 2


def filter_matrix(n, k0, k1, low_ends):
    """Rows k0..k1-1 of the 11-point filter, two-point means nearer the ends, other rows kept."""
    m = np.eye(n)
    for k in range(k0, k1):
        if 5 <= k <= n - 6:
            m[k, k - 5:k + 6] = np.concatenate([TAPS, [0.75390625], TAPS[::-1]])
        elif k > n - 6 or low_ends:
            m[k, k - 1:k + 2] = [0.5, 0.0, 0.5]
    return m


def d_spectral(v, dim, scale):
    """Derivative along a periodic axis of unit length times scale, the Nyquist bin dropped."""
    n = v.shape[dim]
    k = 2 * PI * torch.arange(n // 2 + 1, dtype=F64, device=v.device)
    k[n // 2] = 0.0
    shape = [1] * v.dim()
    shape[dim] = n // 2 + 1
    return torch.fft.irfft(torch.fft.rfft(v, dim=dim) * (1j * scale * k.reshape(shape)), n=n, dim=dim)


def betas(dt):
    o = (1.0, 0.5, f32(0.1665579725791151184), f32(0.03950410250586729987), f32(0.007810706393337838236))
    b = [0.0] * 5
    b[4] = o[1]
    b[3] = o[2] / b[4]
    b[2] = o[3] / (b[4] * b[3])
    b[1] = o[4] / (b[4] * b[3] * b[2])
    return [v * dt for v in b]


class Column:
    """The vertical grid: profiles, levels, derivative and filter matrices."""

    def __init__(self, model, obs=2.0e7):
        self.n = n = model.shape[0]
        self.z = z = model[:, 0]
        self.c, self.rho = model[:, 1] / DIMC, model[:, 2] / DIMRHO
        self.p, self.g = model[:, 3] / (DIMRHO * DIMC ** 2), model[:, 4] * RSUN / DIMC ** 2
        raw = {i: compact_matrix(n, i) for i in range(4)}
        self.unstretch = raw[1][0] @ z
        self.stretch = 1.0 / self.unstretch
        self.D = {i: t64(raw[i][0] * self.stretch[:, None]) for i in raw}
        self.top = t64(raw[3][1] * self.stretch)
        self.drho, self.dp = self.stretch * (raw[1][0] @ self.rho), self.stretch * (raw[1][0] @ self.p)
        self.dt = 2.0 * DIMC / RSUN
        self.e, self.o = self.level(-1.5e7), self.level(obs)
        self.record = t64(filter_matrix(n, 1, n - 1, True))  # FILTER_VAR_Z of the kernel stage

    def level(self, height_cm):
        d = np.abs(self.z - (1.0 + height_cm / RSUN))
        return int(np.flatnonzero(d <= d.min())[-1])

    def absorber(self, bot, top, cbot, ctop, double_bottom=1.0):
        """Damping -a and -a - alpha of the vertical layer and the decay of the background, (nz, ...)."""
        z, n = self.z, self.n
        shape = (n,) + np.shape(cbot)
        a, al = np.zeros(shape), np.zeros(shape)
        decay = np.ones(shape)
        for k in list(range(bot)) + list(range(n - top, n)):
            low = k < bot
            edge, end, c = (z[bot - 1], z[0], cbot * double_bottom) if low else (z[n - top], z[n - 1], ctop)
            width = abs(edge - end)
            alpha = PI * f32(0.005) * RSUN / DIMC * abs(z[k] - end) / width
            a[k] = 9.0 * c / width * ((edge - z[k]) / width) ** 2
            al[k] = alpha
            decay[k] = alpha / (a[k] + alpha)
        return -a, -a - al, decay


def zdot(m, v, dim):
    """The matrix m along one axis of v."""
    return torch.movedim(torch.tensordot(m, v, dims=([1], [dim])), 0, dim)


class Exact2D:
    """Option 17: the linear step of a batch as functions of the state, absorber fields and background."""

    def __init__(self, c, model, psi, cmul):
        col = self.col = Column(model)
        nx, nz, nb = c["nx"], c["nz"], c["nb"]
        self.nx, self.nz, self.nb = nx, nz, nb
        one = lambda v, d: [d if u is None else u for u in (v if isinstance(v, list) else [v])]  # noqa: E731
        cm = np.stack(one(cmul, np.ones((nz, nx))))
        speed = col.c[None, :, None] * cm
        az, bz, fd, gm = [], [], [], None
        for sp in speed:
            a, b, f = col.absorber(c["npmlbot"], 10, sp[0], sp[nz - 6])
            az.append(a), bz.append(b), fd.append(f)
            gm = col.g * f[:, 0] if gm is None else gm
        x, nh = np.arange(nx) / nx, 9
        w = np.zeros(nx)
        al = np.zeros(nx)
        for i in range(nh):
            for j, end, edge in ((i, x[0], x[nh - 1]), (nx - nh + i, x[nx - 1], x[nx - nh])):
                w[j] = 0.25 * 9.0 / abs(edge - end) * ((x[j] - edge) / (edge - end)) ** 2
                al[j] = f32(0.005) * RSUN / DIMC * PI * abs(x[j] - end) / abs(edge - end)
        ax = -speed[:, :, :1] * w
        self.xpml = t64(np.where((np.arange(nx) < nh) | (np.arange(nx) >= nx - nh), 1.0, 0.0))
        self.zpml = t64(np.where((np.arange(nz) < c["npmlbot"]) | (np.arange(nz) >= nz - 10), 1.0, 0.0))[:, None]
        self.az, self.bz = t64(np.stack(az)), t64(np.stack(bz))
        self.ax, self.bx = t64(ax), t64(ax - al)
        v = lambda a: t64(a)[:, None]  # noqa: E731
        fd = t64(np.stack(fd))
        self.gp, self.gr, self.g = v(col.dp) * fd, v(col.drho) * fd, v(gm)
        self.rho, self.c2r = v(col.rho), t64(speed ** 2 * col.rho[:, None])
        self.speed, self.kx = t64(speed), RSUN / (nx * CELL_MM * MM)
        self.ut = float(col.unstretch[nz - 1])
        self.flows = psi is not None
        if self.flows:
            self.v0x, self.v0z = self.flow(t64(np.stack(one(psi, None))))
        nofilter = torch.zeros(nx, dtype=F64, device=DEV)
        nofilter[nh - 1:nx - nh + 1] = 1.0
        self.fcols, self.F = nofilter, t64(filter_matrix(nz, 5, nz - 1, True))
        inside = torch.ones((nz, nx), dtype=F64, device=DEV)
        inside[0], inside[:, 0], inside[:, -1] = 0.0, 0.0, 0.0
        self.inside = inside

    def flow(self, psi):
        pv = self.rho * self.speed * psi / (RSUN / MM)
        return -zdot(self.col.D[1], pv, 1) / self.rho, d_spectral(pv, 2, self.kx) / self.rho

    def rhs(self, X, Z, W, sign, k_inj, forcing):
        D, xi = self.col.D, X[:, 0]
        xz, vx, vz = X[:, 1], X[:, 2], X[:, 3]
        dxx = d_spectral(xi, 2, self.kx)
        dzz = zdot(D[3], xz, 1) - self.col.top[:, None] * (dxx[:, -1:, :] * self.ut)
        Rz0 = self.az * dzz + self.bz * Z[:, 0]
        dzz = dzz + Z[:, 0]
        dxx = dxx + W[:, 0]
        Rw0 = self.ax * dxx + self.bx * W[:, 0]
        div = dxx + dzz
        p = -self.c2r * div - self.gp * xz
        gx = d_spectral(p, 2, self.kx) + W[:, 1]
        Rw1 = self.ax * gx + self.bx * W[:, 1]
        gz = zdot(D[2], p, 1)
        Rz1 = self.az * gz + self.bz * Z[:, 1]
        gz = gz + Z[:, 1]
        rho = -self.rho * div - self.gr * xz
        ax, az = -gx / self.rho, -(gz + rho * self.g) / self.rho
        if forcing is not None:
            pad = torch.zeros_like(az)
            pad[:, k_inj] = forcing
            az = az + pad
        if self.flows:
            ax = ax - 2 * sign * (self.v0x * d_spectral(vx, 2, self.kx) + self.v0z * zdot(D[1], vx, 1))
            az = az - 2 * sign * (self.v0x * d_spectral(vz, 2, self.kx) + self.v0z * zdot(D[1], vz, 1))
        R = torch.stack((vx, vz, ax, az), 1) * self.inside
        return R, torch.stack((Rz0, Rz1), 1) * self.zpml, torch.stack((Rw0, Rw1), 1) * self.xpml

    def rest(self):
        z = lambda n: torch.zeros((self.nb, n, self.nz, self.nx), dtype=F64, device=DEV)  # noqa: E731
        return z(4), z(2), z(2)

    def step(self, a, Z, W, sign=1.0, k_inj=0, forcing=None):
        """(state, absorbers) after one step, and the last stage's acceleration."""
        X, Y, V = a, Z, W
        for s, b in enumerate(betas(self.col.dt)):
            if s:
                X, Y, V = a + b * R, Z + b * RZ, W + b * RW
            R, RZ, RW = self.rhs(X, Y, V, sign, k_inj, forcing)
        dt = self.col.dt
        n = a + dt * R
        n = n + (zdot(self.F, n, 2) - n) * self.fcols
        return n, Z + dt * RZ, W + dt * RW, R[:, 2:]

    def forward_forcing(self, xs, steps):
        """FORWARD_SOURCE: profile (nb, nx) times series (steps,) times the injection factor."""
        nx, col = self.nx, self.col
        l8 = f32(1e-8)
        x, xl = np.arange(nx) / nx, nx * CELL_MM * MM
        rows = []
        for x0 in xs:
            d = (x - 0.5) * xl * l8 - x0
            with np.errstate(invalid="ignore", divide="ignore"):
                sinc = np.sin(f32(0.43) * PI * d) / (f32(0.43) * PI * d)
            sinc[int(np.argmin(np.abs(d)))] = 1.0
            rows.append(np.exp(-d * d / (400.0 * (x[1] * xl * l8) ** 2)) * sinc)
        t, nu, wid = 2.0 * np.arange(steps), f32(0.0017), f32(0.0055)
        ts = np.cos(2 * PI * nu * t) * np.exp(-2.0 * (t - 0.5 / nu) ** 2 * wid ** 2)
        ts[np.abs(ts) < f32(0.00001)] = 0.0
        scale = 2.0 / (col.z[col.e + 1] - col.z[col.e - 1]) / col.rho[col.e]
        return t64(np.stack(rows)), ts * f32(1e-5) * scale

    def forward(self, xs, steps, records=False):
        rows, ts = self.forward_forcing(xs, steps)
        a, Z, W = self.rest()
        until, seis, recs = 15 * ((steps - 1) // 15 + 1), [], []
        for n in range(steps):
            a, Z, W, acc = self.step(a, Z, W, 1.0, self.col.e, ts[n] * rows if n <= until else None)
            if n % 15 == 0:
                seis.append(a[:, 3, self.col.o])
                if records:
                    recs.append(torch.cat((a, acc), 1))
        return torch.stack(seis, 1), a, recs

    def kernels(self, xs, steps, rcv):
        """Forward, adjoint (time-reversed records at the receivers) and the four kernel integrands."""
        col = self.col
        seis, _, recs = self.forward(xs, steps, records=True)
        src = torch.zeros_like(seis)
        src[:, :, rcv] = seis.flip(1)[:, :, rcv]
        scale = 2.0 / (col.z[col.o + 1] - col.z[col.o - 1]) / col.rho[col.o]
        a, Z, W = self.rest()
        out = torch.zeros((self.nb, 4, self.nz, self.nx), dtype=F64, device=DEV)
        dz = lambda v: zdot(col.record, zdot(col.D[1], v, 1), 1)  # noqa: E731
        dx = lambda v: d_spectral(v, 2, self.kx)  # noqa: E731
        until = 15 * ((steps - 1) // 15 + 1)
        for n in range(steps):
            f = scale * interpolate(src, n, 15, steps) if n <= until else None
            a, Z, W, _ = self.step(a, Z, W, -1.0, col.o, f)
            if n % 15 == 0:
                f = recs[len(recs) - 1 - n // 15]
                ax, az = a[:, 2], a[:, 3]
                out[:, 0] += (dx(f[:, 0]) + dz(f[:, 1])) * (dx(ax) + dz(az))
                out[:, 1] += dx(f[:, 2]) * ax + dx(f[:, 3]) * az
                out[:, 2] += dz(f[:, 2]) * ax + dz(f[:, 3]) * az
                out[:, 3] += f[:, 4] ** 2 + f[:, 5] ** 2
        return seis, out


def interpolate(src, step, cadence, steps):
    """LAGRANGE_INTERP: slices src (nb, nrec, ...) of a cadence in steps, at a step (0-based): seven points, fewer
    where they would start before the first slice or pass the end of the source."""
    cad = 2.0 * cadence
    length = 2 * ((int((steps - 1) * 2.0 / cad) + 2) // 2) + 2
    t1, t = int(math.floor(step * 2.0 / cad)) + 1, 2.0 * step
    xs = [(t1 - 4 + j) * cad for j in range(7)]
    out = torch.zeros_like(src[:, 0])
    for j, r in enumerate(range(t1 - 4, t1 + 3)):
        use = xs[j] >= 0 if j < 4 else (True if j == 4 else t1 < length - (j - 5))
        if use and 0 <= r < src.shape[1]:
            w = 1.0
            for m in range(7):
                if m != j:
                    w *= (t - xs[m]) / (xs[j] - xs[m])
            out = out + w * src[:, r]
    return out


def exact_gradient(c, seed):
    run, model, xs, psi, _ = inputs_2d(c, seed)
    sim = Exact2D(c, model, psi, None)
    p = t64(psi)[None].requires_grad_(True)
    sim.v0x, sim.v0z = sim.flow(p)
    # derivatives with respect to the flow and c^2 rho0 themselves, beside those through psi
    sim.v0x.retain_grad(), sim.v0z.retain_grad()
    sim.c2r = sim.c2r.requires_grad_(True)
    seis, _, _ = sim.forward(xs, c["steps"])
    rec = seis[:, :, torch.as_tensor(receivers(c["nx"]), device=DEV)]
    (rec * misfit_weights(c, seed, run.nrec, RECEIVERS)).sum().backward()
    return {"records": rec.detach(), "psi": p.grad[0], "v0x": sim.v0x.grad[0], "v0z": sim.v0z.grad[0],
            "c2rho0": sim.c2r.grad[0]}


class Exact3D:
    """Option 16 on fields (nz, nb, ny, nx), state (6, ...)."""

    def __init__(self, c, model, xl, flow):
        col = self.col = Column(model, record_height(c["nz"]))
        n = col.n
        v = lambda a: t64(a).reshape(n, 1, 1, 1)  # noqa: E731
        az, bz, fd = col.absorber(10, 10, col.c[0], col.c[n - 1], 2.0)
        self.az, self.bz = v(az), v(bz)
        self.layer = v((az != 0) | (bz != 0))
        self.gp, self.gr, self.g = v(col.dp * fd), v(col.drho * fd), v(col.g * fd)
        self.rho, self.c2r = v(col.rho), v(col.c ** 2 * col.rho)
        dep = np.exp(-1e7 * 4.0 * (col.z - col.z[col.e]) ** 2)
        dep[np.abs(np.arange(n) - col.e) > 4] = 0.0
        self.dep, self.k = v(dep), RSUN / xl
        self.inside = torch.ones((n, 1, 1, 1), dtype=F64, device=DEV)
        self.inside[0], self.inside[n - 1] = 0.0, 0.0
        self.flow = [t64(f)[:, None] for f in flow] if flow is not None else None
        self.F = t64(filter_matrix(n, 10, n - 10, False))
        self.shape = (n, c["nb"], c["ny"], c["nx"])

    def grad(self, v, ibc):
        return d_spectral(v, 3, self.k), d_spectral(v, 2, self.k), zdot(self.col.D[ibc], v, 0)

    def rhs(self, X, Z, sign, source):
        d = [d_spectral(X[0], 3, self.k), d_spectral(X[1], 2, self.k), zdot(self.col.D[1], X[2], 0)]
        RZ0 = self.az * d[2] + self.bz * Z[0]
        div = d[0] + d[1] + d[2] + Z[0]
        g = list(self.grad(-self.c2r * div - self.gp * X[2], 0))
        RZ1 = self.az * g[2] + self.bz * Z[1]
        g[2] = g[2] + Z[1]
        g[2] = g[2] + (-self.rho * div - self.gr * X[2]) * self.g
        R = [X[3], X[4], X[5]]
        for j in range(3):
            r = -g[j] / self.rho
            if j == 2:
                r = r + source
            if self.flow is not None:
                dv = self.grad(X[3 + j], 1)
                r = r - 2 * sign * sum(f * q for f, q in zip(self.flow, dv))
            R.append(r)
        return [r * self.inside for r in R], [RZ0 * self.layer, RZ1 * self.layer]

    def step(self, a, Z, n, sign, source):
        X, Y = a, Z
        for s, b in enumerate(betas(self.col.dt)):
            if s:
                X, Y = [u + b * r for u, r in zip(a, R)], [u + b * r for u, r in zip(Z, RZ)]
            R, RZ = self.rhs(X, Y, sign, source)
        a = [u + self.col.dt * r for u, r in zip(a, R)]
        if n % 2 == 1:
            a = [zdot(self.F, u, 0) for u in a]
        return a, [u + self.col.dt * r for u, r in zip(Z, RZ)], R[3:]

    def rest(self):
        return [torch.zeros(self.shape, dtype=F64, device=DEV) for _ in range(6)], \
            [torch.zeros(self.shape, dtype=F64, device=DEV) for _ in range(2)]

    def divergence(self, f):
        return d_spectral(f[0], 3, self.k) + d_spectral(f[1], 2, self.k) + zdot(self.col.record, zdot(self.col.D[1], f[2], 0), 0)

    def forward(self, pats, amp, steps, cadence, records=False):
        a, Z = self.rest()
        pat, seis, recs = t64(pats)[None], [], []
        for n in range(steps):
            a, Z, acc = self.step(a, Z, n, 1.0, pat * float(amp[n]) * self.dep)
            if n % cadence == 0:
                seis.append(a[5][self.col.o].clone())
                if records:
                    recs.append((self.divergence(a), a[3], a[4], a[5], sum(q * q for q in acc)))
        return torch.stack(seis), torch.stack(a), recs

    def kernels(self, pats, amp, steps, cadence):
        col = self.col
        seis, _, recs = self.forward(pats, amp, steps, cadence, records=True)
        src = seis.flip(0).permute(1, 0, 2, 3)
        scale = 2.0 / (col.z[col.o + 1] - col.z[col.o - 1]) / col.rho[col.o]
        a, Z = self.rest()
        out = torch.zeros((5,) + self.shape, dtype=F64, device=DEV)
        for n in range(steps):
            # the 3-D step counter runs one step behind the 2-D one in the interpolation table
            source = torch.zeros(self.shape, dtype=F64, device=DEV)
            source[col.o] = scale * interpolate(src, n + 1, cadence, steps)
            a, Z, _ = self.step(a, Z, n, -1.0, source)
            if n % cadence == 0:
                f = recs[len(recs) - 1 - n // cadence]
                out[0] += f[0] * self.divergence(a[3:])
                for j in range(3):
                    dv = list(self.grad(f[1 + j], 1))
                    dv[2] = zdot(col.record, dv[2], 0)
                    for i in range(3):
                        out[1 + i] += dv[i] * a[3 + j]
                out[4] += f[4]
        return seis, out


def exact_velocity(c, seed):
    """Options 5, 6 and 12 on fields (nz, nb, nx): rho, v_x, v_y, v_z, p (and b_x, b_y, b_z)."""
    model, xl, pats, amp, (box, boz) = inputs_velocity(c, seed)
    col, opt = Column(model), c["option"]
    n, nx, nb = col.n, c["nx"], c["nb"]
    v = lambda a: t64(a).reshape(n, 1, 1)  # noqa: E731
    az, bz, fd = col.absorber(10, 10, col.c[0], col.c[n - 6])
    if opt == 5:
        az, bz, fd = 0 * az, 0 * bz, np.ones(n)
        sponge = (200.0 / (1.0 + np.exp((f32(1.002) - col.z) / f32(0.0001)))
                  + 300.0 / (1.0 + np.exp((col.z - (col.z[0] + f32(0.005))) / f32(0.0005))))
    else:
        sponge = np.zeros(n)
    layer = v((az != 0) | (bz != 0))
    az, bz, sponge = v(az), v(bz), v(sponge)
    gp, gr, g = v(col.dp * fd), v(col.drho * fd), v(col.g * fd)
    rho0, c2r, k = v(col.rho), v(col.c ** 2 * col.rho), RSUN / xl
    dep = np.exp(-1e7 * 4.0 * (col.z - col.z[col.e]) ** 2)
    dep[np.abs(np.arange(n) - col.e) > 4] = 0.0
    dep, pat = v(dep), t64(pats)[None]
    inside = torch.ones((n, 1, 1), dtype=F64, device=DEV)
    inside[0], inside[n - 1] = 0.0, 0.0
    dx, dz = lambda f: d_spectral(f, 2, k), lambda f: zdot(col.D[1], f, 0)  # noqa: E731
    if opt == 12:
        bx0, bz0 = t64(box)[:, None], t64(boz)[:, None]
        curl = dz(bx0) - dx(bz0)
    smooth = torch.zeros((n, 1, 1), dtype=F64, device=DEV)
    smooth[1:10], smooth[n - 10:n - 1] = 1.0, 1.0
    fcols = torch.zeros(nx, dtype=F64, device=DEV)
    fcols[8:nx - 8] = 1.0
    F = t64(filter_matrix(n, 5, n - 1, True))
    zero = torch.zeros((n, nb, nx), dtype=F64, device=DEV)

    def rhs(X, P, source):
        dvz, gz = dz(X[3]), dz(X[4])
        derivs = [gz, dvz]
        if opt == 12:
            flux = -(X[1] * bz0 - X[3] * bx0)
            derivs += [dz(flux), dz(X[5])]
        RP = [(az * q + bz * p) * layer for q, p in zip(derivs, P)]
        derivs = [q + p for q, p in zip(derivs, P)]
        gz, dvz = derivs[:2]
        if opt == 12:
            dvz = torch.where(smooth > 0, 0.5 * (dvz.roll(1, 0) + dvz.roll(-1, 0)), dvz)
        div = dx(X[1]) + dvz
        rc, rp = -gr * X[3] - rho0 * div, -c2r * div - X[3] * gp
        rx, rz = -dx(X[4]) / rho0, -(gz + X[0] * g) / rho0 + source
        if opt == 5:
            return [rc - sponge * X[0], (rx - sponge * X[1]) * inside, zero, (rz - sponge * X[3]) * inside,
                    (rp - sponge * X[4]) * inside], RP
        R = [rc * inside, rx * inside, zero, rz * inside, rp * inside]
        if opt == 12:
            cur = derivs[3] - dx(X[7])
            R[1] = R[1] + inside * (bz0 * cur + X[7] * curl) / rho0
            R[3] = R[3] - inside * (bx0 * cur + X[5] * curl) / rho0
            R += [-derivs[2] * inside, zero, dx(flux) * inside]
        return R, RP

    a = [zero.clone() for _ in range(8 if opt == 12 else 5)]
    P = [zero.clone() for _ in range(4 if opt == 12 else 2)]
    seis = []
    for step in range(c["steps"]):
        X, Y = a, P
        for s, b in enumerate(betas(col.dt)):
            if s:
                X, Y = [u + b * r for u, r in zip(a, R)], [u + b * r for u, r in zip(P, RP)]
            R, RP = rhs(X, Y, pat * float(amp[step]) * dep)
        a = [u + col.dt * r for u, r in zip(a, R)]
        a = [u + (zdot(F, u, 0) - u) * fcols for u in a]
        P = [u + col.dt * r for u, r in zip(P, RP)]
        if step % 5 == 0:
            seis.append(a[3][col.o])
    return {"seis": torch.stack(seis), "state": torch.stack(a)}


# Ridges of the f and p modes in k, f: lower and upper edge (quadratics in k; p2's lower one is
# 4.1004 sqrt(k)), the lowest frequency (driver.f90:1148-1718) and the mode's speed (1936-1944)
RIDGES = (((0.7, 1.7, -0.2), (1.1, 1.9, -0.2), 1.1, 0.44), ((1.1, 2.4, -0.3), (1.4, 3.0, -0.5), 1.6, 0.60),
          (None, (1.6, 3.8, -0.65), 1.6, 0.75), ((2.0, 3.55, -0.7), (2.0, 4.1, -0.8), 1.6, 0.9),
          ((2.15, 4.0, -0.7), (2.3, 4.4, -0.7), 1.6, 1.2), ((2.2, 4.7, -1.0), (2.35, 5.6, -1.1), 1.6, 1.4),
          ((1.80035417224, 7.42939105658, -2.84595764385), (1.98567115899, 8.09108986838, -3.20316331815), 1.6, 1.7),
          ((1.98297334673, 7.94931076885, -3.00725356897), (2.18544600032, 8.68183289647, -3.84478880142), 1.6, 1.9))
BOUNCE = ((-0.000417147774671, 0.313350998096, 17.9609631186), (-0.00028361249034, 0.29270337114, 36.4398734578))


def ridge(p, nx, nt):
    """Mask (nt, nx) of mode p (8: all p modes) times the 1.5 to 6 mHz band."""
    k = 2 * PI * np.abs(np.fft.fftfreq(nx, 1.0 / nx)) / (nx * CELL_MM * MM * f32(1e-8) * nx / (nx - 1.0))
    f = (np.abs(np.fft.fftfreq(nt, 1.0 / nt)) * 1e3 / (nt * 30.0))[:, None]
    poly = lambda q: f32(q[0]) + f32(q[1]) * k + f32(q[2]) * k ** 2  # noqa: E731
    if p == 8:
        m, low = np.ones((nt, nx)), f32(1.6)
    else:
        lo, hi, low, _ = RIDGES[p]
        low = f32(low)
        f0 = f32(4.1004) * np.sqrt(k) if lo is None else poly(lo)
        width = poly(hi) - f0
        with np.errstate(invalid="ignore", divide="ignore"):
            m = np.where((f - f0 < width) & (f > f0), 0.5 * (1 + np.cos(2 * PI * (f - f0 - width / 2) / width)), 0.0)
    taper = np.where(f < low + 0.5, 0.5 * (1 + np.cos(PI * (f - low - 0.5) / 0.5)), 1.0)
    wid = f32(0.4) * f[1]
    band = 1 / (1 + np.exp((1.5 - f) / wid)) - 1 / (1 + np.exp((6.0 - f) / wid))
    # modes without a band of their own get the last one read again (f, p1, p2)
    return np.where(f < low, 0.0, m * taper) * (band * band if p < 3 else band)


def exact_traveltime(c, seed):
    synth, data, x0s, t, modes, kern, hess = inputs_traveltime(c, seed)
    nb, nt, nx, dt = c["nb"], c["nt"], c["nx"], 0.5
    S, D = np.fft.fft2(synth.cpu().numpy()), np.fft.fft2(data.cpu().numpy())
    q = np.fft.fftfreq(nt, 1.0 / nt)
    if nt % 2 == 0:
        q[nt // 2] = nt / 2  # the middle frequency counts as positive
    om = 2 * PI * q / (nt * dt * 60.0)
    gb = 2j * PI * np.where(np.abs(q) < nt // 2, q, 0.0) / (nt * dt)
    simpson = np.where(np.arange(1, nt + 1) % 2 == 0, 4.0, 2.0)
    simpson[[0, nt - 1]] = 1.0
    dist = np.abs(((np.arange(nx) / nx - 0.5) * nx * CELL_MM * MM * f32(1e-8))[None, :] - np.array(x0s)[:, None])
    adj, misfit = np.zeros((nb, nt, nx)), np.zeros(nb)
    for p in range(9):
        m, (near, far, win) = ridge(p, nx, nt), modes[p]
        half = int(math.floor(win / (2 * dt) + 0.5))
        acc, dat = np.fft.ifft2(S * m) * (nx * nt), np.fft.ifft2(D * m) * (nx * nt)
        ccd = np.fft.ifft2(S * m * 1j * om[:, None]) * (nx * nt)
        u0d = np.fft.ifft(np.fft.fft(acc.real, axis=1) * gb[:, None], axis=1).real
        point = np.zeros((nb, nt, nx), dtype=complex)
        for b in range(nb):
            for i in np.flatnonzero((dist[b] > near) & (dist[b] < far)):
                if p < 8:
                    ts = math.floor(dist[b, i] / f32(RIDGES[p][3]) / dt)
                    tf = ts + 40
                else:
                    ts, tf = (math.floor((f32(w[0]) * dist[b, i] ** 2 + f32(w[1]) * dist[b, i] + f32(w[2])) / dt) for w in BOUNCE)
                lo, hi = max(ts, 1), min(tf, nt)
                if lo > hi:
                    continue
                loc = lo + int(np.argmax(np.abs(acc[b, lo - 1:hi, i].real)))
                left, right = max(loc - half, 1), min(loc + half, nt)
                w = slice(left - 1, right)
                u, r = u0d[b, w, i], acc[b, w, i].real - dat[b, w, i].real
                tau = np.sum(simpson[w] * u * r) / np.sum(simpson[w] * u * u)
                point[b, w, i] = (-tau / (np.sum(ccd[b, w, i] ** 2) * dt)).real * ccd[b, w, i]
                misfit[b] += tau ** 2
        adj += (np.fft.ifft2(np.fft.fft2(point) * m) * (nx * nt)).real[:, ::-1]
    # grad.py: kernel and hessian sums, preconditioner, filters, antisymmetry, direction, trial models
    rho = t64(M.polytrope(c["nz"])[:, 2])[:, None]
    h = hess.abs().sum(0) * rho
    h = (h / h.abs().max()).clamp_min(5e-3)
    kx = torch.arange(nx // 2 + 1, dtype=F64, device=DEV)
    g = torch.fft.irfft(torch.fft.rfft(kern.sum(0) / h, dim=1) * torch.exp(-kx ** 2 / 1800.0), n=nx, dim=1)
    g = 0.5 * (g - g.flip(1))
    taps = torch.exp(-0.125 * torch.arange(-8, 9, dtype=F64, device=DEV) ** 2)
    padded = torch.cat((g[:8].flip(0), g, g[-8:].flip(0)))
    g = sum(w * padded[j:j + c["nz"]] for j, w in enumerate(taps / taps.sum()))
    beta = (g * (g - kern[0])).sum() / (kern[0] ** 2).sum()
    u = -g + beta * hess[0]
    rms = (g ** 2).mean().sqrt()
    return {"adjoint": adj * nt / 60.0, "misfit": 0.5 * misfit, "measured": None, "windows": None, "gradient": g,
            "update": u, "beta": float(beta), "trial": torch.stack([g + e * u / u.max() * rms for e in (0.01, 0.02, 0.03)])}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("forward", "kernels"):
        run, model, xs, psi, cmul = inputs_2d(c, seed)
        sim = Exact2D(c, model, psi, cmul)
        if kind == "forward":
            seis, state, _ = sim.forward(xs, c["steps"])
            return {"seis": seis, "state": state}
        seis, out = sim.kernels(xs, c["steps"], torch.as_tensor(receivers(c["nx"]), device=DEV))
        return {"seis": seis, "kernels": list(out.unbind(1))}
    if kind in ("forward3d", "kernels3d"):
        model, xl, pats, amp, flow = inputs_3d(c, seed)
        sim = Exact3D(c, model, xl, flow)
        if kind == "forward3d":
            seis, state, _ = sim.forward(pats, amp, c["steps"], 2)
            return {"seis": seis, "state": state}
        seis, out = sim.kernels(pats, amp, c["steps"], 5)
        return {"seis": seis, "kernels": list(out.unbind(0))}
    if kind == "velocity":
        return exact_velocity(c, seed)
    return exact_gradient(c, seed) if kind == "gradient" else exact_traveltime(c, seed)
