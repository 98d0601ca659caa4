"""Workloads of the solver, as a program that uses it runs them.

Each case is one call (or one short chain of calls) of the public Python
interface with the sizes of this repository's configurations, tests and
benchmark. The kinds:

  krylov  B200IterativeSolver.solve on a built operator with an iteration cap:
          a fixed number of restart cycles of the restarted or recycled GMRES,
          the work of every solve (a capped solve is also what the batch tuner
          times). Forward and adjoint, all three vector precisions.
  field   HelmholtzB200Solver: right-hand side of the current phases and the
          converged field (air scene).
  scenes  solve_scenes_batched: several scenes of different sizes in one call.
  apply   DeviceOperator.apply: one matrix-free operator application.
  setup   building a scene: operator records, aperture columns, right-hand
          sides.
  basis   one phase-optimisation step on a response basis: field, focal
          contrast loss with its cotangent, phase gradient.
  adjoint one gradient step of the differentiable path: field, loss, A^H
          solve, phase gradient, material gradient.
"""
from __future__ import annotations

import math

import numpy as np
import torch

FACES = ("-x", "+x", "-y", "+y", "-z", "+z")
F0 = 40000.0
OMEGA = 2 * math.pi * F0
C0, RHO0 = 343.0, 1.2
H = 1.0e-3
PML = {"cells": 10, "strength": 2.0, "order": 2}
# the boundary sets of the configurations: open box over a reflecting baffle,
# the same with one reflecting side, and one with an impedance wall as well
BOUNDARIES = {
    "open": {"-x": "open", "+x": "open", "-y": "open", "+y": "open", "-z": "reflecting",
             "+z": "open"},
    "wall": {"-x": "open", "+x": "reflecting", "-y": "open", "+y": "open", "-z": "reflecting",
             "+z": "open"},
    "impedance": {"-x": "open", "+x": "reflecting",
                  "-y": {"type": "impedance", "impedance": [2 * RHO0 * C0, 0.0]}, "+y": "open",
                  "-z": "reflecting", "+z": "open"},
}
DEV = "cuda"


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the benchmark's solver setting and scene: bfloat16 GCRO-DR(32,8),
        # batch of four right-hand sides at 128^3
        dict(name="recycled_bf16_128_b4", kind="krylov", nx=128, ny=128, nz=128, nrhs=4,
             precision="bf16", restart=32, recycle=8, iters=184, adjoint=False, faces="wall"),
        # the default setting (complex64 GMRES(30), one right-hand side), adjoint
        dict(name="restarted_c64_128_adjoint", kind="krylov", nx=128, ny=128, nz=128, nrhs=1,
             precision="mixed", restart=30, recycle=0, iters=90, adjoint=True, faces="wall"),
        # full precision, uneven odd grid, two right-hand sides, impedance wall
        dict(name="restarted_fp64_97x90x83_b2", kind="krylov", nx=97, ny=90, nz=83, nrhs=2,
             precision="fp64", restart=30, recycle=0, iters=60, adjoint=False,
             faces="impedance"),
        # a small odd grid of the size of the tests, three right-hand sides:
        # launches and latency count
        dict(name="recycled_bf16_41x37x33_b3", kind="krylov", nx=41, ny=37, nz=33, nrhs=3,
             precision="bf16", restart=32, recycle=8, iters=400, adjoint=False, faces="wall"),
        # the 64^3 air scene, solved to 1e-10 with the default GMRES(30)
        dict(name="field_64_air", kind="field", n=64, array=4, rtol=1e-10),
        # uneven scene batch (edges of the scene-batch configuration)
        dict(name="scenes_48_to_80", kind="scenes", edges="48,80,64,48,64,80", restart=36,
             recycle=8, iters=100),
        # the operator alone: the benchmark's stencil entry, and a small
        # ragged complex128 adjoint product
        dict(name="apply_k_c64_128_b4", kind="apply", variant="K", nx=128, ny=128, nz=128, nrhs=4,
             faces="wall"),
        dict(name="apply_ah_fp64_65x50x37", kind="apply", variant="AH", nx=65, ny=50, nz=37,
             nrhs=1, faces="impedance"),
        # scene set-up of the response-basis configuration: 96^3, 16 x 16 array
        dict(name="setup_96_array16", kind="setup", n=96, array=16, columns=8),
        # response basis of that scene (256 columns): complex128 as stored, and
        # a small complex64 one
        dict(name="basis_c128_96_m256", kind="basis", nx=96, ny=96, nz=96, emitters=256,
             precision="complex128"),
        dict(name="basis_c64_45x40x35_m64", kind="basis", nx=45, ny=40, nz=35, emitters=64,
             precision="complex64"),
        # gradient of a focal loss through forward and adjoint solves
        dict(name="adjoint_step_48", kind="adjoint", n=48, array=4, rtol=1e-7),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["krylov", "krylov", "krylov", "krylov", "scenes", "apply", "apply", "setup",
                       "basis", "basis", "field", "adjoint"])
    if kind == "krylov":
        nx, ny, nz = (_log_int(rng, 24, 128) for _ in range(3))
        precision = rng.choice(["bf16", "bf16", "mixed", "fp64"])
        restart = rng.randint(16, 40)
        recycle = rng.choice([0, 4, 8, rng.randint(2, 10)])
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, nrhs=rng.randint(1, 4), precision=precision,
                    restart=restart, recycle=recycle, iters=3 * restart,
                    adjoint=rng.random() < 0.4, faces=rng.choice(sorted(BOUNDARIES)))
    if kind == "scenes":
        edges = [rng.randint(32, 80) for _ in range(rng.randint(2, 6))]
        return dict(kind=kind, edges=",".join(map(str, edges)), restart=rng.randint(20, 36),
                    recycle=rng.choice([0, 8]), iters=72)
    if kind == "apply":
        nx, ny, nz = (_log_int(rng, 16, 128) for _ in range(3))
        return dict(kind=kind, variant=rng.choice(["K", "KH", "A", "AH", "K64"]), nx=nx, ny=ny,
                    nz=nz, nrhs=rng.randint(1, 4), faces=rng.choice(sorted(BOUNDARIES)))
    if kind == "setup":
        return dict(kind=kind, n=_log_int(rng, 40, 96), array=rng.randint(2, 6),
                    columns=rng.randint(1, 8))
    if kind == "basis":
        nx, ny, nz = (_log_int(rng, 24, 96) for _ in range(3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, emitters=_log_int(rng, 4, 256),
                    precision=rng.choice(["complex64", "complex128"]))
    if kind == "field":
        return dict(kind=kind, n=rng.randint(40, 64), array=rng.randint(1, 3), rtol=1e-10)
    return dict(kind="adjoint", n=rng.randint(40, 52), array=rng.randint(1, 4), rtol=1e-7)


# ------------------------------------------------------------------ inputs
def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(1000003 * (seed + 1) + salt)


def _smooth_field(shape, gen, sigma=4.0):
    """Gaussian random field (unit variance, clipped at 3), correlation ~sigma nodes; Fortran order."""
    g = torch.randn(shape[::-1], dtype=torch.float64, device=DEV, generator=gen)
    f = torch.fft.rfftn(g)
    k2 = sum(k * k for k in torch.meshgrid(
        *[2 * math.pi * torch.fft.fftfreq(n, device=DEV, dtype=torch.float64) for n in shape[:0:-1]],
        2 * math.pi * torch.fft.rfftfreq(shape[0], device=DEV, dtype=torch.float64), indexing="ij"))
    g = torch.fft.irfftn(f * torch.exp(-0.5 * sigma * sigma * k2), s=shape[::-1])
    g = (g - g.mean()) / g.std()
    return g.clamp(-3, 3).reshape(-1)


def _medium(shape, seed):
    """rho, c of a random medium with a smoothed sphere in its middle (Fortran-order vectors)."""
    gen = _gen(seed)
    c = C0 * (1 + 0.05 * _smooth_field(shape, gen))
    rho = RHO0 * (1 + 0.1 * _smooth_field(shape, gen))
    x, y, z = (torch.arange(n, dtype=torch.float64, device=DEV) * H for n in shape)
    ctr = [(n - 1) * H / 2 for n in shape]
    d = torch.sqrt((x[None, None, :] - ctr[0]) ** 2 + (y[None, :, None] - ctr[1]) ** 2
                   + (z[:, None, None] - ctr[2]) ** 2).reshape(-1) - 0.12 * (min(shape) - 1) * H
    t = (d / (1.2 * H)).clamp(-1, 1)
    step = 0.5 * (1 + t + torch.sin(math.pi * t) / math.pi)
    inv_rho = 1 / 1250.0 + (1 / rho - 1 / 1250.0) * step
    comp_o = 1 / (1250.0 * 2200.0 ** 2)
    comp = comp_o + (1 / (rho * c * c) - comp_o) * step
    return 1 / inv_rho, torch.sqrt(inv_rho / comp)


def _pml(shape):
    return dict(PML, cells=min(10, min(shape) // 4))


def _aperture_rhs(shape, nrhs, seed):
    """Right-hand sides of a baffled array: phased discs on the z = 0 plane."""
    gen = _gen(seed, 7)
    nx, ny, nz = shape
    cells = _pml(shape)["cells"]
    rhs = torch.zeros((nrhs, nz, ny, nx), dtype=torch.complex128, device=DEV)
    x = torch.arange(nx, device=DEV)[None, :]
    y = torch.arange(ny, device=DEV)[:, None]
    pitch = 6
    for cx in range(cells + 3, nx - cells - 3, pitch):
        for cy in range(cells + 3, ny - cells - 3, pitch):
            ph = 2 * math.pi * torch.rand(nrhs, dtype=torch.float64, device=DEV, generator=gen)
            disc = (((x - cx) ** 2 + (y - cy) ** 2) <= 6).to(torch.float64)
            rhs[:, 0] += torch.exp(1j * ph)[:, None, None] * disc
    return (-2 * math.pi / (RHO0 * H ** 3) * 1e-3) * rhs.reshape(nrhs, -1)


def _scene_dict(n, array, faces, solver, obstacle=None, target=None):
    from ultrasound_solver_b200.workloads import fit_array, scene_dict
    pitch, diameter = fit_array(array, n, H)
    c = (n - 1) * H / 2
    return scene_dict(n, H, array, pitch, diameter, boundaries=BOUNDARIES[faces],
                      obstacle=obstacle, targets=[(c, c, 0.6 * (n - 1) * H)] if target else (),
                      solver=solver)


def _solver(cfg):
    from ultrasound_solver_b200.config import SimulationConfig
    from ultrasound_solver_b200.helmholtz_solver import HelmholtzB200Solver
    return HelmholtzB200Solver(SimulationConfig.from_dict(cfg))


def _phases(count, seed):
    return np.random.default_rng(seed + 17).uniform(0, 2 * np.pi, count)


def _grid(case):
    return case["nx"], case["ny"], case["nz"]


def _operator(shape, faces, rho, c):
    from ultrasound_solver_b200.scene import DeviceOperator
    return DeviceOperator(shape, H, OMEGA, BOUNDARIES[faces], rho, c, pml=_pml(shape))


def _edges(case):
    return [int(v) for v in case["edges"].split(",")]


def _scene_sphere(n):
    return {"type": "sphere", "center": [(n - 1) * H / 2] * 3, "radius": 0.12 * (n - 1) * H,
            "smoothing_width_cells": 1.2, "material": {"density": 1250.0, "sound_speed": 2200.0}}


def _random_vectors(nrhs, n, dtype, seed):
    return torch.randn((nrhs, n), dtype=dtype, device=DEV, generator=_gen(seed, 11))


def _loss_config(shape):
    from ultrasound_solver_b200.config import SimulationConfig
    box = [(n - 1) * H for n in shape]
    return SimulationConfig.from_dict({
        "mode": "phase_optimization", "physics": {"sound_speed": C0, "medium_density": RHO0},
        "transducer_specs": {"frequency": F0, "array_n": 1, "diameter": 4e-3, "pitch": 4e-3,
                             "geometry": "ideal_grid"},
        "domain": {"box_size": box, "grid_size": list(shape)},
        "boundary_conditions": BOUNDARIES["open"],
        "targets": [{"point": [0.4 * box[0], 0.5 * box[1], 0.6 * box[2]]},
                    {"point": [0.6 * box[0], 0.5 * box[1], 0.6 * box[2]]}],
        "training": {"target_radius": 0.006, "source_exclusion_layers": 4}})


def _basis_columns(case, seed):
    """Response columns: spherical waves of a transducer plane below the grid, (M, N)."""
    nx, ny, nz = _grid(case)
    m = case["emitters"]
    dtype = torch.complex64 if case["precision"] == "complex64" else torch.complex128
    gen = _gen(seed, 3)
    cx = torch.rand(m, dtype=torch.float64, device=DEV, generator=gen) * (nx - 1)
    cy = torch.rand(m, dtype=torch.float64, device=DEV, generator=gen) * (ny - 1)
    x = torch.arange(nx, dtype=torch.float64, device=DEV)[None, None, :]
    y = torch.arange(ny, dtype=torch.float64, device=DEV)[None, :, None]
    z = torch.arange(nz, dtype=torch.float64, device=DEV)[:, None, None]
    out = torch.empty((m, nx * ny * nz), dtype=dtype, device=DEV)
    k = OMEGA / C0 * H
    for i in range(m):
        r = torch.sqrt((x - cx[i]) ** 2 + (y - cy[i]) ** 2 + (z + 4.0) ** 2).reshape(-1)
        out[i] = torch.polar(4.0 / r, k * r).to(dtype)
    return out


class _BasisScene:
    """What a response basis needs of its solver to answer device queries."""

    def __init__(self, shape, emitters):
        self.shape = shape
        self.total_dofs = int(np.prod(shape))
        self.device = torch.device("cuda", torch.cuda.current_device())
        self.transducers = type("T", (), {"num_transducers": emitters})()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "krylov":
        from ultrasound_solver_b200.iterative_solver import B200IterativeSolver
        shape = _grid(case)
        rho, c = _medium(shape, seed)
        it = B200IterativeSolver(restart=case["restart"], maxiter=case["iters"], rtol=1e-9,
                                 precision=case["precision"], recycle=case["recycle"])
        return dict(case=case, op=_operator(shape, case["faces"], rho, c), it=it,
                    rhs=_aperture_rhs(shape, case["nrhs"], seed))
    if kind == "field":
        s = _solver(_scene_dict(case["n"], case["array"], "open",
                                {"gmres_restart": 30, "gmres_rtol": case["rtol"],
                                 "gmres_maxiter": 20000}))
        s.set_phases(_phases(s.transducers.num_transducers, seed))
        s.assemble_matrix()
        return dict(case=case, solver=s)
    if kind == "scenes":
        settings = {"gmres_restart": case["restart"], "gmres_maxiter": case["iters"],
                    "gmres_rtol": 1e-9, "precision": "bf16", "gmres_recycle": case["recycle"],
                    "gmres_recycle_every": 2}
        solvers, rhs = [], []
        for i, n in enumerate(_edges(case)):
            s = _solver(_scene_dict(n, 2, "wall", settings, obstacle=_scene_sphere(n)))
            s.assemble_matrix()
            solvers.append(s)
            rhs.append(_aperture_rhs((n, n, n), 1, seed + 31 * i)[0])
        return dict(case=case, solvers=solvers, rhs=rhs)
    if kind == "apply":
        shape = _grid(case)
        rho, c = _medium(shape, seed)
        single = case["variant"] in ("K", "KH")
        x = _random_vectors(case["nrhs"], int(np.prod(shape)),
                            torch.complex64 if single else torch.complex128, seed)
        return dict(case=case, op=_operator(shape, case["faces"], rho, c), x=x)
    if kind == "setup":
        from ultrasound_solver_b200.workloads import fit_array
        n, m = case["n"], case["array"]
        rho, c = _medium((n, n, n), seed)
        pitch, diameter = fit_array(m, n, H)
        axis = (n - 1) * H / 2 + (np.arange(m) - (m - 1) / 2) * pitch
        centers = np.zeros((m * m, 3))
        centers[:, 0], centers[:, 1] = np.repeat(axis, m), np.tile(axis, m)
        w = np.random.default_rng(seed).standard_normal((case["columns"], m * m, 2))
        coeff = torch.from_numpy(w[..., 0] + 1j * w[..., 1]).to(DEV)
        return dict(case=case, rho=rho, c=c, centers=centers, diameter=diameter, coeff=coeff)
    if kind == "basis":
        from ultrasound_solver_b200.losses import FocalContrastLoss
        from ultrasound_solver_b200.phase_response_basis import PhaseResponseBasis
        shape = _grid(case)
        basis = PhaseResponseBasis(_BasisScene(shape, case["emitters"]), "basis.npy",
                                   device_precision=case["precision"])
        basis.basis_gpu = _basis_columns(case, seed)
        loss = FocalContrastLoss(_loss_config(shape))
        return dict(case=case, basis=basis, loss=loss,
                    phases=torch.from_numpy(_phases(case["emitters"], seed)).to(DEV))
    # adjoint
    from ultrasound_solver_b200.losses import FocalContrastLoss
    n = case["n"]
    s = _solver(_scene_dict(n, case["array"], "wall",
                            {"gmres_restart": 30, "gmres_rtol": case["rtol"],
                             "gmres_maxiter": 20000, "gmres_backward_error_tol": 1.0,
                             "precision": "mixed"}, target=True))
    rho, c = (v.cpu().numpy().reshape((n, n, n), order="F") for v in _medium((n, n, n), seed))
    s.set_material_fields(rho, c)
    ph = _phases(s.transducers.num_transducers, seed)
    s.set_phases(ph)
    s.assemble_matrix()
    return dict(case=case, solver=s, loss=FocalContrastLoss(s.cfg), phases=torch.from_numpy(ph))


# ------------------------------------------------------------------ one pass
def run(state):
    from ultrasound_solver_b200 import _native as N
    case = state["case"]
    kind = case["kind"]
    if kind == "krylov":
        return state["it"].solve(state["op"], state["rhs"], adjoint=case["adjoint"],
                                 raise_on_failure=False)
    if kind == "field":
        s = state["solver"]
        return s.solve_rhs_device(s.update_rhs_device())
    if kind == "scenes":
        from ultrasound_solver_b200.scene_batch import solve_scenes_batched
        return solve_scenes_batched(state["solvers"], state["rhs"], raise_on_failure=False)
    if kind == "apply":
        variant, precision = {"K": (N.APPLY_K, N.PREC_MIXED), "KH": (N.APPLY_KH, N.PREC_MIXED),
                              "A": (N.APPLY_A, N.PREC_FP64), "AH": (N.APPLY_AH, N.PREC_FP64),
                              "K64": (N.APPLY_K, N.PREC_FP64)}[case["variant"]]
        return state["op"].apply(state["x"], variant, precision)
    if kind == "setup":
        from ultrasound_solver_b200.scene import SourceColumns
        n = case["n"]
        op = _operator((n, n, n), "wall", state["rho"], state["c"])
        src = SourceColumns(op, state["centers"], state["diameter"], RHO0)
        return [*op.export(), src.mass_matrix, src.rhs(state["coeff"])]
    if kind == "basis":
        u = state["basis"].field_device(state["phases"])
        value, cot = state["loss"].evaluate_vector(u)
        return [u, value, cot, state["basis"].phase_vjp_device(cot, state["phases"])]
    from ultrasound_solver_b200.autograd import loss_of_field, phase_field
    s = state["solver"]
    ph = state["phases"].clone().requires_grad_(True)
    u = phase_field(ph, s)
    value = loss_of_field(u, state["loss"])
    u.retain_grad()
    value.backward()
    lam = s.solve_rhs_device(u.grad, adjoint=True)
    return [u.detach(), value.detach(), ph.grad, *s.material_vjp_device(u.detach(), lam)]


# ------------------------------------------------------------------ work
_VECTOR = {"bf16": 4, "mixed": 8, "fp64": 16}
_ROWS = {"bf16": 24, "mixed": 48, "fp64": 48}  # six row coefficients at the path's precision


def _krylov_work(n, nrhs, precision, restart, recycle, iters):
    """Arnoldi steps of `iters` iterations: each reads its basis twice (the
    update needs every inner product of the step first), reads and writes one
    new vector, and reads the row coefficients once per batch; each cycle
    updates the double-precision solution and residual."""
    vb = _VECTOR[precision]
    by = fl = 0.0
    done, cycle = 0, 0
    while done < iters:
        kc = recycle if cycle >= 2 else 0
        for j in range(kc, restart):
            by += nrhs * vb * (2 * (j + 1) + 2) + _ROWS[precision]
            fl += nrhs * (16 * (j + 1) + 56)
        by += nrhs * (vb * (restart + 1) + 5 * 16) + 7 * 16 + 32
        fl += nrhs * (8 * restart + 64)
        if recycle and cycle >= 2:
            by += nrhs * vb * (restart + 1 + 3 * recycle + restart + 1 + recycle + 2 * recycle + 3)
            fl += nrhs * 8 * recycle * (3 * restart + 2)
        done += restart - kc
        cycle += 1
    return by * n, fl * n


def work(case):
    kind = case["kind"]
    if kind == "krylov":
        by, fl = _krylov_work(int(np.prod(_grid(case))), case["nrhs"], case["precision"],
                              case["restart"], case["recycle"], case["iters"])
    elif kind == "field":
        # about 68 n iterations of GMRES(30) to 1e-10 in the open air scene
        by, fl = _krylov_work(case["n"] ** 3, 1, "mixed", 30, 0, 68 * case["n"])
    elif kind == "scenes":
        parts = [_krylov_work(n ** 3, 1, "bf16", case["restart"], case["recycle"], case["iters"])
                 for n in _edges(case)]
        by, fl = (sum(p[i] for p in parts) for i in (0, 1))
    elif kind == "apply":
        n, b = int(np.prod(_grid(case))), case["nrhs"]
        single = case["variant"] in ("K", "KH")
        # node record {rho, R, s} and the vectors
        by = n * ((16 if single else 32) + b * (16 if single else 32))
        fl = n * b * 56
    elif kind == "setup":
        n, m = case["n"] ** 3, case["array"] ** 2
        by = n * (16 + 2 * 16 + 3 * 16) + case["n"] ** 2 * 8 * m + 16 * n * case["columns"]
        fl = n * 300 + m * 64 * 256 * 4 * 6
    elif kind == "basis":
        n, m = int(np.prod(_grid(case))), case["emitters"]
        vb = 8 if case["precision"] == "complex64" else 16
        by = 2 * n * m * vb + n * (16 + 1 + 16)
        fl = 16 * n * m
    else:
        by, fl = _krylov_work(case["n"] ** 3, 1, "mixed", 30, 0, 3 * 50 * case["n"])
    return {"bytes": float(by), "flops": float(fl)}


# ------------------------------------------------------------------ tolerance
def tolerance(case):
    kind = case["kind"]
    if kind == "krylov":
        # measured with other summation orders: up to 7e-3, 1.3e-8 and 8e-16
        return {"rel": {"bf16": 3e-2, "mixed": 1e-6, "fp64": 1e-12}[case["precision"]]}
    if kind == "field":
        return {"rel": 1e-9}
    if kind == "scenes":
        return {"rel": 3e-2}
    if kind == "apply":
        return {"rel": 3e-7 if case["variant"] in ("K", "KH") else 1e-15}
    if kind == "setup":
        return {"rel": 1e-15}
    if kind == "basis":
        return {"rel": 1e-13}
    # a solve stopped at 1e-7 is this far from the exact gradients (measured:
    # 2e-5 between summation orders, 2e-3 against the exact ones)
    return {"rel": 2e-3}


# ------------------------------------------------------------------ 64-bit restatement
def _axis(n, cells_lo, cells_hi, strength, order):
    d = torch.arange(n, dtype=torch.float64, device=DEV)
    sigma = torch.zeros(n, dtype=torch.float64, device=DEV)
    if cells_lo:
        sigma += strength * (1 - d / cells_lo).clamp(min=0) ** order
    if cells_hi:
        sigma += strength * (1 - d.flip(0) / cells_hi).clamp(min=0) ** order
    w = torch.ones(n, dtype=torch.float64, device=DEV)
    w[0] = w[-1] = 0.5
    s = torch.complex(torch.ones_like(sigma), sigma)
    return w * s, 1 / (0.5 * (s[:-1] + s[1:]) * H * H)


class _Matrix:
    """The finite-volume operator A on the (z, y, x) grid in complex128: the
    edge coefficients per axis, the diagonal, the row scale and Jacobi factor."""

    def __init__(self, shape, faces, rho, c, pml):
        nx, ny, nz = shape
        bc = BOUNDARIES[faces]
        kind = [v["type"] if isinstance(v, dict) else v for v in (bc[f] for f in FACES)]
        cells = [pml["cells"] if k == "open" else 0 for k in kind]
        (tx, qx), (ty, qy), (tz, qz) = (
            _axis(n, cells[2 * a], cells[2 * a + 1], pml["strength"], pml["order"])
            for a, n in enumerate(shape))
        T = {0: tz[:, None, None], 1: ty[None, :, None], 2: tx[None, None, :]}
        Q = {0: qz[:, None, None], 1: qy[None, :, None], 2: qx[None, None, :]}
        self.shape = (nz, ny, nx)
        self.rho, self.c = rho.view(self.shape), c.view(self.shape)
        self.T, self.kind = T, kind
        diag = T[0] * T[1] * T[2] * (OMEGA ** 2 / (self.rho * self.c ** 2))
        self.edge, self.geom = {}, {}
        big = torch.zeros(self.shape, dtype=torch.float64, device=DEV)
        for ax in range(3):
            n = self.shape[ax]
            others = [T[a] for a in range(3) if a != ax]
            F = others[0] * others[1] * Q[ax]
            r0, r1 = self.rho.narrow(ax, 0, n - 1), self.rho.narrow(ax, 1, n - 1)
            e = F * (2 / (r0 + r1))
            self.geom[ax], self.edge[ax] = F, e
            diag.narrow(ax, 0, n - 1).sub_(e)
            diag.narrow(ax, 1, n - 1).sub_(e)
            for lo in (0, 1):
                v = big.narrow(ax, lo, n - 1)
                torch.maximum(v, e.abs(), out=v)
        self.face_terms = []
        for f in range(6):
            ax = 2 - f // 2
            if kind[f] not in ("open", "impedance"):
                continue
            pos = 0 if f % 2 == 0 else self.shape[ax] - 1
            others = [T[a] for a in range(3) if a != ax]
            area = (others[0] * others[1] / H).expand(
                [1 if a == ax else self.shape[a] for a in range(3)])
            if kind[f] == "open":
                adm = 1 / (self.rho * self.c).narrow(ax, pos, 1)
            else:
                adm = 1 / complex(*bc[FACES[f]]["impedance"])
            term = 1j * OMEGA * area * adm
            diag.narrow(ax, pos, 1).add_(term)
            if kind[f] == "open":
                self.face_terms.append((ax, pos, term))
        self.diag = diag
        self.R = 1 / torch.maximum(diag.abs(), big)
        self.s = 1 / (self.R * diag)

    def off(self, x, conj=False):
        x = x.view(self.shape)
        y = torch.zeros_like(x)
        for ax in range(3):
            n = self.shape[ax]
            e = self.edge[ax].conj() if conj else self.edge[ax]
            y.narrow(ax, 0, n - 1).add_(e * x.narrow(ax, 1, n - 1))
            y.narrow(ax, 1, n - 1).add_(e * x.narrow(ax, 0, n - 1))
        return y

    def A(self, x, conj=False):
        d = self.diag.conj() if conj else self.diag
        return (d * x.view(self.shape) + self.off(x, conj)).reshape(-1)

    def K(self, u, conj=False):
        s = self.s.conj() if conj else self.s
        y = u.view(self.shape) + self.R * self.off((s * u.view(self.shape)).reshape(-1), conj)
        return y.reshape(-1)


def _least_squares(G, rhs):
    return torch.linalg.lstsq(G, rhs[:, None]).solution[:, 0]


def _krylov(mat, b, m, maxiter, rtol, k=0, every=1, conj=False):
    """Restarted GMRES(m), or GCRO-DR(m, k) with the harmonic Ritz vectors of
    the cycle before the previous one, right-preconditioned by the Jacobi
    factor: iterations counted per cycle, tested at restarts."""
    R = mat.R.reshape(-1)
    s = (mat.s.conj() if conj else mat.s).reshape(-1)
    x = torch.zeros_like(b)
    bn = torch.linalg.norm(R * b)
    iters, cycle = 0, 0
    U = C = None
    ready = None
    V = torch.empty((m + 1, b.numel()), dtype=b.dtype, device=b.device)
    while True:
        r = R * (b - mat.A(x, conj)) if cycle else R * b
        if torch.linalg.norm(r) <= rtol * bn or iters >= maxiter:
            return x
        if ready is not None:
            U, C = ready
            ready = None
        kc = 0 if U is None else k
        V = torch.empty_like(V)
        alpha = None
        if kc:
            d = 1 / torch.linalg.norm(U, dim=1)
            alpha = C.conj() @ r
            r = r - alpha @ C
            V[:kc] = C
        beta = torch.linalg.norm(r)
        V[kc] = r / beta
        G = torch.zeros((m + 1, m), dtype=b.dtype, device=b.device)
        for t in range(kc):
            G[t, t] = d[t]
        for j in range(kc, m):
            w = mat.K(V[j], conj)
            h = V[:j + 1].conj() @ w
            w = w - h @ V[:j + 1]
            G[:j + 1, j] = h
            nb = torch.linalg.norm(w)
            G[j + 1, j] = nb
            V[j + 1] = w / nb
        rhs = torch.zeros(m + 1, dtype=b.dtype, device=b.device)
        rhs[kc] = beta
        y = _least_squares(G, rhs)
        W = torch.cat([U * d[:, None], V[kc:m]]) if kc else V[:m]
        corr = y @ W
        if kc:
            corr = corr + alpha @ U
        x = x + s * corr
        iters += m - kc
        # the pair for the cycle after the next one
        if k:
            if cycle > 0 and pending is not None:
                ready = pending
            pending = None
            if cycle % every == 0:
                P = _harmonic(G, V.conj() @ W.T, k)
                Qm, Rm = torch.linalg.qr(G @ P)
                pending = (torch.linalg.solve(Rm.T, P.T) @ W, Qm.T @ V)
        cycle += 1


def _harmonic(G, VW, k):
    lhs = (G.conj().T @ G).cpu()
    rhs = (G.conj().T @ VW).cpu()
    theta, Z = torch.linalg.eig(torch.linalg.solve(rhs, lhs))
    pick = torch.argsort(theta.abs())[:k]
    Z = Z[:, pick]
    return (Z / torch.linalg.norm(Z, dim=0)).to(G.device)


def _aperture_masses(n, centers, diameter, radial=64, angular=256):
    """Bilinear unit-mass deposition of disc quadrature points, (M, n*n)."""
    mu, w = np.polynomial.legendre.leggauss(radial)
    mu, w = (mu + 1) / 2, w / 2
    r = diameter / 2 * np.sqrt(1 - mu * mu)
    phi = 2 * np.pi * np.arange(angular) / angular
    px, py = (r[:, None] * np.cos(phi)).ravel(), (r[:, None] * np.sin(phi)).ravel()
    pw = np.repeat(w / angular, angular)
    out = np.zeros((len(centers), n * n))
    for row, (cx, cy, _) in zip(out, centers):
        gx, gy = (cx + px) / H, (cy + py) / H
        ix, iy = np.floor(gx).astype(int), np.floor(gy).astype(int)
        fx, fy = gx - ix, gy - iy
        for a in (0, 1):
            for b in (0, 1):
                np.add.at(row, (iy + b) * n + ix + a,
                          pw * (fx if a else 1 - fx) * (fy if b else 1 - fy))
    return out


def _source_rhs(n, masses, coeff):
    """-2 pi / (rho dx^3) sum_m masses_m coeff_m in the z = 0 plane, (K, N)."""
    out = torch.zeros((coeff.shape[0], n ** 3), dtype=torch.complex128, device=DEV)
    mt = torch.from_numpy(masses).to(DEV).to(torch.complex128)
    out[:, :n * n] = (-2 * math.pi / (RHO0 * H ** 3)) * (coeff @ mt)
    return out


def _array_centers(n, array, pitch):
    axis = (n - 1) * H / 2 + (np.arange(array) - (array - 1) / 2) * pitch
    centers = np.zeros((array * array, 3))
    centers[:, 0], centers[:, 1] = np.repeat(axis, array), np.tile(axis, array)
    return centers


def _contrast_loss(u, shape, box, targets, training):
    """Focal contrast: -w_t mean |u_t| + w_s soft maximum of |u| over the background."""
    xs, ys, zs = (torch.from_numpy(np.linspace(0.0, b, n)).to(DEV) for b, n in zip(box, shape))
    mask = torch.ones(shape[::-1], dtype=torch.bool, device=DEV)
    mask[:max(int(training.source_exclusion_layers), 0)] = False
    for p in targets:
        dx, dy, dz = ((v - float(q)) ** 2 for v, q in zip((xs, ys, zs), p))
        r2 = dx[None, None, :] + dy[None, :, None] + dz[:, None, None]
        mask &= r2 > training.target_radius * training.target_radius
    mask = mask.reshape(-1)
    T, wt, ws = training.sidelobe_temperature, training.target_weight, training.background_weight
    amp = u.abs()
    idx = [int(i + shape[0] * (j + shape[1] * k)) for i, j, k in
           (np.rint(np.asarray(p) / H).astype(int) for p in targets)]
    lse = torch.logsumexp(amp[mask] / T, 0)
    value = -wt * amp[idx].mean() + ws * T * (lse - math.log(int(mask.sum())))
    cot = torch.zeros_like(u)
    p = torch.where(mask, torch.exp(amp / T - lse), torch.zeros_like(amp))
    cot = ws * p * u / (amp + 1e-12)
    for i in idx:
        cot[i] -= wt / len(idx) * u[i] / (amp[i] + 1e-12)
    return value, cot


def _phase_gradient(response, phases):
    """Re(conj(response) i e^{i phases})."""
    return (response.conj() * 1j * torch.exp(1j * phases)).real


def _material_gradient(mat, u, lam):
    """Gradients of dL = -Re(lam^H dA u) with respect to rho and c."""
    u, l = u.view(mat.shape), lam.view(mat.shape)
    rho, c = mat.rho, mat.c
    mass = mat.T[0] * mat.T[1] * mat.T[2] * (OMEGA ** 2 / (rho * c * c))
    prod = (l.conj() * u * mass).real
    gr, gc = prod / rho, 2 * prod / c
    for ax in range(3):
        n = mat.shape[ax]
        lo, hi = (lambda v: v.narrow(ax, 0, n - 1)), (lambda v: v.narrow(ax, 1, n - 1))
        de = mat.geom[ax] * (-2 / (lo(rho) + hi(rho)) ** 2)
        g = -((lo(l) - hi(l)).conj() * (hi(u) - lo(u)) * de).real
        lo(gr).add_(g)
        hi(gr).add_(g)
    for ax, pos, term in mat.face_terms:
        t = (l.narrow(ax, pos, 1).conj() * u.narrow(ax, pos, 1) * term).real
        gr.narrow(ax, pos, 1).add_(t / rho.narrow(ax, pos, 1))
        gc.narrow(ax, pos, 1).add_(t / c.narrow(ax, pos, 1))
    return gr.reshape(-1), gc.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "krylov":
        shape = _grid(case)
        mat = _Matrix(shape, case["faces"], *_medium(shape, seed), _pml(shape))
        rhs = _aperture_rhs(shape, case["nrhs"], seed)
        return torch.stack([_krylov(mat, b, case["restart"], case["iters"], 1e-9, case["recycle"],
                                    conj=case["adjoint"]) for b in rhs])
    if kind == "field":
        from ultrasound_solver_b200.workloads import fit_array
        n = case["n"]
        pitch, diameter = fit_array(case["array"], n, H)
        full = lambda v: torch.full((n ** 3,), v, dtype=torch.float64, device=DEV)
        mat = _Matrix((n, n, n), "open", full(RHO0), full(C0), PML)
        masses = _aperture_masses(n, _array_centers(n, case["array"], pitch), diameter)
        ph = torch.from_numpy(_phases(case["array"] ** 2, seed)).to(DEV)
        b = _source_rhs(n, masses, torch.exp(1j * ph)[None])[0]
        return _krylov(mat, b, 60, 20000, 1e-13)
    if kind == "scenes":
        out = []
        for i, n in enumerate(_edges(case)):
            full = lambda v: torch.full((n ** 3,), v, dtype=torch.float64, device=DEV)
            x = torch.arange(n, dtype=torch.float64, device=DEV) * H - (n - 1) * H / 2
            d = torch.sqrt(x[None, None, :] ** 2 + x[None, :, None] ** 2
                           + x[:, None, None] ** 2).reshape(-1) - 0.12 * (n - 1) * H
            t = (d / (1.2 * H)).clamp(-1, 1)
            step = 0.5 * (1 + t + torch.sin(math.pi * t) / math.pi)
            inv_rho = 1 / 1250.0 + (1 / RHO0 - 1 / 1250.0) * step
            comp_o = 1 / (1250.0 * 2200.0 ** 2)
            comp = comp_o + (1 / (RHO0 * C0 * C0) - comp_o) * step
            mat = _Matrix((n, n, n), "wall", 1 / inv_rho, torch.sqrt(inv_rho / comp), PML)
            out.append(_krylov(mat, _aperture_rhs((n, n, n), 1, seed + 31 * i)[0], case["restart"],
                               case["iters"], 1e-9, case["recycle"], every=2))
        return out
    if kind == "apply":
        shape = _grid(case)
        mat = _Matrix(shape, case["faces"], *_medium(shape, seed), _pml(shape))
        single = case["variant"] in ("K", "KH")
        x = _random_vectors(case["nrhs"], int(np.prod(shape)),
                            torch.complex64 if single else torch.complex128, seed)
        f = mat.K if case["variant"].startswith("K") else mat.A
        return torch.stack([f(v.to(torch.complex128), conj=case["variant"].endswith("H"))
                            for v in x])
    if kind == "setup":
        n = case["n"]
        st = prepare(case, seed)
        mat = _Matrix((n, n, n), "wall", st["rho"], st["c"], _pml((n, n, n)))
        masses = _aperture_masses(n, st["centers"], st["diameter"])
        flat = lambda v: v.reshape(-1)
        return [flat(mat.diag), flat(mat.R), flat(mat.s), flat(mat.R), flat(mat.s.conj()).clone(),
                torch.from_numpy(masses), _source_rhs(n, masses, st["coeff"])]
    if kind == "basis":
        shape = _grid(case)
        G = _basis_columns(case, seed)
        ph = torch.from_numpy(_phases(case["emitters"], seed)).to(DEV)
        w = torch.exp(1j * ph)
        u = torch.zeros(G.shape[1], dtype=torch.complex128, device=DEV)
        for col, wm in zip(G, w):
            u += wm * col.to(torch.complex128)
        cfg = _loss_config(shape)
        value, cot = _contrast_loss(u, shape, cfg.domain.box_size, cfg.targets, cfg.training)
        resp = torch.stack([torch.vdot(col.to(torch.complex128), cot) for col in G])
        return [u, value, cot, _phase_gradient(resp, ph)]
    from ultrasound_solver_b200.config import SimulationConfig
    from ultrasound_solver_b200.workloads import fit_array
    n = case["n"]
    cfg = SimulationConfig.from_dict(_scene_dict(n, case["array"], "wall", {}, target=True))
    pitch, diameter = fit_array(case["array"], n, H)
    mat = _Matrix((n, n, n), "wall", *_medium((n, n, n), seed), PML)
    masses = _aperture_masses(n, _array_centers(n, case["array"], pitch), diameter)
    ph = torch.from_numpy(_phases(case["array"] ** 2, seed)).to(DEV)
    u = _krylov(mat, _source_rhs(n, masses, torch.exp(1j * ph)[None])[0], 60, 20000, 1e-12)
    value, cot = _contrast_loss(u, (n, n, n), cfg.domain.box_size, cfg.targets, cfg.training)
    lam = _krylov(mat, cot, 60, 20000, 1e-12, conj=True)
    mt = torch.from_numpy(masses).to(DEV).to(torch.complex128)
    resp = (-2 * math.pi / (RHO0 * H ** 3)) * (mt @ lam[:n * n])
    return [u, value, _phase_gradient(resp, ph).cpu(), *_material_gradient(mat, u, lam)]
