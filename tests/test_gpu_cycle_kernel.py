"""The cycle kernel (all Arnoldi steps of a restart cycle in one launch) against
one launch per Arnoldi pass, on the same capped solves.

A CTA cap larger than any grid keeps the per-pass kernels, which the other
files compare with the reference; everything else is the same. The two differ
in summation order and in the scale at which w is rounded. Bounds: FP64
rounding grown by the basis (1e-11); complex64 rounding over two cycles
(1e-5; measured 2e-8); for bfloat16 the spread between per-pass variants of
the same solve (measured up to 7e-3) times four.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-11, "mixed": 1e-5, "bf16": 3e-2}
FACES = {"-x": "open", "+x": "reflecting", "-y": {"type": "impedance", "impedance": [800.0, 100.0]},
         "+y": "open", "-z": "reflecting", "+z": "soft"}


def _operator(shape, seed):
    from ultrasound_solver_b200.scene import DeviceOperator
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = int(np.prod(shape))
    rand = lambda: torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
    return DeviceOperator(shape, 1e-3, 2 * np.pi * 4e4, FACES, 1.2 * (1 + 0.2 * rand()),
                          343 * (1 + 0.1 * rand()), pml={"cells": 2, "strength": 2.0, "order": 2})


def _rhs(nrhs, n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((nrhs, n), dtype=torch.complex128, device="cuda", generator=gen)


def _both(op, rhs, precision, **kw):
    from ultrasound_solver_b200.iterative_solver import B200IterativeSolver
    adjoint = kw.pop("adjoint", False)
    out = []
    for cap in (0, 1 << 20):
        it = B200IterativeSolver(rtol=1e-13, precision=precision, max_ctas=cap, **kw)
        x = it.solve(op, rhs, adjoint=adjoint, raise_on_failure=False)
        out.append((x, it.last_stats))
    return out


@pytest.mark.parametrize("precision", ["fp64", "mixed", "bf16"])
@pytest.mark.parametrize("shape,nrhs,restart,recycle,adjoint", [
    ((6, 5, 7), 1, 12, 0, False),        # less than one 64-node group per CTA
    ((9, 8, 8), 3, 30, 8, True),         # 576 nodes: most CTAs own none
    ((33, 31, 29), 2, 17, 0, True),      # ragged ranges, basis resident
    ((64, 63, 61), 1, 30, 5, False),     # part of the basis read from global memory
    ((41, 40, 39), 4, 40, 3, False),     # more vector groups than warps hold at once
    ((24, 23, 22), 1, 100, 0, False),    # long basis
    ((70, 69, 68), 1, 12, 3, False),     # 2240 nodes per CTA (complex128: both sides per-pass kernels)
    ((80, 79, 78), 1, 9, 4, True),       # 3392 nodes per CTA (complex128: as above)
    ((90, 91, 89), 1, 11, 0, False),     # 4928 nodes per CTA (bfloat16 only)
])
def test_against_per_pass_kernels(precision, shape, nrhs, restart, recycle, adjoint):
    op = _operator(shape, 5)
    rhs = _rhs(nrhs, op.n, 7)
    (x, st), (y, st2) = _both(op, rhs, precision, restart=restart, recycle=recycle,
                              maxiter=3 * restart, adjoint=adjoint)
    for b in range(nrhs):
        assert st[b]["iterations"] == st2[b]["iterations"]
        err = float(torch.linalg.norm(x[b] - y[b]) / torch.linalg.norm(y[b]))
        assert err <= TOL[precision], (b, err)


@pytest.mark.parametrize("precision", ["fp64", "mixed", "bf16"])
def test_scenes_and_finished_columns(precision):
    """Scenes of different sizes in one launch; a zero right-hand side ends at
    once, so its CTAs go to the others from the first cycle on."""
    from ultrasound_solver_b200 import _native as N
    import ctypes as C
    shapes = [(12, 11, 10), (30, 29, 28), (21, 20, 22), (12, 11, 10)]
    ops = [_operator(s, 3 + i) for i, s in enumerate(shapes)]
    ld = max(o.n for o in ops)
    rhs = torch.zeros((4, ld), dtype=torch.complex128, device="cuda")
    for i, o in enumerate(ops[:3]):
        rhs[i, :o.n] = _rhs(1, o.n, 20 + i)[0]
    from ultrasound_solver_b200.iterative_solver import B200IterativeSolver
    got = []
    for cap in (0, 1 << 20):
        it = B200IterativeSolver(restart=14, maxiter=42, rtol=1e-13, precision=precision,
                                 recycle=4, max_ctas=cap)
        p = it.params()
        scenes = (N.Scene * 4)(*[o.scene for o in ops])
        bufs = (C.c_void_p * 4)(*[o.buffer.data_ptr() for o in ops])
        of = (C.c_int * 4)(0, 1, 2, 3)
        nbytes = C.c_size_t()
        lib = N.load()
        N.check(lib.usv_gmres_scenes_workspace_bytes(4, scenes, of, C.byref(p), 4, C.byref(nbytes)))
        ws = torch.empty(nbytes.value, dtype=torch.uint8, device="cuda")
        x = torch.empty_like(rhs)
        stats = (N.GmresStats * 4)()
        hist = (C.c_double * (4 * p.history_capacity))()
        p.history = C.cast(hist, C.POINTER(C.c_double))
        N.check(lib.usv_gmres_solve_scenes(4, scenes, bufs, of, C.byref(p), N.ptr(rhs), N.ptr(x), 4,
                                           ld, N.ptr(ws), nbytes.value, stats,
                                           N.stream_handle(torch, x.device)))
        assert stats[3].iterations == 0 and stats[3].status == N.USV_OK
        got.append(x)
    for i, o in enumerate(ops[:3]):
        a, b = got[0][i, :o.n], got[1][i, :o.n]
        err = float(torch.linalg.norm(a - b) / torch.linalg.norm(b))
        assert err <= TOL[precision], (i, err)


def _solve_scenes(ops, rhs, cap, **kw):
    """usv_gmres_solve_scenes with one right-hand side per scene, up to the iteration cap."""
    import ctypes as C
    from ultrasound_solver_b200 import _native as N
    from ultrasound_solver_b200.iterative_solver import B200IterativeSolver
    count = len(ops)
    it = B200IterativeSolver(max_ctas=cap, **kw)
    p = it.params()
    p.history_capacity = 0
    scenes = (N.Scene * count)(*[o.scene for o in ops])
    bufs = (C.c_void_p * count)(*[o.buffer.data_ptr() for o in ops])
    of = (C.c_int * count)(*range(count))
    nbytes = C.c_size_t()
    lib = N.load()
    N.check(lib.usv_gmres_scenes_workspace_bytes(count, scenes, of, C.byref(p), count, C.byref(nbytes)))
    ws = torch.empty(nbytes.value, dtype=torch.uint8, device="cuda")
    x = torch.empty_like(rhs)
    stats = (N.GmresStats * count)()
    N.check(lib.usv_gmres_solve_scenes(count, scenes, bufs, of, C.byref(p), N.ptr(rhs), N.ptr(x), count,
                                       rhs.shape[1], N.ptr(ws), nbytes.value, stats,
                                       N.stream_handle(torch, x.device)))
    return x, stats


@pytest.mark.parametrize("finished", ["zero", "easy"])
@pytest.mark.parametrize("precision,edges", [("bf16", (12, 42, 64, 64)), ("mixed", (10, 40, 35, 35)),
                                             ("fp64", (10, 33, 28, 45))])
def test_share_that_grows_when_a_scene_finishes(precision, edges, finished):
    """Scenes whose largest range is that of an instance while all are active
    and one group of 64 nodes more once the first has finished: before the
    first cycle (zero right-hand side) or between cycles (at a hundred times
    the frequency its Jacobi-scaled rows are near the identity). Bounds as above."""
    from ultrasound_solver_b200 import _native as N
    from ultrasound_solver_b200.scene import DeviceOperator
    ops = [_operator((n, n, n), 40 + i) for i, n in enumerate(edges)]
    if finished == "easy":
        n = edges[0]
        full = lambda v: torch.full((n ** 3,), v, dtype=torch.float64, device="cuda")
        ops[0] = DeviceOperator((n, n, n), 1e-3, 2 * np.pi * 4e6, FACES, full(1.2), full(343.0),
                                pml={"cells": 2, "strength": 2.0, "order": 2})
    ld = max(o.n for o in ops)
    rhs = torch.zeros((len(ops), ld), dtype=torch.complex128, device="cuda")
    for i, o in enumerate(ops):
        if i > 0 or finished == "easy":
            rhs[i, :o.n] = _rhs(1, o.n, 60 + i)[0]
    kw = dict(restart=14, recycle=4, maxiter=56, rtol=1e-4, backward_error_tol=1.0, precision=precision)
    (x, st), (y, st2) = (_solve_scenes(ops, rhs, cap, **kw) for cap in (0, 1 << 20))
    assert st[0].status == N.USV_OK and st[0].iterations <= 28
    for i, o in enumerate(ops):
        assert st[i].iterations == st2[i].iterations
        if i > 0:
            assert st[i].iterations >= 48  # (whole cycles up to the cap)
        if i > 0 or finished == "easy":
            a, b = x[i, :o.n], y[i, :o.n]
            err = float(torch.linalg.norm(a - b) / torch.linalg.norm(b))
            assert err <= TOL[precision], (i, err)


@pytest.mark.parametrize("restart", [12, 100])
def test_more_than_8192_nodes_per_cta(restart):
    """The largest bfloat16 instance (three segments of nodes per CTA), with
    more dots tasks than a short basis has (25 groups of vectors)."""
    shape = (87, 86, 85)
    ops = [_operator(shape, 70 + i) for i in range(2)]
    rhs = torch.cat([_rhs(1, o.n, 80 + i) for i, o in enumerate(ops)])
    kw = dict(restart=restart, maxiter=2 * restart, rtol=1e-13, precision="bf16")
    (x, st), (y, st2) = (_solve_scenes(ops, rhs, cap, **kw) for cap in (0, 1 << 20))
    for b in range(2):
        assert st[b].iterations == st2[b].iterations
        err = float(torch.linalg.norm(x[b] - y[b]) / torch.linalg.norm(y[b]))
        assert err <= TOL["bf16"], (b, err)


@pytest.mark.parametrize("precision,shape,scenes,recycle", [
    ("bf16", (105, 106, 107), 1, 4),    # 8064 of 8192 nodes per CTA
    ("mixed", (84, 84, 85), 1, 0),      # 4096 of 4096
    ("fp64", (66, 65, 67), 1, 3),       # 1984 of 2048
    ("mixed", (75, 76, 77), 2, 4),      # 5952 of 8192, scenes in one launch
])
def test_largest_instances(precision, shape, scenes, recycle):
    """The instances with most nodes per CTA, near the sizes where they end. Bounds as above."""
    ops = [_operator(shape, 90 + i) for i in range(scenes)]
    rhs = torch.cat([_rhs(1, o.n, 95 + i) for i, o in enumerate(ops)])
    kw = dict(restart=13, recycle=recycle, maxiter=39)
    if scenes == 1:
        (x, st), (y, st2) = _both(ops[0], rhs, precision, **kw)
        assert st[0]["iterations"] == st2[0]["iterations"]
    else:
        (x, _), (y, _) = (_solve_scenes(ops, rhs, cap, rtol=1e-13, precision=precision, **kw) for cap in (0, 1 << 20))
    for b in range(scenes):
        err = float(torch.linalg.norm(x[b] - y[b]) / torch.linalg.norm(y[b]))
        assert err <= TOL[precision], (b, err)
