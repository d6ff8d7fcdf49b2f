"""Timing cases of the library's main paths, through its public entry points.

Five kinds of work:

poisson   one pressure solve from x = 0 with MG-FGMRES (or ILU-BiCGStab) to a
          relative residual: the cut-cell Poisson operator on a box of cells
          with four spheres, Neumann walls and the two pinned rows, its mesh
          and operator built on the device from the spheres (lsg_mesh_build,
          lsg_set_matrix_mesh); the right-hand side is the divergence of a
          random velocity through the operator's open faces, so it is
          compatible, as the projection's is.  The pressure of solid cells is
          read by nobody and no equation fixes it; it is returned apart from
          the fluid cells'.
momentum  one momentum equation: ILU(0)-FGMRES on the implicit operator of one
          velocity component, from the current velocity, to the flow task's
          absolute tolerance.  The operator goes in as CSR in device memory
          (lsg_set_matrix_csr_device), as a GPU host program hands it over.
adjoint   one solve with the transposed pressure operator (host arrays, as the
          adjoint sweep's callers hold them).
flow      one time step of a flow past fixed bodies with the native stepper:
          three momentum equations, the pressure equation, the projection.
          Every pass sets the state (device copies) and takes the step, so
          that each pass does the same work.
gradient  a drag gradient: a few forward steps, the reverse sweep with its
          transposed solves (FlowAdjointDevice).

`api` "device" hands vectors over as device pointers, "host" as numpy arrays.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "ls-stag-3d_parallel_b200"))

from lsstag_b200 import _lib as L  # noqa: E402
from lsstag_b200 import cases as LC  # noqa: E402
from lsstag_b200 import flow as LF  # noqa: E402
from lsstag_b200 import flow_adjoint as LA  # noqa: E402
from lsstag_b200 import mesh as LM  # noqa: E402
from lsstag_b200 import solver as LS  # noqa: E402

DEV = "cuda:0"


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    p = dict(kind="poisson", method="fgmres", precision="fp64", gs="mgs", smoother="adlj", api="device", rel=1e-10)
    return [
        # a drop-in call from a host program on a test-sized grid: launches and latency
        dict(p, name="poisson_32x24x20_host", N=32, M=24, K=20, api="host"),
        # an ordinary mixed-precision solve
        dict(p, name="poisson_64_fp32", N=64, M=64, K=64, precision="fp32", gs="lowsync"),
        # a grid whose coarsening meets odd sizes, the reference's default options
        dict(p, name="poisson_150x90x70_fp64", N=150, M=90, K=70),
        # the benchmark's size, both precisions of the multigrid cycle
        dict(p, name="poisson_256_fp32", N=256, M=256, K=256, precision="fp32", gs="lowsync"),
        dict(p, name="poisson_256_fp64", N=256, M=256, K=256, gs="lowsync"),
        # the Gauss-Seidel smoother of the mixed-precision variant
        dict(p, name="poisson_128_rbgs_fp32", N=128, M=128, K=128, precision="fp32", gs="lowsync", smoother="rbgs"),
        # the reference's other solver, from host arrays
        dict(p, name="bicgstab_64x48x40_host", N=64, M=48, K=40, method="bicgstab", api="host"),
        # one momentum equation at the flow benchmark's size and on a larger ragged grid
        dict(kind="momentum", name="momentum_127x64x64", N=127, M=64, K=64, api="device"),
        # the transposed solve of the projection's adjoint
        dict(kind="adjoint", name="adjoint_96x80x64_host", N=96, M=80, K=64, rel=1e-10, precision="fp64"),
        # time steps: the flow benchmark (all FP64), a larger one with the FP32 cycle
        dict(kind="flow", name="flow_128x64x64_fp64", N=128, M=64, K=64, precision="fp64", bodies="sphere", p_rel=0.0),
        dict(kind="flow", name="flow_256x128x128_fp32", N=256, M=128, K=128, precision="fp32", bodies="ellipsoids",
             p_rel=1e-9),
        # reverse mode through time steps
        dict(kind="gradient", name="gradient_64x32x32_4steps", N=64, M=32, K=32, steps=4, every=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["poisson", "poisson", "poisson", "momentum", "adjoint", "flow", "gradient"])
    if kind == "poisson":
        n = _log(rng, 20, 224)
        dims = [max(16, int(n * rng.uniform(0.7, 1.3))) for _ in range(3)]
        # half of the grids are multiples of 16, as a user picks them; the rest as they fall
        if rng.random() < 0.5:
            dims = [max(16, 16 * round(d / 16)) for d in dims]
        while dims[0] * dims[1] * dims[2] > 12_000_000:
            dims[dims.index(max(dims))] //= 2
        if rng.random() < 0.2:
            while dims[0] * dims[1] * dims[2] > 400_000:
                dims[dims.index(max(dims))] = max(16, dims[dims.index(max(dims))] // 2)
            return dict(kind="poisson", N=dims[0], M=dims[1], K=dims[2], method="bicgstab", precision="fp64",
                        gs="mgs", smoother="adlj", api=rng.choice(["device", "host"]), rel=1e-10)
        precision = rng.choice(["fp64", "fp32"])
        return dict(kind="poisson", N=dims[0], M=dims[1], K=dims[2], method="fgmres", precision=precision,
                    gs=rng.choice(["mgs", "lowsync"]), smoother="adlj", api=rng.choice(["device", "host"]), rel=1e-10)
    if kind == "momentum":
        return dict(kind="momentum", N=_log(rng, 16, 255), M=_log(rng, 16, 128), K=_log(rng, 16, 128),
                    api=rng.choice(["device", "host"]))
    if kind == "adjoint":
        return dict(kind="adjoint", N=16 * rng.randint(1, 8), M=16 * rng.randint(1, 6), K=_log(rng, 16, 96), rel=1e-10,
                    precision=rng.choice(["fp64", "fp32"]))
    if kind == "flow":
        m = 16 * rng.randint(2, 6)
        return dict(kind="flow", N=2 * m + 16 * rng.randint(0, 3), M=m, K=m, precision=rng.choice(["fp64", "fp32"]),
                    bodies=rng.choice(["sphere", "ellipsoids"]), p_rel=rng.choice([0.0, 1e-8, 1e-9]))
    m = 16 * rng.randint(1, 3)
    return dict(kind="gradient", N=2 * m, M=m, K=m, steps=rng.randint(2, 5), every=rng.randint(1, 3))


# --------------------------------------------------------------------------
# operators and vectors of the solver cases, in plain torch
# --------------------------------------------------------------------------
def _gen(seed, dev):
    g = torch.Generator(device=dev)
    g.manual_seed(1000 * int(seed) + 7)
    return g


def _balls(dims, seed):
    """Four spheres that do not touch, (cx, cy, cz, r) each, and the cell size
    (the longest edge of the box is 1)."""
    h = 1.0 / max(dims)
    ext = [n * h for n in dims]
    r = np.random.default_rng(int(seed) + 11)
    corners = [(0.3, 0.3, 0.3), (0.7, 0.3, 0.7), (0.3, 0.7, 0.7), (0.7, 0.7, 0.3)]
    return [(*((c + r.uniform(-0.05, 0.05)) * e for c, e in zip(q, ext)), r.uniform(0.06, 0.14) * min(ext))
            for q in corners], h


def _openness(dims, seed, dev):
    """Open fractions of the east, north and top faces (zero on the box's own
    walls) around the spheres, from the signed distance at the face centres."""
    N, M, K = dims
    balls, h = _balls(dims, seed)
    ax = [torch.arange(n, device=dev, dtype=torch.float64) for n in (N, M, K)]
    out = []
    for d in range(3):
        pos = [(ax[k] + (1.0 if k == d else 0.5)) * h for k in range(3)]
        phi = torch.full((K, M, N), -1e30, device=dev, dtype=torch.float64)
        for cx, cy, cz, rad in balls:
            dist = ((pos[2][:, None, None] - cz) ** 2 + (pos[1][None, :, None] - cy) ** 2
                    + (pos[0][None, None, :] - cx) ** 2).sqrt()
            phi = torch.maximum(phi, rad - dist)
        th = (0.5 - phi / h).clamp(0.0, 1.0)
        th = torch.where(th < 1e-3, torch.zeros_like(th), th)
        th.select(2 - d, th.shape[2 - d] - 1).zero_()
        out.append(th)
    return out, h


def _shift(a, dim):
    """a's value at the previous index along dim, 0 before the first."""
    z = torch.zeros_like(a.narrow(dim, 0, 1))
    return torch.cat([z, a.narrow(dim, 0, a.shape[dim] - 1)], dim)


def _planes(th, scale, diag0):
    """(b, s, w, p, e, n, t) of -scale * (graph Laplacian of th) - diag0."""
    e, n, t = (a * scale for a in th)
    w, s, b = _shift(e, 2), _shift(n, 1), _shift(t, 0)
    p = -(e + w + n + s + t + b) - diag0
    return [b, s, w, p, e, n, t]


def _pins(dims):
    return [dims[0] - 1, dims[0] * dims[1] - 1]


def _build(s, dims, seed, task, setup=True):
    """The mesh and the pressure operator of the spheres on s's device."""
    balls, h = _balls(dims, seed)
    s.build_mesh(dims, (h,) * 3, LM.flow_block(dims, (h,) * 3, balls), bodies=LM.bodies_array(balls))
    s.set_from_mesh(_pins(dims), task=task, setup=setup)
    return s.planes()


def _poisson_rhs(P, dims, seed):
    """Right-hand side on the device, and the mask of the cells that it and
    the solution live on, for the operator's seven planes P."""
    N, M, K = dims
    fluid = torch.as_tensor(P[3], device=DEV).abs() > 1e-15
    g = _gen(seed, DEV)
    b = torch.zeros((K, M, N), device=DEV, dtype=torch.float64)
    for d in range(3):
        f = torch.as_tensor(P[4 + d], device=DEV).reshape(K, M, N)
        f = f * torch.randn((K, M, N), generator=g, device=DEV, dtype=torch.float64) / max(dims)
        b += f - _shift(f, 2 - d)
    b = b.reshape(-1)
    b[~fluid] = 0.0
    for q in _pins(dims):
        b[q] = 0.0
    return b, fluid


def _momentum(case, seed, dev):
    """The implicit operator 1.5/dt V u - nu lap u of one velocity component
    (dt 0.01, Re 100, h = 1/16), its right-hand side and the current velocity."""
    dims = (case["N"], case["M"], case["K"])
    N, M, K = dims
    th, _ = _openness(dims, seed, dev)
    h, nu, dt = 1.0 / 16, 0.01, 0.01
    P = -torch.stack(_planes(th, nu * h, 0.0)).reshape(7, -1)
    solid = P[3] == 0.0
    P[3] += 1.5 / dt * h ** 3
    P[3][solid] = 1e-16
    g = _gen(seed, dev)
    noise = 0.05 * torch.randn(N * M * K, generator=g, device=dev, dtype=torch.float64)
    x0 = torch.where(solid, torch.zeros_like(noise), 1.0 + noise)
    step = 0.05 * torch.randn(N * M * K, generator=g, device=dev, dtype=torch.float64)
    b = torch.where(solid, torch.zeros_like(noise), 1.5 / dt * h ** 3 * (x0 + step))
    return P, b, x0


def _neighbours(dims, dev):
    N, M, K = dims
    i = torch.arange(N * M * K, device=dev, dtype=torch.int64)
    x, y, z = i % N, (i // N) % M, i // (N * M)
    ok = [z > 0, y > 0, x > 0, x >= 0, x < N - 1, y < M - 1, z < K - 1]
    return i, ok, [-N * M, -N, -1, 0, 1, N, N * M]


def _csr(P, dims):
    """CSR on the device with every in-grid neighbour of each row."""
    i, ok, offs = _neighbours(dims, P.device)
    keep = torch.stack(ok, 1)
    col = torch.stack([i + o for o in offs], 1)[keep].to(torch.int32)
    val = P.t()[keep].contiguous()
    rowptr = torch.zeros(i.numel() + 1, dtype=torch.int32, device=P.device)
    rowptr[1:] = torch.cumsum(keep.sum(1), 0)
    return rowptr, col, val


def _set_csr(s, P, dims, task):
    """set() of the solver class with the operator in device memory."""
    rowptr, col, val = _csr(P, dims)
    torch.cuda.synchronize()
    s.task, s.eps, s.dims = task, float(task.eps), dims
    s.ctx.check(s.ctx.lib.lsg_set_matrix_csr_device(s.ctx.h, *dims, *(C.c_void_p(t.data_ptr())
                                                                     for t in (rowptr, col, val)), val.numel()))
    s.rebuildPreconditioner()


def _solver(case):
    kw = dict(mg_precision=L.FP32 if case.get("precision") == "fp32" else L.FP64,
              gram_schmidt=L.GS_LOWSYNC if case.get("gs") == "lowsync" else L.GS_MGS)
    if case["kind"] == "momentum":
        return LS.ILUFGMRES()
    if case.get("method") == "bicgstab":
        return LS.ILUBiCGStab()
    if case.get("smoother") == "rbgs":
        return LS.MGFGMRES(smoother=L.SMOOTHER_RBGS, n_pre=2, **kw)
    return LS.MGFGMRES(**kw)


# --------------------------------------------------------------------------
# prepare
# --------------------------------------------------------------------------
def prepare(case, seed):
    return {"poisson": _prepare_solve, "momentum": _prepare_solve, "adjoint": _prepare_solve,
            "flow": _prepare_flow, "gradient": _prepare_gradient}[case["kind"]](case, seed)


def _prepare_solve(case, seed):
    dims = (case["N"], case["M"], case["K"])
    s = _solver(case)
    st = {"kind": "solve", "api": case.get("api", "host"), "s": s}
    if case["kind"] == "momentum":
        P, b, x0 = _momentum(case, seed, DEV)
        _set_csr(s, P, dims, LS.Task(eps=1e-5, MAX_ITER=200, FGMRES_RESTART_NUM=13))
        fluid = None
    else:
        task = LS.Task(eps=0.0, MAX_ITER=400, FGMRES_RESTART_NUM=30, n_post=2 if case.get("smoother") == "rbgs" else 3)
        b, fluid = _poisson_rhs(_build(s, dims, seed, task, setup=False), dims, seed)
        task.eps = s.eps = case["rel"] * float(b.norm())
        s.rebuildPreconditioner()
        x0 = torch.zeros_like(b)
    if case["kind"] == "adjoint":
        st["kind"] = "adjoint"
    if st["api"] == "host":
        st.update(b=b.cpu().numpy(), x0=x0.cpu().numpy(), fluid=None if fluid is None else fluid.cpu().numpy())
    else:
        st.update(b=b, x0=x0, x=torch.empty_like(b), fluid=fluid)
    return st


def _split(x, fluid):
    """x on the fluid cells and on the others, 0 elsewhere."""
    if isinstance(x, np.ndarray):
        return [np.where(fluid, x, 0.0), np.where(fluid, 0.0, x)]
    return [torch.where(fluid, x, 0.0), torch.where(fluid, 0.0, x)]


def _bodies(case, seed, h):
    r = np.random.default_rng(int(seed) + 23)
    Lx, Ly, Lz = case["N"] * h, case["M"] * h, case["K"] * h
    if case.get("bodies") == "ellipsoids":
        out = []
        for k in range(3):
            q = r.standard_normal((3, 3))
            rot, _ = np.linalg.qr(q)
            if np.linalg.det(rot) < 0:
                rot[0] = -rot[0]
            c = np.array([(0.16 + 0.17 * k + 0.01 * r.random()) * Lx, (0.4 + 0.2 * r.random()) * Ly,
                          (0.4 + 0.2 * r.random()) * Lz])
            out.append((c, (0.05 + 0.06 * r.random(3)) * Ly, rot))
        return dict(ellipsoids=out)
    return dict(spheres=[(0.25 * Lx + 0.3 * h * r.random(), 0.5 * Ly + h * r.random(), 0.5 * Lz + h * r.random(),
                          0.125 * Ly)])


def _flow_case(case, seed, eps):
    """Mesh arrays and parameters of a flow past the bodies, and an initial
    velocity of the uniform stream with a few smooth disturbances."""
    dims = (case["N"], case["M"], case["K"])
    h = 4.0 / case["M"]
    g, dims, par, (u0, v0, w0, p0) = LC.flow_case_on_device(dims, (h, h, h), Re=100.0, dt=0.16 * h, eps=eps,
                                                            **_bodies(case, seed, h))
    r = np.random.default_rng(int(seed) + 37)

    def disturb(a, types, shape):
        z, y, x = (np.arange(n)[(slice(None),) + (None,) * (2 - k)] / n for k, n in enumerate(shape))
        f = np.zeros(shape)
        for _ in range(4):
            k = r.integers(1, 5, 3)
            f += 0.03 * r.standard_normal() * (np.sin(2 * np.pi * (k[0] * x + r.random()))
                                               * np.sin(np.pi * k[1] * y) * np.sin(np.pi * k[2] * z))
        return np.where(types != 0, a + f.reshape(-1), a)

    N, M, K = dims
    u0 = disturb(u0, g["xtype"], (K, M, N - 1))
    v0 = disturb(v0, g["ytype"], (K, M - 1, N))
    w0 = disturb(w0, g["ztype"], (K - 1, M, N))
    return g, dims, par, (u0, v0, w0, p0)


def _prepare_flow(case, seed):
    g, dims, par, st = _flow_case(case, seed, 1e-5)
    fs = LF.FlowStepperNative(g, dims, par, *st, pressure_mg_fp32=case["precision"] == "fp32",
                              p_rel_tol=case["p_rel"] or None)
    dev = [torch.as_tensor(np.ascontiguousarray(a), device=DEV) for a in st]
    return {"kind": "flow", "fs": fs, "state": dev, "out": [torch.empty_like(a) for a in dev]}


def _prepare_gradient(case, seed):
    g, dims, par, (u0, v0, w0, p0) = _flow_case(case, seed, 1e-9)
    par = dict(par, fcoef=float(g["fcoef"]))
    ops = LA.GpuFlowOps(g, dims, par)
    r = np.random.default_rng(int(seed) + 41)
    theta = 0.05 * r.standard_normal(8)
    forcing = [0.01 * r.standard_normal(a.size) for a in (u0, v0, w0)]
    return {"kind": "gradient", "fa": LA.FlowAdjointDevice(ops, case["steps"], every=case["every"]), "theta": theta,
            "forcing": forcing, "u": (u0, v0, w0), "p": p0}


# --------------------------------------------------------------------------
# run
# --------------------------------------------------------------------------
def run(st):
    if st["kind"] in ("solve", "adjoint"):
        s = st["s"]
        if st["kind"] == "adjoint":
            x = s.solve_adjoint(st["b"])
        elif st["api"] == "host":
            x = st["x0"].copy()
            s.solve(st["b"], x)
        else:
            x = st["x"]
            x.copy_(st["x0"])
            torch.cuda.current_stream().synchronize()      # the solver works on a stream of its own
            s.ctx.check(s.ctx.lib.lsg_solve_device(s.ctx.h, C.c_void_p(st["b"].data_ptr()),
                                                   C.c_void_p(x.data_ptr()), C.byref(s.stats)))
        return x if st["fluid"] is None else _split(x, st["fluid"])
    if st["kind"] == "flow":
        fs = st["fs"]
        arr3 = C.c_void_p * 3
        u = arr3(*[a.data_ptr() for a in st["state"][:3]])
        fs._check(fs.lib.lsg_flow_set_state(fs.h, u, u, C.c_void_p(st["state"][3].data_ptr()), None))
        fs.step()
        fs._check(fs.lib.lsg_flow_state(fs.h, arr3(*[a.data_ptr() for a in st["out"][:3]]),
                                        C.c_void_p(st["out"][3].data_ptr()), None))
        return st["out"]
    J, gth, gf = st["fa"].gradient(st["theta"], st["forcing"], st["u"], st["p"])
    return [J, gth, gf]


# --------------------------------------------------------------------------
# what a pass cannot do without, how close results are, exact results
# --------------------------------------------------------------------------
def work(case):
    """Inputs read once and outputs written once: the operator as its seven
    coefficients, the right-hand side and the solution; flops of one operator
    application.  How many iterations an algorithm takes is its own matter."""
    n = case["N"] * case["M"] * case["K"]
    if case["kind"] in ("poisson", "adjoint"):
        return {"bytes": n * (7 * 8 + 8 + 8), "flops": 14.0 * n}
    if case["kind"] == "momentum":
        return {"bytes": n * (7 * 8 + 3 * 8), "flops": 14.0 * n}
    # a step: four operators, the staggered geometry (types, face fractions,
    # cell sizes, volumes), state in and out
    step = {"bytes": n * (4 * 7 * 8 + 4 * 4 + 12 * 8 + 3 * 4 * 8 + 8 * 8), "flops": 200.0 * n}
    if case["kind"] == "flow":
        return step
    k = 3 * case["steps"]          # forward, recomputed, reverse
    return {"bytes": k * step["bytes"], "flops": k * step["flops"]}


def tolerance(case):
    """Two correct solvers stop below the same residual, not at the same
    iterate: their solutions differ by the stopping tolerance times what the
    operator's smallest singular value makes of it.  About four times what was
    measured over the ranges: the stopped solutions' distance from the exact
    ones (5e-6 for the pressure solves to 1e-10, 2e-5 for BiCGStab, 1.5e-8 for
    the momentum solves), and for the time steps and gradients their distance
    from the same ones with the other smoother schedule and the other
    Gram-Schmidt form (3e-7 and, largest value, 2e-5; gradients 1e-8, 4e-7)."""
    if case["kind"] == "momentum":
        return {"rel": 1e-7, "max": 1e-5}
    if case["kind"] == "flow":
        return {"rel": 2e-6, "max": 1e-4}
    if case["kind"] == "gradient":
        return {"rel": 1e-7, "max": 4e-6}
    if case.get("method") == "bicgstab":
        return {"rel": 1e-4, "max": 1e-3}
    return {"rel": 2e-5, "max": 2e-4}


def _cg(P, dims, b, x0, limit, rel):
    """Conjugate gradients with the diagonal preconditioner; rows without a
    diagonal of note (solid cells) stay out."""
    N, M, K = dims
    A = P.reshape(7, K, M, N)
    free = A[3].abs() > 1e-15
    inv = torch.where(free, 1.0 / A[3], torch.zeros_like(A[3]))

    def mul(x):
        y = A[3] * x
        y[1:] += A[0][1:] * x[:-1]
        y[:, 1:] += A[1][:, 1:] * x[:, :-1]
        y[:, :, 1:] += A[2][:, :, 1:] * x[:, :, :-1]
        y[:, :, :-1] += A[4][:, :, :-1] * x[:, :, 1:]
        y[:, :-1] += A[5][:, :-1] * x[:, 1:]
        y[:-1] += A[6][:-1] * x[1:]
        return y

    bb = b.reshape(K, M, N)
    x = x0.reshape(K, M, N).clone()
    r = torch.where(free, bb - mul(x), torch.zeros_like(bb))
    z = inv * r
    p, rz, stop = z.clone(), (r * z).sum(), rel * float(bb.norm())
    for it in range(limit):
        q = mul(p)
        a = rz / (p * q).sum()
        x += a * p
        r -= a * q
        if it % 20 == 19 and float(r.norm()) <= stop:
            break
        z = inv * r
        rz, old = (r * z).sum(), rz
        p = z + (rz / old) * p
    return x.reshape(-1)


def exact(case, seed):
    """The solver cases' solutions from conjugate gradients in plain torch, in
    64 bits; the pressure operator, an input of the solve, is the assembled
    one.  Nothing fixes the solid cells' values, and whole time steps and
    their gradients have no such short form: None."""
    dims = (case["N"], case["M"], case["K"])
    N, M, K = dims
    if case["kind"] == "momentum":
        P, b, x0 = _momentum(case, seed, DEV)
        x = _cg(P, dims, b, x0, 2000, 1e-14)
    elif case["kind"] in ("poisson", "adjoint"):
        s = LS.MGFGMRES()
        planes = _build(s, dims, seed, LS.Task(), setup=False)
        s.close()
        b, fluid = _poisson_rhs(planes, dims, seed)
        P = torch.as_tensor(planes, device=DEV)
        full, pins = P.clone(), _pins(dims)
        offs = [-N * M, -N, -1, 0, 1, N, N * M]
        cut = []                                # x is 0 at the pins: their columns drop out
        for q in pins:
            for k, o in enumerate(offs):
                if k != 3 and 0 <= q - o < P.shape[1]:
                    cut.append((q, k, q - o))
                    P[k, q - o] = 0.0
        x = _cg(P, dims, b, torch.zeros_like(b), 12000, 1e-13)
        if case["kind"] == "adjoint":           # the pins' rows of A^T hold the columns dropped above
            for q in pins:
                x[q] = (b[q] - sum(full[k, j] * x[j] for p, k, j in cut if p == q)) / full[3, q]
        x = [torch.where(fluid, x, 0.0), None]
    else:
        return None
    torch.cuda.synchronize()
    if case.get("api", "host") == "device":
        return x
    return [v if v is None else v.cpu().numpy() for v in x] if isinstance(x, list) else x.cpu().numpy()
