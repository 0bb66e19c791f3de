"""Performance cases: the work a user of this framework has it do, timed one pass at a time.

Every case is one program's call sequence on the public API: the device-resident
run (`GpuWorkspace.run`), the drop-in loop of the reference's driver
(`compute_dt_gpu` / `advance_second_order_gpu` / `swap`), the same loop as a whole
session on host arrays, a batch of uneven instances (`Batch.run`) and the adjoint
gradient (`OTAdjoint.gradient`).  A pass restarts from the state that `prepare`
made, as a parameter scan or an ensemble does, so it is the same work each time.

`exact` is the same scheme in plain torch, 64 bits, written from the method:
MUSCL-Hancock (minmod or van Leer, the positivity fallbacks), HLL / HLLC / HLLD /
FORCE with the GLM interface values, x- then y-sweep, psi damping.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import mhd_gpu_acc_b200 as mhd
from mhd_gpu_acc_b200.adjoint import OTAdjoint
from mhd_gpu_acc_b200.batch import Batch, instance

NG = 2
CR = 0.18
SOLVERS = {"hll": 0, "hllc": 1, "hlld": 2, "force": 3}
LIMITERS = {"minmod": 0, "vanleer": 1}
BCS = {"periodic": (0, 0, 0, 0), "outflow": (1, 1, 1, 1), "channel": (0, 0, 2, 2), "tube": (1, 1, 0, 0)}
GAMMA = {"vortex": 5.0 / 3.0, "bubble": 5.0 / 3.0, "tube": 2.0, "shear": 1.4}
RHO, MX, MY, MZ, BX, BY, BZ, EN, PSI = range(9)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _grid(name, kind, nx, ny, dtype, flow, solver, limiter, bc, cfl, steps):
    return dict(name=name, kind=kind, nx=nx, ny=ny, dtype=dtype, flow=flow, solver=solver, limiter=limiter, bc=bc,
                cfl=cfl, steps=steps)


def listed():
    return [
        # the headline: a production-size Orszag-Tang-like vortex, FP32-bulk, device-resident loop
        _grid("run_f32_4096", "run", 4096, 4096, "f32", "vortex", "hlld", "vanleer", "periodic", 0.4, 6),
        # the same at the size of parameter scans and of the accuracy runs
        _grid("run_f32_512", "run", 512, 512, "f32", "vortex", "hlld", "vanleer", "periodic", 0.4, 24),
        # the plain FP64 step, which reproduces the reference, at a middling size
        _grid("run_f64_2048", "run", 2048, 2048, "f64", "vortex", "hlld", "vanleer", "periodic", 0.4, 4),
        # the smallest: the Brio-Wu tube as a thin 2D grid, FP64, minmod, all sides open
        _grid("run_f64_tube_800x4", "run", 800, 4, "f64", "tube", "hlld", "minmod", "outflow", 0.8, 32),
        # a Mach-10 shock meeting a dense bubble, outflow sides, HLLC
        _grid("run_f32_bubble_2048", "run", 2048, 2048, "f32", "bubble", "hllc", "vanleer", "outflow", 0.4, 8),
        # a shear layer in a channel with reflecting walls, odd extents, FP64 HLL
        _grid("run_f64_shear_515x1031", "run", 515, 1031, "f64", "shear", "hll", "minmod", "channel", 0.4, 8),
        # the reference driver's own loop on device states: dt read back each step, three states, swap
        _grid("dropin_f64_1000x500", "dropin", 1000, 500, "f64", "bubble", "hllc", "minmod", "outflow", 0.4, 6),
        # a whole short session on the reference's host arrays: upload, drop-in steps, download
        _grid("session_f64_512", "session", 512, 512, "f64", "vortex", "hlld", "minmod", "periodic", 0.4, 8),
        # uneven Orszag-Tang instances advanced together: a small sweep and a wide one
        dict(name="batch_f32_32", kind="batch", count=32, side_min=64, side_max=512, dtype="f32", solver="hlld",
             limiter="vanleer", steps=10),
        dict(name="batch_f32_96", kind="batch", count=96, side_min=64, side_max=1024, dtype="f32", solver="hlld",
             limiter="vanleer", steps=6),
        # gradients of the Orszag-Tang objective: the FP32 one that an optimiser iterates on, the FP64 one it is held to
        dict(name="adjoint_f32_512", kind="adjoint", n=512, dtype="f32", solver="hll", limiter="vanleer", steps=30),
        dict(name="adjoint_f64_256", kind="adjoint", n=256, dtype="f64", solver="hlld", limiter="vanleer", steps=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "dropin", "session", "batch", "adjoint"])
    dtype = "f64" if kind == "session" else rng.choice(["f32", "f64"])
    solver = rng.choice(["hll", "hllc", "hlld", "hlld", "force"])
    limiter = rng.choice(["minmod", "vanleer"])
    if kind == "batch":
        lo = rng.choice([32, 64, 96])
        return dict(kind=kind, count=rng.randint(6, 48), side_min=lo, side_max=rng.randint(160, 640), dtype=dtype,
                    solver=solver, limiter=limiter, steps=rng.randint(3, 8 if dtype == "f32" else 4))
    if kind == "adjoint":
        n = _log_int(rng, 48, 512 if dtype == "f32" else 320)
        return dict(kind=kind, n=n, dtype=dtype, solver=rng.choice(["hll", "hlld"]), limiter=limiter,
                    steps=rng.randint(6, 24))
    flow = rng.choice(["vortex", "vortex", "bubble", "tube", "shear"])
    bc = {"vortex": "periodic", "bubble": "outflow", "tube": rng.choice(["tube", "outflow"]), "shear": "channel"}[flow]
    top = 1024 if kind == "session" else 4096 if dtype == "f32" else 2300
    nx = _log_int(rng, 200 if flow == "tube" else 48, top)
    ny = rng.randint(4, 40) if flow == "tube" else max(33, min(top, int(nx * math.exp(rng.uniform(-0.7, 0.7)))))
    most = 1.0e8 if dtype == "f32" else 1.6e7  # cell-updates of a pass
    steps = max(2, min(rng.randint(4, 24), int(most / (nx * ny))))
    return dict(kind=kind, nx=nx, ny=ny, dtype=dtype, flow=flow, solver=solver, limiter=limiter, bc=bc,
                cfl=round(rng.uniform(0.3, 0.45), 3), steps=steps)


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _to_cons(rho, u, v, w, bx, by, bz, p, gamma):
    e = p / (gamma - 1.0) + 0.5 * rho * (u * u + v * v + w * w) + 0.5 * (bx * bx + by * by + bz * bz)
    return torch.stack([rho, rho * u, rho * v, rho * w, bx, by, bz, e, torch.zeros_like(rho)])


def _initial(case, seed):
    """Conserved FP64 state (9, ny + 4, nx + 4) of a grid case: interior cells, ghosts filled by the boundary rules."""
    nx, ny, flow = case["nx"], case["ny"], case["flow"]
    gamma, dev = GAMMA[flow], _device()
    r = np.random.default_rng([seed, nx, ny])
    x = ((torch.arange(nx, dtype=torch.float64, device=dev) + 0.5) / nx)[None, :]
    y = ((torch.arange(ny, dtype=torch.float64, device=dev) + 0.5) / ny)[:, None]
    one = torch.ones(ny, nx, dtype=torch.float64, device=dev)
    tau = 2.0 * math.pi
    if flow == "vortex":  # Orszag-Tang with random modes on top and discs of another density and pressure
        b0 = 1.0 / math.sqrt(4.0 * math.pi)
        u, v = -torch.sin(tau * y) * one, torch.sin(tau * x) * one
        bx, by = -b0 * torch.sin(tau * y) * one, b0 * torch.sin(2.0 * tau * x) * one
        for mx, my in ((1, 0), (0, 1), (1, 1), (1, -1), (2, 1), (1, 2), (3, -2)):
            a, b, p0, p1 = r.normal(0.0, 0.06, 2).tolist() + r.uniform(0.0, tau, 2).tolist()
            k = math.hypot(mx, my)
            s, q = torch.sin(tau * (mx * x + my * y) + p0) / k, torch.sin(tau * (mx * x + my * y) + p1) / k
            u, v = u - a * s * my, v + a * s * mx
            bx, by = bx - 0.4 * b * q * my, by + 0.4 * b * q * mx
        rho, p = 25.0 / (36.0 * math.pi) * one, 5.0 / (12.0 * math.pi) * one
        for _ in range(4):
            cx, cy, rad = r.uniform(0, 1), r.uniform(0, 1), r.uniform(0.05, 0.15)
            inside = ((x - cx + 0.5) % 1.0 - 0.5) ** 2 + ((y - cy + 0.5) % 1.0 - 0.5) ** 2 < rad * rad
            rho = torch.where(inside, rho * float(r.uniform(0.6, 2.5)), rho)
            p = torch.where(inside, p * float(r.uniform(0.7, 3.0)), p)
        w, bz = 0.1 * torch.sin(tau * (x + y)) * one, 0.05 * torch.cos(tau * (x - y)) * one
    elif flow == "bubble":  # a Rankine-Hugoniot shock running into a dense bubble
        mach, xs = float(r.uniform(6.0, 10.0)), float(r.uniform(0.5, 0.6))
        cx, cy, rad, dense = (float(r.uniform(*q)) for q in ((0.75, 0.85), (0.4, 0.6), (0.1, 0.15), (4.0, 10.0)))
        rho2 = (gamma + 1.0) * mach**2 / ((gamma - 1.0) * mach**2 + 2.0)
        p2 = (2.0 * gamma * mach**2 - (gamma - 1.0)) / (gamma + 1.0)
        u2 = mach * math.sqrt(gamma) * (1.0 - 1.0 / rho2)
        post = (x < xs) & (y > -1.0)
        inside = (x - cx) ** 2 + (y - cy) ** 2 < rad * rad
        rho = torch.where(post, rho2 * one, torch.where(inside, dense * one, one))
        p, u = torch.where(post, p2 * one, one), torch.where(post, u2 * one, 0.0 * one)
        v, w, bx, bz = 0.0 * one, 0.0 * one, 0.0 * one, 0.0 * one
        by = 2.0 / math.sqrt(4.0 * math.pi) * one
    elif flow == "tube":  # Brio-Wu with the states varied
        left, s = (x < float(r.uniform(0.45, 0.55))) & (y > -1.0), r.uniform(0.9, 1.1, 4)
        pick = lambda a, b: torch.where(left, float(a) * one, float(b) * one)  # noqa: E731
        rho, p, by = pick(s[0], 0.125 * s[1]), pick(s[2], 0.1 * s[3]), pick(s[1], -s[0])
        u, v, w, bz, bx = 0.0 * one, 0.0 * one, 0.0 * one, 0.0 * one, 0.75 * one
    else:  # "shear": two shear layers with a perturbed normal velocity
        width, a = float(r.uniform(15.0, 25.0)), float(r.uniform(0.2, 0.3))
        u = 5.0 * (torch.tanh(width * (y - 0.25)) - torch.tanh(width * (y - 0.75)) - 1.0) * one
        v = a * torch.sin(tau * x) * (torch.exp(-100.0 * (y - 0.25) ** 2) - torch.exp(-100.0 * (y - 0.75) ** 2))
        w, bz, by, bx = 0.0 * one, 0.0 * one, 0.0 * one, one
        rho, p = one + 0.2 * torch.sin(tau * x + float(r.uniform(0, tau))) * one, 50.0 * one
    U = torch.zeros(9, ny + 2 * NG, nx + 2 * NG, dtype=torch.float64, device=dev)
    U[:, NG:-NG, NG:-NG] = _to_cons(rho, u, v, w, bx, by, bz, p, gamma)
    _fill_ghosts(U, BCS[case["bc"]])
    return U.to(torch.float32).to(torch.float64) if case["dtype"] == "f32" else U


def _amplitudes(seed):
    return np.random.default_rng([seed, 16]).normal(0.0, 0.01, 16)


def _target(n, seed):
    """A density the gradient is taken against: the uniform start plus smooth modes."""
    r, s = np.random.default_rng([seed, n]), (np.arange(n) + 0.5) / n
    rho = np.full((n, n), 25.0 / (36.0 * math.pi))
    for mx, my in ((1, 0), (0, 1), (1, 1), (2, 1)):
        rho += 0.02 * r.normal() * np.sin(2.0 * math.pi * (mx * s[None, :] + my * s[:, None]))
    return rho


def _batch_members(case, seed):
    """The instances of a batch: sides, field amplitudes, gammas and CFL numbers (the uneven Orszag-Tang sweep)."""
    # sides belong to the case, so that every seed is the same work
    sides = np.random.default_rng([case["count"], case["side_max"]]).integers(case["side_min"], case["side_max"] + 1,
                                                                               (case["count"], 2))
    r = np.random.default_rng([seed, case["count"]])
    return [dict(nx=int(a), ny=int(a if k % 4 else b), b0=float(r.uniform(0.5, 1.5) / math.sqrt(4.0 * math.pi)),
                 gamma=float(r.choice([5.0 / 3.0, 2.0])), cfl=float(r.uniform(0.3, 0.5)))
            for k, (a, b) in enumerate(sides)]


_MODES = ((1, 0), (0, 1), (1, 1), (1, -1), (2, 0), (0, 2), (2, 1), (1, 2))


def _orszag_tang(nx, ny, b0, gamma, amp=None):
    """Orszag-Tang on [0,1]^2 at every cell centre, ghosts included; `amp`: 16 Fourier amplitudes (a tensor)."""
    dev, tau = _device(), 2.0 * math.pi
    x = ((torch.arange(-NG, nx + NG, dtype=torch.float64, device=dev) + 0.5) / nx)[None, :]
    y = ((torch.arange(-NG, ny + NG, dtype=torch.float64, device=dev) + 0.5) / ny)[:, None]
    one = torch.ones(ny + 2 * NG, nx + 2 * NG, dtype=torch.float64, device=dev)
    u, v = -torch.sin(tau * y) * one, torch.sin(tau * x) * one
    bx, by = -b0 * torch.sin(tau * y) * one, b0 * torch.sin(2.0 * tau * x) * one
    if amp is not None:
        for m, (mx, my) in enumerate(_MODES):
            s = torch.sin(tau * (mx * x + my * y)) / math.hypot(mx, my)
            u, v = u - amp[m] * s * my, v + amp[m] * s * mx
            bx, by = bx - amp[8 + m] * s * my, by + amp[8 + m] * s * mx
    rho, p = 25.0 / (36.0 * math.pi) * one, 5.0 / (12.0 * math.pi) * one
    return _to_cons(rho, u, v, 0.0 * one, bx, by, 0.0 * one, p, gamma)


# ---------------------------------------------------------------------------
# the framework's side
# ---------------------------------------------------------------------------
class _Ptr:
    """Device memory for torch; a tensor made from it holds it, and with it the memory's owner."""

    def __init__(self, owner, ptr, shape, strides, kind):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, strides=strides, typestr=kind, data=(int(ptr), False), version=3)


def _views(g, owner):
    """(state as (9, ny + 4, nx + 4), the whole padded slab) as torch tensors on a grid's memory, which `owner` frees."""
    e = 4 if g.dtype == mhd.F32 else 8
    shape = (9, g.ny + 2 * g.ng, g.nx + 2 * g.ng)
    return (torch.as_tensor(_Ptr(owner, g.data, shape, (g.plane * e, g.pitch * e, e), "<f%d" % e), device="cuda"),
            torch.as_tensor(_Ptr(owner, g.data, (9 * g.plane,), (e,), "<f%d" % e), device="cuda"))


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def _workspace(grid, gamma, limiter):
    ws = mhd.GpuWorkspace()
    mhd.init_gpu_workspace(ws, grid)
    mhd.set_gpu_physics_gamma(ws, gamma)
    mhd.set_gpu_physics_ch(ws, 0.0)
    ws.set_limiter(LIMITERS[limiter])
    return ws


def _prepare_grid(case, seed):
    dtype = mhd.F32 if case["dtype"] == "f32" else mhd.F64
    U0 = _initial(case, seed)
    grids = [mhd.Grid2DGPU(case["nx"], case["ny"], NG, 0.0, 1.0, 0.0, 1.0, dtype)
             for _ in range(2 if case["kind"] == "run" else 3)]
    s = dict(case, grids=grids, ws=_workspace(grids[0], GAMMA[case["flow"]], case["limiter"]))
    if case["kind"] == "session":
        s["aos"] = np.ascontiguousarray(U0.permute(1, 2, 0).reshape(-1, 9).cpu().numpy())
        return s
    s["views"] = {g.g.data: _views(g.g, grids) for g in grids}
    for state, _ in s["views"].values():
        state.copy_(U0)
    s["start"] = s["views"][grids[0].g.data][1].clone()
    return s


def _run_device(s):
    U, T = s["grids"]
    state, slab = s["views"][U.g.data]
    slab.copy_(s["start"])
    mhd.set_gpu_physics_ch(s["ws"], 0.0)
    info = s["ws"].run(U, T, s["cfl"], 10.0, s["steps"], SOLVERS[s["solver"]], BCS[s["bc"]])
    real = np.float32 if s["dtype"] == "f32" else np.float64
    return {"U": state, "t": real(info.t), "dt": real(info.last_dt), "ch": real(info.ch)}


def _steps(s):
    old, tmp, new = s["grids"]
    mhd.set_gpu_physics_ch(s["ws"], 0.0)
    t = 0.0
    for _ in range(s["steps"]):
        dt = mhd.compute_dt_gpu(old, s["ws"], s["cfl"])
        mhd.advance_second_order_gpu(old, tmp, new, s["ws"], dt, SOLVERS[s["solver"]], BCS[s["bc"]])
        old.swap(new)
        t += dt
    return t


def _run_dropin(s):
    s["views"][s["grids"][0].g.data][1].copy_(s["start"])
    t = _steps(s)
    return {"U": s["views"][s["grids"][0].g.data][0], "t": np.float32(t) if s["dtype"] == "f32" else t}


def _run_session(s):
    s["grids"][0].upload_from_aos(s["aos"])
    t = _steps(s)
    return {"aos": s["grids"][0].download_to_aos(), "t": t}


def _prepare_batch(case, seed):
    members = _batch_members(case, seed)
    b = Batch([instance(m["nx"], m["ny"], m["gamma"], m["cfl"], 10.0) for m in members],
              dtype=mhd.F32 if case["dtype"] == "f32" else mhd.F64, solver=SOLVERS[case["solver"]],
              limiter=LIMITERS[case["limiter"]])
    views = [_views(b.grid(i), b) for i in range(len(members))]
    for m, (state, _) in zip(members, views):
        state.copy_(_orszag_tang(m["nx"], m["ny"], m["b0"], m["gamma"]))
    return dict(case, batch=b, states=[v[0] for v in views], slabs=[v[1] for v in views],
                start=[v[1].clone() for v in views])


def _run_batch(s):
    torch._foreach_copy_(s["slabs"], s["start"])
    infos = s["batch"].run(s["steps"])
    # cell values of all instances, one after the other
    real = np.float32 if s["dtype"] == "f32" else np.float64
    return {"U": torch.cat([v.reshape(-1) for v in s["states"]]), "t": np.array([i.t for i in infos], real)}


def _prepare_adjoint(case, seed):
    a = OTAdjoint(case["n"], case["steps"], mhd.F32 if case["dtype"] == "f32" else mhd.F64, LIMITERS[case["limiter"]],
                  solver=SOLVERS[case["solver"]])
    a.set_target(_target(case["n"], seed))
    return dict(case, adjoint=a, amp=_amplitudes(seed))


def _run_adjoint(s):
    J, grad = s["adjoint"].gradient(s["amp"])
    real = np.float32 if s["dtype"] == "f32" else np.float64  # the gradient in the precision that it was computed in
    return {"J": real(J), "grad": grad.astype(real)}


_PREPARE = {"run": _prepare_grid, "dropin": _prepare_grid, "session": _prepare_grid, "batch": _prepare_batch,
            "adjoint": _prepare_adjoint}
_RUN = {"run": _run_device, "dropin": _run_dropin, "session": _run_session, "batch": _run_batch,
        "adjoint": _run_adjoint}


# ---------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------
# floating operations of one cell and sweep: the slopes and the half step, the
# solver, the update; counted from the formulas below, a division or root as one
_SWEEP_FLOPS = {"hll": 340, "hllc": 360, "hlld": 430, "force": 420}


def work(case):
    size = 4 if case["dtype"] == "f32" else 8
    if case["kind"] == "batch":
        cells = sum(m["nx"] * m["ny"] for m in _batch_members(case, 0))
    else:
        cells = case["n"] ** 2 if case["kind"] == "adjoint" else case["nx"] * case["ny"]
    updates = cells * case["steps"]
    flops = 2 * _SWEEP_FLOPS[case["solver"]] * updates
    if case["kind"] == "adjoint":
        # a step forward, and backward: the state and its cotangent in, the cotangent out; three times the operations
        return {"bytes": 9 * size * 5 * updates, "flops": 4 * flops}
    # a step reads the nine fields once and writes them once
    return {"bytes": 9 * size * 2 * updates, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _fill_ghosts(U, bc):
    """Ghost cells of a (9, ny + 4, nx + 4) state by the four sides' rules, in place."""
    for axis, (lo, hi), comps in ((2, bc[:2], (MX, BX)), (1, bc[2:], (MY, BY))):
        V = U if axis == 2 else U.transpose(1, 2)
        n = V.shape[2] - 2 * NG
        for q in range(NG):
            for rule, dst, src in ((lo, NG - 1 - q, (NG + n - 1 - q, NG, NG + q)[min(lo, 2)]),
                                   (hi, NG + n + q, (NG + q, NG + n - 1, NG + n - 1 - q)[min(hi, 2)])):
                col = V[:, :, src].clone()
                if rule == 2:
                    for k in comps:
                        col[k] = -col[k]
                V[:, :, dst] = col


def _ratio(a, b, ok):
    """a / b where ok, else 0, with no division by what is not ok (so that gradients stay finite)."""
    return torch.where(ok, a / torch.where(ok, b, torch.ones_like(b)), torch.zeros_like(a))


def _root(a):
    ok = a > 0.0
    return torch.where(ok, torch.sqrt(torch.where(ok, a, torch.ones_like(a))), torch.zeros_like(a))


def _prim(U, g):
    rho = U[0]
    u, v, w = U[1] / rho, U[2] / rho, U[3] / rho
    p = (g - 1.0) * (U[7] - 0.5 * rho * (u * u + v * v + w * w) - 0.5 * (U[4] ** 2 + U[5] ** 2 + U[6] ** 2))
    return [rho, u, v, w, U[4], U[5], U[6], p, U[8]]


def _cons(W, g):
    rho, u, v, w, bx, by, bz, p, psi = W
    e = p / (g - 1.0) + 0.5 * rho * (u * u + v * v + w * w) + 0.5 * (bx * bx + by * by + bz * bz)
    return [rho, rho * u, rho * v, rho * w, bx, by, bz, e, psi]


def _flux(U, W, ch):
    """Flux along the first direction (components 1 and 4 are the normal ones)."""
    rho, u, v, w, bx, by, bz, p, psi = W
    pt = p + 0.5 * (bx * bx + by * by + bz * bz)
    ub = u * bx + v * by + w * bz
    return [U[1], U[1] * u + pt - bx * bx, U[1] * v - bx * by, U[1] * w - bx * bz, psi, by * u - bx * v,
            bz * u - bx * w, (U[7] + pt) * u - bx * ub, ch * ch * bx]


def _fast(W, g, bn):
    a2, b2 = g * W[7] / W[0], (W[4] ** 2 + W[5] ** 2 + W[6] ** 2) / W[0]
    s = a2 + b2
    return _root(0.5 * (s + _root(s * s - 4.0 * a2 * bn * bn / W[0])))


def _usable(W):
    return torch.isfinite(W[0]) & torch.isfinite(W[7]) & (W[0] > 0.0) & (W[7] > 0.0)


def _sel(ok, a, b):
    return [torch.where(ok, x, y) for x, y in zip(a, b)]


def _hll(UL, WL, FL, UR, WR, FR, ch, g):
    cl, cr = _fast(WL, g, WL[4]), _fast(WR, g, WR[4])
    c = ch * torch.ones_like(cl)
    SL = torch.minimum(torch.minimum(WL[1] - cl, WR[1] - cr), -c)
    SR = torch.maximum(torch.maximum(WL[1] + cl, WR[1] + cr), c)
    wide = (SR - SL).abs() >= 1e-14
    F = [_ratio(SR * a - SL * b + SL * SR * (y - x), SR - SL, wide) for a, b, x, y in zip(FL, FR, UL, UR)]
    mean = [0.5 * (a + b) for a, b in zip(FL, FR)]
    F = _sel(SL >= 0.0, FL, _sel(SR <= 0.0, FR, _sel(wide, F, mean)))
    return _sel(_usable(WL) & _usable(WR), F, mean)


def _star_solver(UL, WL, FL, UR, WR, FR, ch, g, double):
    """HLLC (or HLLD, `double`) flux and where the solver stands."""
    cl, cr = _fast(WL, g, WL[4]), _fast(WR, g, WR[4])
    rl, ul, vl, wl, bl, btl, bwl, pl = WL[:8]
    rr, ur, vr, wr, br, btr, bwr, pr = WR[:8]
    SL, SR = torch.minimum(ul - cl, ur - cr), torch.maximum(ul + cl, ur + cr)
    ptl, ptr = pl + 0.5 * (bl**2 + btl**2 + bwl**2), pr + 0.5 * (br**2 + btr**2 + bwr**2)
    den = (SR - ur) * rr - (SL - ul) * rl
    stands = _usable(WL) & _usable(WR) & ((SR - SL).abs() >= 1e-14) & (den.abs() >= 1e-14)
    SM = _ratio((SR - ur) * rr * ur - (SL - ul) * rl * ul + ptl - ptr, den, stands)
    rls, rrs = _ratio(rl * (SL - ul), SL - SM, stands), _ratio(rr * (SR - ur), SR - SM, stands)
    outer = (SL >= 0.0) | (SR <= 0.0)
    stars = (rls > 0.0) & (rrs > 0.0) & torch.isfinite(rls) & torch.isfinite(rrs)
    stands = stands & (stars if double else (stars | outer))
    in_star = stands & ~outer & stars
    one = torch.ones_like(rls)
    rls, rrs = torch.where(in_star, rls, one), torch.where(in_star, rrs, one)
    psi = 0.5 * (WL[8] + WR[8]) - 0.5 * ch * (br - bl)
    star = ptl + rl * (SL - ul) * (SM - ul)

    def side(U, W, S, pt, rs):
        r, u, v, w, bn, bt, bw = W[:7]
        vs, ws, bts, bws, ps = v, w, bt, bw, star
        if double:
            d = r * (S - u) * (S - SM) - bn * bn
            ok = d.abs() >= 1e-14
            a, b = _ratio(bn * (SM - u), d, ok), _ratio(r * (S - u) ** 2 - bn * bn, d, ok)
            vs, ws = torch.where(ok, v - bt * a, v), torch.where(ok, w - bw * a, w)
            bts, bws = torch.where(ok, bt * b, bt), torch.where(ok, bw * b, bw)
        else:
            ps = pt + r * (S - u) * (SM - u)
        bu, bus = bn * u + bt * v + bw * w, bn * SM + bts * vs + bws * ws
        e = _ratio((S - u) * U[7] - pt * u + ps * SM + bn * (bus - bu), S - SM, in_star)
        return [rs, rs * SM, rs * vs, rs * ws, bn, bts, bws, e, psi], vs, ws, bus

    Ls, vls, wls, buls = side(UL, WL, SL, ptl, rls)
    Rs, vrs, wrs, burs = side(UR, WR, SR, ptr, rrs)
    FLs = [f + SL * (s - u) for f, s, u in zip(FL, Ls, UL)]
    FRs = [f + SR * (s - u) for f, s, u in zip(FR, Rs, UR)]
    if double:
        ql, qr = torch.sqrt(rls), torch.sqrt(rrs)
        sg = torch.where(bl >= 0.0, one, -one)
        d2 = ql + qr
        v2 = (ql * vls + qr * vrs + sg * (Rs[5] - Ls[5])) / d2
        w2 = (ql * wls + qr * wrs + sg * (Rs[6] - Ls[6])) / d2
        bt2 = (ql * Rs[5] + qr * Ls[5] + sg * ql * qr * (vrs - vls)) / d2
        bw2 = (ql * Rs[6] + qr * Ls[6] + sg * ql * qr * (wrs - wls)) / d2
        SLs, SRs = SM - bl.abs() / ql, SM + br.abs() / qr
        for F1, U1, W, S1, q, sgn, bus, rs in ((FLs, Ls, WL, SLs, ql, -sg, buls, rls), (FRs, Rs, WR, SRs, qr, sg, burs, rrs)):
            e2 = U1[7] + q * sgn * (W[4] * SM + bt2 * v2 + bw2 * w2 - bus)
            U2 = [rs, rs * SM, rs * v2, rs * w2, W[4], bt2, bw2, e2, psi]
            F2 = [f + S1 * (b - a) for f, a, b in zip(F1, U1, U2)]
            if F1 is FLs:
                FLs = _sel(S1 >= 0.0, F1, F2)
            else:
                FRs = _sel(S1 <= 0.0, F1, F2)
    F = _sel(SL >= 0.0, FL, _sel(SR <= 0.0, FR, _sel(SM >= 0.0, FLs, FRs)))
    return F, stands


def _force(UL, WL, FL, UR, WR, FR, ch, g):
    a = torch.maximum(torch.maximum(WL[1].abs() + _fast(WL, g, WL[4]), WR[1].abs() + _fast(WR, g, WR[4])),
                      ch * torch.ones_like(WL[1]))
    lf = [0.5 * (p + q) - 0.5 * a * (y - x) for p, q, x, y in zip(FL, FR, UL, UR)]
    Uri = [0.5 * (x + y) - 0.5 / a * (q - p) for p, q, x, y in zip(FL, FR, UL, UR)]
    Wri = _prim(Uri, g)
    F = _sel(_usable(Wri), [0.5 * (p + q) for p, q in zip(lf, _flux(Uri, Wri, ch))], lf)
    mean = [0.5 * (p + q) for p, q in zip(FL, FR)]
    return _sel(_usable(WL) & _usable(WR), F, mean)


def _riemann(UL, UR, ch, g, solver):
    WL, WR = _prim(UL, g), _prim(UR, g)
    FL, FR = _flux(UL, WL, ch), _flux(UR, WR, ch)
    hll = _hll(UL, WL, FL, UR, WR, FR, ch, g)
    if solver == "hll":
        return hll
    if solver == "force":
        F, stands = _force(UL, WL, FL, UR, WR, FR, ch, g), torch.ones_like(UL[0], dtype=torch.bool)
    else:
        F, stands = _star_solver(UL, WL, FL, UR, WR, FR, ch, g, solver == "hlld")
    fine = lambda f: torch.isfinite(f[0]) & torch.isfinite(f[7]) & torch.isfinite(f[4]) & torch.isfinite(f[8])  # noqa: E731
    own = fine(F)
    glm = torch.where(stands, own, fine(hll))
    F = _sel(stands & own, F, hll)
    bn = 0.5 * (UL[4] + UR[4]) - 0.5 / ch * (UR[8] - UL[8])
    F[4] = torch.where(glm, 0.5 * (UL[8] + UR[8]) - 0.5 * ch * (UR[4] - UL[4]), F[4])
    F[8] = torch.where(glm, ch * ch * bn, F[8])
    return F


def _sound(W):
    ok = (W[0] > 1e-12) & (W[7] > 1e-12)
    for k in range(9):
        ok = ok & torch.isfinite(W[k])
    return ok


def _sweep(rows, dtd, ch, g, solver, limiter):
    """New interior cells of `rows`: nine (lines, n + 4) tensors, the sweep along the last axis, normal component first."""
    W = _prim(rows, g)
    Wl, Wr = [], []
    for q in W:
        a, b = q[:, 1:-1] - q[:, :-2], q[:, 2:] - q[:, 1:-1]
        ok = a * b > 0.0
        if limiter == "vanleer":
            s = _ratio(2.0 * a * b, a + b, ok)
        else:
            s = torch.where(ok, torch.where(a > 0.0, torch.minimum(a, b), torch.maximum(a, b)), torch.zeros_like(a))
        Wl.append(q[:, 1:-1] - 0.5 * s)
        Wr.append(q[:, 1:-1] + 0.5 * s)
    Wc = [q[:, 1:-1] for q in W]
    Wl, Wr = _sel(_sound(Wl), Wl, Wc), _sel(_sound(Wr), Wr, Wc)
    Ul, Ur = _cons(Wl, g), _cons(Wr, g)
    d = [0.5 * dtd * (b - a) for a, b in zip(_flux(Ul, _prim(Ul, g), ch), _flux(Ur, _prim(Ur, g), ch))]
    Ul2, Ur2 = [u - x for u, x in zip(Ul, d)], [u - x for u, x in zip(Ur, d)]
    Ul, Ur = _sel(_sound(_prim(Ul2, g)), Ul2, Ul), _sel(_sound(_prim(Ur2, g)), Ur2, Ur)
    F = _riemann([u[:, :-1] for u in Ur], [u[:, 1:] for u in Ul], ch, g, solver)
    new = [u[:, NG:-NG] - dtd * (f[:, 1:] - f[:, :-1]) for u, f in zip(rows, F)]
    keep = ~(torch.isfinite(new[0]) & torch.isfinite(new[7]))
    return [torch.where(keep, u[:, NG:-NG], v) for u, v in zip(rows, new)]


def _padded(cells, bc):
    """Nine interior (ny, nx) tensors with their ghosts, as one (9, ny + 4, nx + 4) tensor, differentiably."""
    U = torch.stack(cells)
    if bc == (0, 0, 0, 0):
        U = torch.cat([U[:, :, -NG:], U, U[:, :, :NG]], 2)
        return torch.cat([U[:, -NG:], U, U[:, :NG]], 1)
    V = torch.zeros(9, U.shape[1] + 2 * NG, U.shape[2] + 2 * NG, dtype=U.dtype, device=U.device)
    V[:, NG:-NG, NG:-NG] = U
    _fill_ghosts(V, bc)
    return V


_TURN = (0, 2, 1, 3, 5, 4, 6, 7, 8)  # the fields with the second direction's components first


def _step(U, dt, ch, dx, dy, g, solver, limiter, bc):
    T = _padded(_sweep([q[NG:-NG] for q in U], dt / dx, ch, g, solver, limiter), bc)
    cols = _sweep([T[k][:, NG:-NG].t() for k in _TURN], dt / dy, ch, g, solver, limiter)
    cells = [cols[k].t() for k in _TURN]
    V = _padded(cells, bc)
    # psi is damped in the interior, after the ghosts are filled
    damp = torch.exp(-dt * ch / CR)
    return torch.cat([V[:8], torch.cat([V[8:, :NG], torch.cat(
        [V[8:, NG:-NG, :NG], V[8:, NG:-NG, NG:-NG] * damp, V[8:, NG:-NG, -NG:]], 2), V[8:, -NG:]], 1)], 0)


def _speed(U, g):
    W = _prim([q[NG:-NG, NG:-NG] for q in U], g)
    s = torch.maximum(W[1].abs() + _fast(W, g, W[4]), W[2].abs() + _fast(W, g, W[5]))
    return torch.where(_usable(W) & torch.isfinite(s), s, torch.zeros_like(s)).reshape(-1).max()


def _march(U, steps, cfl, dx, dy, g, solver, limiter, bc, each=None):
    ch = torch.zeros((), dtype=torch.float64, device=U.device)
    t, dt = ch, ch
    for _ in range(steps):
        m = _speed(U, g)
        ch = torch.where(m > ch, m, ch)
        dt = cfl * min(dx, dy) / ch
        U = (each or (lambda f, *a: f(*a)))(_step, U, dt, ch, dx, dy, g, solver, limiter, bc)
        t = t + dt
    return U, t, dt, ch


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        cells, times = [], []
        for m in _batch_members(case, seed):
            U = _orszag_tang(m["nx"], m["ny"], m["b0"], m["gamma"])
            U = U.to(torch.float32).to(torch.float64) if case["dtype"] == "f32" else U
            U, t, _, _ = _march(U, case["steps"], m["cfl"], 1.0 / m["nx"], 1.0 / m["ny"], m["gamma"], case["solver"],
                                case["limiter"], BCS["periodic"])
            cells.append(U.reshape(-1))
            times.append(float(t))
        return {"U": torch.cat(cells), "t": np.array(times)}
    if kind == "adjoint":
        from torch.utils.checkpoint import checkpoint

        n, g = case["n"], 5.0 / 3.0
        amp = torch.tensor(_amplitudes(seed), dtype=torch.float64, device=_device(), requires_grad=True)
        U = _orszag_tang(n, n, 1.0 / math.sqrt(4.0 * math.pi), g, amp)
        U, _, _, _ = _march(U, case["steps"], 0.4, 1.0 / n, 1.0 / n, g, case["solver"], case["limiter"],
                            BCS["periodic"], each=lambda f, *a: checkpoint(f, *a, use_reentrant=False))
        J = 0.5 * ((U[RHO, NG:-NG, NG:-NG] - torch.as_tensor(_target(n, seed), device=U.device)) ** 2).sum()
        J.backward()
        return {"J": np.float64(J.detach().item()), "grad": amp.grad.cpu().numpy()}
    U, t, dt, ch = _march(_initial(case, seed), case["steps"], case["cfl"], 1.0 / case["nx"], 1.0 / case["ny"],
                          GAMMA[case["flow"]], case["solver"], case["limiter"], BCS[case["bc"]])
    if kind == "session":
        return {"aos": U.permute(1, 2, 0).reshape(-1, 9), "t": np.float64(t.item())}
    if kind == "dropin":
        return {"U": U, "t": np.float64(t.item())}
    return {"U": U, "t": np.float64(t.item()), "dt": np.float64(dt.item()), "ch": np.float64(ch.item())}
