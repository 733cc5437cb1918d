"""Measured cases of the timestep pipeline: what a program has the library do
through its public entry points, from the smallest calls to the largest.

Families (the "kind" of a case):
  advdiff    cup2d_adv_diff_noalloc on device buffers that the caller owns
             (torch tensors): latency-bound on a small grid, bandwidth-bound
             on a large one;
  poisson    the Poisson solver alone, as a host program's own
             PoissonSolver::solve: right-hand side in, pressure out, in the
             program's pinned buffers (FP64, or FP32 transforms);
  graph      whole steps replayed from the captured graph
             (Context.advance), then the velocity and the body states read:
             one frame of a simulation;
  operators  the reference's own loop, operator by operator, with dt and the
             body state read by the host every step (iterated and
             variable-density pressure included: they run only this way);
  ensemble   many small simulations advanced by one graph launch per step;
  adjoint    the gradient of the mean drag by the discrete adjoint.

The grids, bodies and parameters are those of the benchmark workloads and of
the tests.  Flows start as seeded vortices with seeded 1e-6 noise, so the
first pass already meets a developed field, and go on from pass to pass; the
iterated and variable-density cases start each pass from a saved state (their
iteration counts depend on the steps before).
"""
import ctypes
import math

import numpy as np
import torch

from cubismup_2d_b200 import Ensemble, Simulation, abi
from cubismup_2d_b200.synthetic import ensemble_configs, fish_length_ok, noise_field

BS = 32
STATE = ["center_x", "center_y", "orientation", "u", "v", "omega", "forcex", "forcey", "torque", "drag"]


def listed():
    return [
        # a coupled code's own advection step on a small grid: launches and latency
        {"name": "advdiff_256x128", "kind": "advdiff", "bx": 8, "by": 4},
        # ... on a ragged grid that fills the chip about once
        {"name": "advdiff_1184x608", "kind": "advdiff", "bx": 37, "by": 19},
        # ... on the large case's grid: memory bandwidth
        {"name": "advdiff_4096x2048", "kind": "advdiff", "bx": 128, "by": 64},
        # the solver as a plug-in, FP32 transforms, on a grid that is padded to a power of two
        {"name": "poisson_fp32_768x384", "kind": "poisson", "bx": 24, "by": 12, "solver": "freespace", "fp32": True},
        # the reference's driver loop on a small grid, dt and forces read every step
        {"name": "operators_disk_256x128", "kind": "operators", "bx": 8, "by": 4, "solver": "freespace",
         "body": "disk", "steps": 10},
        # the reference's default (cosine) solver, forced cylinder
        {"name": "disk_cosine_512x256", "kind": "graph", "bx": 16, "by": 8, "solver": "cosine", "body": "disk",
         "steps": 20},
        # periodic box
        {"name": "disk_periodic_1024x1024", "kind": "graph", "bx": 32, "by": 32, "solver": "periodic", "body": "disk",
         "steps": 10},
        # the flagship workload: a self-propelled swimmer
        {"name": "swimmer_1024x512", "kind": "graph", "bx": 32, "by": 16, "solver": "freespace",
         "body": "stefanfish", "steps": 20},
        # the large single-GPU workload: two swimmers in tandem
        {"name": "tandem_4096x2048", "kind": "graph", "bx": 128, "by": 64, "solver": "freespace", "body": "tandem",
         "steps": 10},
        # a design sweep: seeded members of mixed grids, bodies and Reynolds numbers
        {"name": "ensemble_16", "kind": "ensemble", "members": 16, "steps": 10},
        # gradient of a cylinder's mean drag
        {"name": "adjoint_disk_512x256", "kind": "adjoint", "bx": 16, "by": 8, "solver": "freespace", "steps": 20},
        # a falling disk heavier than the fluid: the variable-density pipeline
        {"name": "falling_disk_256x128", "kind": "operators", "bx": 8, "by": 4, "solver": "freespace",
         "body": "falling", "steps": 1},
    ]


def draw(rng):
    """One more case of the same families; sizes log-uniform, odd ones among them."""
    def blocks(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["advdiff", "advdiff", "poisson", "graph", "graph", "graph", "operators", "operators",
                       "ensemble", "adjoint"])
    if kind == "advdiff":
        return {"kind": kind, "bx": blocks(1, 128), "by": blocks(1, 64)}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(2, 16), "steps": rng.randint(4, 10)}
    if kind == "adjoint":
        bx = blocks(6, 20)
        return {"kind": kind, "bx": bx, "by": max(4, bx // 2), "solver": "freespace", "steps": rng.randint(8, 24)}
    body = rng.choice(["disk", "disk", "stefanfish", "carlingfish"])
    if kind == "operators":
        body = rng.choice([body, body, "iterated", "falling"])
    solver = rng.choice(["freespace", "freespace", "freespace", "cosine", "periodic"])
    bx = blocks(8, 24 if kind == "operators" else 64)
    by = max(4, min(64, int(round(bx * rng.uniform(0.4, 1.0)))))
    if solver != "freespace":                        # their grids are powers of two
        bx, by = 1 << (bx.bit_length() - 1), 1 << (by.bit_length() - 1)
    if kind == "poisson":
        return {"kind": kind, "bx": bx, "by": by, "solver": solver, "fp32": solver != "cosine" and rng.random() < 0.5}
    return {"kind": kind, "bx": bx, "by": by, "solver": solver, "body": body,
            "steps": 1 if body in ("iterated", "falling") else rng.randint(5, 20)}


# ---- set-up -------------------------------------------------------------------

def _bodies(case, seed):
    """The shapes of a case; the domain is 1 x by/bx (2 x 1 for the tandem)."""
    X, Y = _extents(case)
    m = min(X, Y)
    r = np.random.default_rng(seed)
    x, y = X * (0.35 + 0.1 * r.random()), Y * (0.45 + 0.1 * r.random())
    body = case.get("body", "disk")
    if body == "disk":
        return f"disk radius={0.1 * m:.17g} xpos={x:.17g} ypos={y:.17g} bForced=1 bFixed=1 xvel=0.2"
    if body == "iterated":
        return f"disk radius={0.1 * m:.17g} xpos={x:.17g} ypos={y:.17g}"
    if body == "falling":
        return f"disk radius={0.1 * m:.17g} xpos={x:.17g} ypos={y:.17g} rhoS=1.5"
    h = _spacing(case)
    L = 0.1 if body == "tandem" else min(0.4 * m, 200 * h)
    while not fish_length_ok(L, h):
        L *= 0.99
    if body == "tandem":
        return (f"stefanfish L={L:.17g} T=1 xpos={x:.17g} ypos={y:.17g}, "
                f"stefanfish L={L:.17g} T=1 xpos={x + 0.15:.17g} ypos={y:.17g} phi=0.5")
    return f"{body} L={L:.17g} T=1 xpos={x:.17g} ypos={y:.17g}"


def _extents(case):
    e = 2.0 if case.get("body") == "tandem" else 1.0
    n = max(case["bx"], case["by"])
    return e * case["bx"] / n, e * case["by"] / n


def _spacing(case):
    return _extents(case)[0] / (BS * case["bx"])


def _nu(case):
    return 0.02 * _spacing(case)                     # cell Reynolds number of about 10 at the bodies' speeds


def _argline(case, seed):
    more = " -precision fp32" if case.get("fp32") else ""
    if case.get("body") in ("iterated", "falling"):
        more += " -iterativePenalization 1 -gravity '0 -1'"
    return (f"-bpdx {case['bx']} -bpdy {case['by']} -extent {max(_extents(case)):.17g} -CFL 0.1 "
            f"-nu {_nu(case):.17g} -lambda 1e4 -poissonType {case['solver']} -muteAll 1{more} "
            f"-shapes '{_bodies(case, seed)}'")


def _vortices(nx, ny, h, seed):
    """Velocity of eight Gaussian vortices plus the 1e-6 noise, (2, ny, nx)."""
    r = np.random.default_rng([seed, nx, ny])
    x, y = (np.arange(nx) + 0.5) * h, (np.arange(ny) + 0.5) * h
    f = np.zeros((2, ny, nx))
    for _ in range(8):
        s = min(nx, ny) * h * r.uniform(0.05, 0.15)
        a = r.uniform(-0.1, 0.1)
        dx, dy = x - nx * h * r.uniform(0.1, 0.9), y - ny * h * r.uniform(0.1, 0.9)
        ex, ey = np.exp(-0.5 * (dx / s) ** 2), np.exp(-0.5 * (dy / s) ** 2)
        f[0] -= np.outer(a * dy / s * ey, ex)
        f[1] += np.outer(a * ey, dx / s * ex)
    for c in range(2):
        f[c] += noise_field(seed % 65536, c, ny, nx)
    return f


def _start(argline, seed, step=100):
    """An initialised context with a developed flow, past the dt ramp."""
    sim = Simulation(argline)
    sim.init()
    ctx = sim.ctx
    f = _vortices(ctx.nx, ctx.ny, ctx.h, seed)
    ctx.set("u", f[0])
    ctx.set("v", f[1])
    s = ctx.scalars()
    ctx.set_scalars(s["time"], s["dt"], step, s["uinfx"], s["uinfy"])
    return sim


def _pinned(ctx):
    return [torch.empty(ctx.ny, ctx.nx, dtype=torch.float64, pin_memory=True) for _ in range(2)]


def _pointer(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "advdiff":
        nx, ny = BS * case["bx"], BS * case["by"]
        h = 1.0 / max(nx, ny)
        f = torch.from_numpy(_vortices(nx, ny, h, seed)).cuda()
        return {"kind": kind, "lib": abi.lib(), "in": f, "out": torch.empty_like(f), "bx": case["bx"],
                "by": case["by"], "par": _advdiff_parameters(h)}
    if kind == "ensemble":
        sims = [_start(a, seed + 7 * k) for k, a in enumerate(ensemble_configs(case["members"], seed=3))]
        return {"kind": kind, "sims": sims, "ens": Ensemble(sims), "steps": case["steps"],
                "host": [_pinned(s.ctx) for s in sims]}
    sim = _start(_argline(case, seed), seed)
    ctx = sim.ctx
    state = {"kind": kind, "sim": sim, "ctx": ctx, "steps": case.get("steps"), "saved": None,
             "host": None if kind == "adjoint" else _pinned(ctx)}
    if kind == "poisson":
        state["host"][0].numpy()[:] = _source(ctx.nx, ctx.ny, seed)
    if case.get("body") in ("iterated", "falling"):
        state["saved"] = ctx.checkpoint(torch.empty(ctx.checkpoint_size(), dtype=torch.uint8, device="cuda"))
    return state


def _source(nx, ny, seed):
    """A right-hand side: the vorticity-like difference of the vortices."""
    f = _vortices(nx, ny, 1.0 / max(nx, ny), seed)
    return np.diff(f[1], axis=1, prepend=0.0) - np.diff(f[0], axis=0, prepend=0.0)


def _advdiff_parameters(h):
    """h, nu, dt, uinfx, uinfy: a frame that moves with a body at 0.2."""
    return h, 0.02 * h, 0.1 * h / 0.5, 0.2, 0.01


# ---- one pass -----------------------------------------------------------------

def _check(ctx, rc):
    if rc != abi.OK:
        raise abi.Cup2DError(rc, ctx.L.cup2d_last_error(ctx.h_).decode())


def _velocity(ctx, host):
    """The velocity planes, read into the program's own pinned buffers."""
    for name, t in zip("uv", host):
        _check(ctx, ctx.L.cup2d_get_field(ctx.h_, abi.FIELDS[name], _pointer(t)))
    return {"u": host[0], "v": host[1]}


def _shapes(ctx):
    out = []
    for k in range(ctx.nshapes):
        s = ctx.shape_state(k)
        out.append([getattr(s, n) for n in STATE])
    return np.array(out)


def run(state):
    kind = state["kind"]
    if kind == "advdiff":
        (u, v), (a, b) = state["in"], state["out"]
        rc = state["lib"].cup2d_adv_diff_noalloc(u.data_ptr(), v.data_ptr(), a.data_ptr(), b.data_ptr(), state["bx"],
                                                 state["by"], *state["par"], torch.cuda.current_stream().cuda_stream)
        if rc != abi.OK:
            raise abi.Cup2DError(rc, "cup2d_adv_diff_noalloc")
        return {"u": a, "v": b}
    if kind == "ensemble":
        state["ens"].advance(state["steps"])
        shapes = state["ens"].shape_states()
        keep = [abi.SHAPE_STATE_FIELDS.index(n) for n in STATE]
        return {"shapes": np.ascontiguousarray(shapes[:, keep]),
                "members": [_velocity(s.ctx, h) for s, h in zip(state["sims"], state["host"])]}
    ctx = state["ctx"]
    if kind == "adjoint":
        J, gu, gv, gb, dts, _ = ctx.adjoint(state["steps"], every=10, w_energy=0.0, w_force=(1.0, 0.0))
        return {"J": J, "grad_u": gu, "grad_v": gv, "grad_body": gb, "dt": dts}
    if kind == "poisson":
        b, p = state["host"]
        _check(ctx, ctx.L.cup2d_set_field(ctx.h_, abi.FIELDS["tmp"], _pointer(b)))
        ctx.poisson_solve("tmp", "pres")
        _check(ctx, ctx.L.cup2d_get_field(ctx.h_, abi.FIELDS["pres"], _pointer(p)))
        return {"p": p}
    if kind == "graph":
        ctx.advance(state["steps"])
        return {**_velocity(ctx, state["host"]), "shapes": _shapes(ctx)}
    forces = []
    if state["saved"] is not None:
        ctx.restore(state["saved"])
    for _ in range(state["steps"]):
        dt = state["sim"].calcMaxTimestep()
        for op in state["sim"].pipeline:
            op(dt)
        ctx.end_step()
        forces.append(_shapes(ctx))
    return {**_velocity(ctx, state["host"]), "shapes": np.stack(forces)}


# ---- what a pass cannot do without ----------------------------------------------

def _solve_work(nx, ny, solver, fp32):
    """(bytes, flops) of one Poisson solve: the right-hand side read, the
    half spectrum written, taken through the columns with the kernel, and
    read back, the pressure written; the transforms' 5 n log2 n."""
    mx, my = (2 * nx, 2 * ny) if solver != "periodic" else (nx, ny)
    rows = 2 * ny * 2.5 * mx * math.log2(mx)
    cols = (mx / 2 if solver != "cosine" else nx / 2) * 2 * 5 * my * math.log2(my)
    return nx * ny * (16 + 9 * (4 if fp32 else 8)), rows + cols


def _step_work(bx, by, solver):
    """... of one constant-density step: advDiff (u, v read and written), the
    right-hand side written, the solve, the correction (p, u, v read; u, v
    written)."""
    nx, ny = BS * bx, BS * by
    b, f = _solve_work(nx, ny, solver, False)
    return b + nx * ny * 80, f + nx * ny * 120


def work(case):
    kind = case["kind"]
    if kind == "advdiff":
        nc = BS * BS * case["bx"] * case["by"]
        return {"bytes": 32 * nc, "flops": 40 * nc}
    if kind == "ensemble":
        b = f = 0
        for line in ensemble_configs(case["members"], seed=3):
            t = line.split()
            x = _step_work(int(t[t.index("-bpdx") + 1]), int(t[t.index("-bpdy") + 1]), "freespace")
            b, f = b + x[0], f + x[1]
        return {"bytes": b * case["steps"], "flops": f * case["steps"]}
    if kind == "poisson":
        nx, ny = BS * case["bx"], BS * case["by"]
        b, f = _solve_work(nx, ny, case["solver"], case["fp32"])
        return {"bytes": b, "flops": f}
    b, f = _step_work(case["bx"], case["by"], case["solver"])
    n = case["steps"] * (2 if kind == "adjoint" else 1)       # forward and transposed steps
    if case.get("body") in ("iterated", "falling"):
        n *= 20                                               # pressure iterations, each about a step's work
    return {"bytes": b * n, "flops": f * n}


# ---- the same in plain numpy, 64 bits --------------------------------------------

EPS = np.finfo(np.float64).eps


def exact(case, seed):
    """advDiff of any size, the Poisson solve and whole steps with a forced
    disk, in numpy.  The swimmers' midline and rasterisation, the adjoint and
    the iterated pressure have no such short restatement: None."""
    if case["kind"] == "advdiff":
        nx, ny = BS * case["bx"], BS * case["by"]
        h, nu, dt, ux, uy = _advdiff_parameters(1.0 / max(nx, ny))
        u, v = _advdiff(*_vortices(nx, ny, h, seed), (ux, uy), dt, h, nu)
        return {"u": u, "v": v}
    if case["kind"] == "poisson":
        nx, ny = BS * case["bx"], BS * case["by"]
        h = 1.0 / max(nx, ny)
        return {"p": _solver(case["solver"], nx, ny, h)(_faded(_source(nx, ny, seed), _fade2(nx, ny, h, 0.01)))}
    if case["kind"] not in ("graph", "operators") or case["body"] != "disk":
        return None
    if BS * BS * case["bx"] * case["by"] * case["steps"] > 2e7:
        return None
    u, v = _disk_flow(case, seed)
    return {"u": u, "v": v, "shapes": None}


def _edge(a):
    return np.pad(a, 1, mode="edge")


def _advdiff(u, v, uinf, dt, h, nu):
    """Explicit Euler of central advection and 5-point diffusion with faded
    inflow ghosts, then the mean outflow taken from the boundary cells."""
    dfac, afac = (nu / h) * (dt / h), -0.5 * dt / h
    n = max(abs(uinf[0]), abs(uinf[1]), EPS)
    fade = [1 - (max(uinf[0], 0) / n) ** 2 / 100, 1 - (min(uinf[0], 0) / n) ** 2 / 100,
            1 - (max(uinf[1], 0) / n) ** 2 / 100, 1 - (min(uinf[1], 0) / n) ** 2 / 100]
    out = []
    for a in (u, v):
        A = _edge(a)
        A[:, 0] *= fade[0]
        A[:, -1] *= fade[1]
        A[0, :] *= fade[2]
        A[-1, :] *= fade[3]
        w, e, s, t = A[1:-1, :-2], A[1:-1, 2:], A[:-2, 1:-1], A[2:, 1:-1]
        out.append(a + (afac * ((u + uinf[0]) * (e - w) + (v + uinf[1]) * (t - s)) +
                        dfac * (e + t + w + s - 4 * a)))
    a, b = out
    c = (-a[:, 0].sum() + a[:, -1].sum() - b[0].sum() + b[-1].sum()) / (2 * sum(u.shape))
    a[:, 0] += c
    a[:, -1] -= c
    b[0] += c
    b[-1] -= c
    return a, b


def _disk_chi(X, Y, h, cx, cy, r):
    """Towers' characteristic function of a disk's signed distance, and the
    cells of the 32x32 blocks under its bounding box of r + 2h."""
    d = r - np.sqrt((X - cx) ** 2 + (Y - cy) ** 2)
    ny, nx = d.shape
    mask = np.zeros(d.shape, dtype=bool)
    for by in range(0, ny, BS):
        for bx in range(0, nx, BS):
            x0, x1, y0, y1 = X[0, bx], X[0, bx + BS - 1], Y[by, 0], Y[by + BS - 1, 0]
            if min(x1, cx + r + 2 * h) > max(x0, cx - r - 2 * h) and min(y1, cy + r + 2 * h) > max(y0, cy - r - 2 * h):
                mask[by:by + BS, bx:bx + BS] = True
    D = _edge(np.where(mask, np.maximum(-1.0, d), -1.0))
    own = _edge(np.where(mask, d, -1.0))
    ix, iy = np.arange(nx) % BS, np.arange(ny)[:, None] % BS
    e = np.where(ix == BS - 1, D[1:-1, 2:], own[1:-1, 2:])
    w = np.where(ix == 0, D[1:-1, :-2], own[1:-1, :-2])
    t = np.where(iy == BS - 1, D[2:, 1:-1], own[2:, 1:-1])
    s = np.where(iy == 0, D[:-2, 1:-1], own[:-2, 1:-1])
    up = lambda a: np.maximum(a, 0.0)  # noqa: E731
    gx, gy = (e - w) * (0.5 / h), (t - s) * (0.5 / h)
    ix, iy = (up(e) - up(w)) * (0.5 / h), (up(t) - up(s)) * (0.5 / h)
    g2 = gx * gx + gy * gy
    chi = np.where(np.abs(d) > 2 * h, np.where(d > 0, 1.0, 0.0), (ix * gx + iy * gy) / np.where(g2 < EPS, EPS, g2))
    return np.where(mask, chi, 0.0), mask


def _fade2(nx, ny, h, width):
    """The square of the edge fade: 1 at the domain's edge, 0 from `width` inwards."""
    x, y = h * (np.arange(nx) + 0.5), h * (np.arange(ny) + 0.5)
    d = [np.maximum(np.maximum(width - n * h + a, width - a), 0.0) / width for n, a in ((nx, x), (ny, y))]
    return np.minimum(np.maximum(d[0][None, :], d[1][:, None]), 1.0) ** 2


def _faded(b, f2):
    """The edge fade of a right-hand side and its mean correction."""
    q = b * f2
    c = q.sum() / max(q[q > 0].sum(), EPS) if q.sum() > 0 else q.sum() / max(-q[q < 0].sum(), EPS)
    return b * (1 - f2) + c * (np.maximum(q, 0.0) if c > 0 else -np.minimum(q, 0.0))


def _disk_flow(case, seed):
    nx, ny, h, nu = BS * case["bx"], BS * case["by"], _spacing(case), _nu(case)
    kv = dict(p.split("=") for p in _bodies(case, seed).split()[1:])
    cx, cy, r, us = float(kv["xpos"]), float(kv["ypos"]), float(kv["radius"]), -0.2
    x, y = h * (np.arange(nx) + 0.5), h * (np.arange(ny) + 0.5)
    X, Y = np.meshgrid(x, y)
    chi, mask = _disk_chi(X, Y, h, cx, cy, r)
    chi = np.where(chi > 0, chi, 0.0)
    C = _edge(chi)
    perim = (C[1:-1, 2:] - C[1:-1, :-2]) ** 2 + (C[2:, 1:-1] - C[:-2, 1:-1]) ** 2 > 0
    f2 = _fade2(nx, ny, h, 0.01 * max(_extents(case)))
    solve = _solver(case["solver"], nx, ny, h)
    u, v = _vortices(nx, ny, h, seed)
    uinf = (-us, 0.0)
    for _ in range(case["steps"]):
        top = max(np.abs(u + uinf[0]).max(), np.abs(v).max(), np.abs(u).max())
        dt = 0.1 * min(h / top, h * h / nu, h / abs(us))
        u, v = _advdiff(u, v, uinf, dt, h, nu)
        U, V = _edge(u), _edge(v)
        b = 0.5 * h / dt * ((U[1:-1, 2:] - U[1:-1, :-2]) + (V[2:, 1:-1] - V[:-2, 1:-1]))
        total = -(chi * b)[mask].sum()               # the body's source and its perimeter correction
        b = np.where(mask, b - chi * b, b)
        at = mask & perim
        if total > 0:
            b = np.where(at & (b > 0), b - total / max(b[at & (b > 0)].sum(), EPS) * b, b)
        else:
            b = np.where(at & (b < 0), b + total / max(-b[at & (b < 0)].sum(), EPS) * b, b)
        P = _edge(solve(_faded(b, f2)))
        u = u - 0.5 * dt / h * (P[1:-1, 2:] - P[1:-1, :-2])
        v = v - 0.5 * dt / h * (P[2:, 1:-1] - P[:-2, 1:-1])
        u, v = (1 - chi) * u + chi * us, (1 - chi) * v
    return u, v


def _solver(kind, nx, ny, h):
    """The Poisson solve of a right-hand side (times h^2), as a function."""
    if kind == "freespace":                          # convolution with ln(r) / 2 pi on the doubled grid
        i, j = np.arange(2 * nx), np.arange(2 * ny)
        rx, ry = np.minimum(i, 2 * nx - i), np.minimum(j, 2 * ny - j)
        R = np.sqrt((rx * rx)[None, :] + (ry * ry)[:, None].astype(float))
        R[0, 0] = 1.0
        G = np.log(h * R) / (2 * np.pi)
        G[0, 0] = (2 * np.log(h / np.sqrt(np.pi)) - 1) / (4 * np.pi)
        K = np.fft.rfft2(G).real

        def solve(b):
            p = np.zeros((2 * ny, 2 * nx))
            p[:ny, :nx] = b
            return np.fft.irfft2(np.fft.rfft2(p) * K, s=p.shape)[:ny, :nx]
    elif kind == "periodic":
        kx, ky = 2 * np.pi * np.fft.rfftfreq(nx), 2 * np.pi * np.fft.fftfreq(ny)
        k2 = (kx * kx)[None, :] + (ky * ky)[:, None]
        k2[0, 0] = np.inf

        def solve(b):
            return np.fft.irfft2(-np.fft.rfft2(b) / k2, s=b.shape)
    else:                                            # cosine: the blended finite-difference / spectral multiplier
        f32 = np.float32
        cx, cy = (np.cos(np.pi / n * 2.0 * np.arange(n)).astype(f32) for n in (nx, ny))
        fd = (f32(1) - cx[None, :] / f32(2) - cy[:, None] / f32(2)).astype(np.float64)
        kx, ky = (np.arange(nx) + 0.5) * (np.pi / nx), (np.arange(ny) + 0.5) * (np.pi / ny)
        M = -1 / (0.9 * fd + 0.1 * ((kx * kx)[None, :] + (ky * ky)[:, None]))
        M[0, 0] = 0

        def solve(b):
            return _cosine(_cosine(b, True) * M, False)
    return solve


def _cosine(a, forward):
    """DCT-II along both axes, or its inverse, by the FFT of the even extension."""
    for axis in (0, 1):
        a = np.swapaxes(a, 0, axis)
        n = a.shape[0]
        w = np.exp(-0.5j * np.pi * np.arange(n) / n)[:, None]
        if forward:
            a = (np.fft.fft(np.concatenate([a, a[::-1]]), axis=0)[:n] * w).real
        else:
            z = np.zeros((n + 1, a.shape[1]), dtype=complex)
            z[:n] = a * w.conj()
            a = np.fft.irfft(z, n=2 * n, axis=0)[:n]
        a = np.swapaxes(a, 0, axis)
    return a
