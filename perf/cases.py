"""The work that users of the framework have it do, as measurable cases.

Each case is one call (or one short chain of calls) through the public entry points: a time step of a solver
in its plain FP64 form or its mixed-precision form with captured steps, a step whose state comes from and
goes back to host memory, a batch step of several instances, the two linear-solve backends a host program
calls instead of its own, and the gradient of a step.  Sizes and physics are those of the repository's own
benchmark (the rising bubble), its ensemble, its test configurations and the reference's case files (static
droplet, shear droplet, Hysing bubble); every state gets a seeded interface (modes 2-8).

The step of a trajectory follows the one before it, so a state steps on each time it is run.  Time steps lie
below the solver's own stability limits, so trajectories stay bounded.
"""
import math

import numpy as np
import torch

import ding_nsch_core_solver_b200 as dn
from ding_nsch_core_solver_b200 import autograd, capi
from ding_nsch_core_solver_b200.ensemble import ShardedEnsemble, droplet_cfgs

OUTPUTS = ("c", "mu", "u", "v", "p")
RESTART = ("c", "c_prev", "c_prev2", "p", "p_prev", "u", "v", "u_prev", "v_prev", "e_prev", "hu_prev", "hv_prev")
GRADIENT_STATE = {"c": "c", "c_old": "c_prev", "e_prev": "e_prev", "u": "u", "v": "v", "p": "p",
                  "p_prev": "p_prev", "hu_prev": "hu_prev", "hv_prev": "hv_prev"}


# ---------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the static droplet of the reference's case files, periodic both ways: the smallest grid in use, where
        # launches and latencies count
        dict(name="droplet_64x64", form="step", setup="periodic", nx=64, ny=64, scheme="icpcg"),
        # the shear droplet between moving walls (periodic x), split pressure form
        dict(name="shear_128x128", form="step", setup="channel", nx=128, ny=128, scheme="split_icpcg"),
        # the Hysing bubble as a drop-in step: the host owns the state, so all restart fields go up before the
        # step and come back after it; variable-coefficient pressure operator
        dict(name="host_bubble_96x192", form="host_step", setup="box", nx=96, ny=192, scheme="icpcg"),
        # odd, ragged extents and the LDLT preconditioner
        dict(name="ragged_101x237", form="step", setup="box", nx=101, ny=237, scheme="ildlt_pcg"),
        # the benchmark's rising bubble in the plain form, and the same on a finer grid
        dict(name="bubble_192x384", form="step", setup="box", nx=192, ny=384, scheme="split_icpcg"),
        dict(name="bubble_512x1024", form="step", setup="box", nx=512, ny=1024, scheme="split_icpcg"),
        # the mixed-precision form with captured steps, at the benchmark's size and at the largest grid in use
        dict(name="mixed_192x384", form="mixed_step", setup="box", nx=192, ny=384, scheme="split_icpcg"),
        dict(name="mixed_1024x2048", form="mixed_step", setup="box", nx=1024, ny=2048, scheme="split_icpcg"),
        # the uneven droplet ensemble (mixed form, captured steps) in one batch step
        dict(name="ensemble_16", form="ensemble", count=16, pick=4),
        # a batch of plain instances sharing the device
        dict(name="batch_8x192x384", form="batch", setup="box", nx=192, ny=384, scheme="split_icpcg", count=8),
        # the backends a host program calls for its CH and pressure solves, host buffers in and out
        dict(name="backends_160x250", form="backends", setup="box", nx=160, ny=250, scheme="split_icpcg"),
        # the gradient of a whole step
        dict(name="gradient_96x192", form="gradient", setup="box", nx=96, ny=192, scheme="split_icpcg"),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges: any extents, odd ones among them."""
    form = rng.choice(("step", "step", "step", "mixed_step", "mixed_step", "host_step", "batch", "ensemble",
                       "backends", "gradient"))
    schemes = ("icpcg", "ildlt_pcg", "split_icpcg", "split_icpcg", "split_ildlt_pcg")
    if form == "ensemble":
        return dict(form=form, count=rng.randint(4, 16), pick=rng.randint(10, 10000))
    if form == "mixed_step":
        nx = 16 * _size(rng, 5, 48) if rng.random() < 0.75 else _size(rng, 80, 240)
        ny = 2 * nx if nx % 16 == 0 else nx + rng.randint(0, nx)
        return dict(form=form, setup="box", nx=nx, ny=ny, scheme="split_icpcg")
    if form == "step":
        setup = rng.choice(("box", "box", "channel", "periodic"))
        lo, hi = {"box": (40, 400), "channel": (48, 224), "periodic": (32, 96)}[setup]
        nx = _size(rng, lo, hi)
        ny = int(nx * rng.uniform(1.5, 2.2)) if setup == "box" else int(nx * rng.uniform(0.7, 1.4))
        return dict(form=form, setup=setup, nx=nx, ny=ny, scheme=rng.choice(schemes))
    nx = _size(rng, 48, 192)
    case = dict(form=form, setup="box", nx=nx, ny=int(nx * rng.uniform(1.5, 2.2)),
                scheme="split_icpcg" if form in ("backends", "gradient") else rng.choice(schemes))
    if form == "batch":
        case["count"] = rng.randint(2, 8)
    return case


# ---------------------------------------------------------------------------------------------------------
# configurations and states
# ---------------------------------------------------------------------------------------------------------
def _config(case, **more):
    nx, ny, setup = case["nx"], case["ny"], case["setup"]
    cfg = dict(name="case", mode="coupled", nx=nx, ny=ny, ghost=3, pressure_scheme=case["scheme"],
               poisson_iterations=50000, pressure_tolerance=1e-10, ch_inner_iterations=5000, ch_tolerance=1e-10,
               momentum_iterations=500, momentum_tolerance=1e-10, surface_tension_multiplier=1.0)
    if setup == "box":  # the rising bubble: no-slip bottom and top, free-slip sides, ratios 10
        cfg.update(lx=4.0, ly=8.0, periodic_x=False, periodic_y=False, v_bc_left_type="neumann", v_bc_left_value=0.0,
                   v_bc_right_type="neumann", v_bc_right_value=0.0, interface_center_x=2.0, interface_center_y=2.0,
                   interface_radius=1.0, re=12.374368670764582, ca=0.02020305007471719, cn=0.04, pe=150.0,
                   density_ratio=10.0, viscosity_ratio=10.0, body_force_y=-1.0, dt=5e-5)
    elif setup == "channel":  # the shear droplet: walls at +-2, periodic x
        cfg.update(lx=4.0, ly=4.0, periodic_x=True, periodic_y=False, top_wall_velocity_x=2.0,
                   bottom_wall_velocity_x=-2.0, interface_center_x=2.0, interface_center_y=2.0, interface_radius=1.0,
                   re=0.1, ca=0.45, cn=0.03, pe=150.0, density_ratio=1.0, viscosity_ratio=1.0, dt=1.2e-4)
    else:  # the static droplet, periodic both ways
        cfg.update(lx=1.0, ly=1.0, periodic_x=True, periodic_y=True, interface_center_x=0.5, interface_center_y=0.5,
                   interface_radius=0.16, re=50.0, ca=1.0, cn=0.02, pe=150.0, density_ratio=10.0,
                   viscosity_ratio=10.0, dt=1e-6)
    h = min(cfg["lx"] / nx, cfg["ly"] / ny)
    cfg["cn"] = max(cfg["cn"], h)
    # at most half of the capillary and explicit CH limits (populate_timestep_limits' formulas)
    cap = 0.5 * math.sqrt(cfg["re"] * cfg["ca"] * h ** 3 / max(1.0, cfg["density_ratio"]))
    chx = 0.25 * h * h * cfg["pe"] * cfg["cn"] / (6.0 * math.sqrt(2.0) * 0.25 * 0.5)
    cfg["dt"] = min(cfg["dt"], 0.5 * cap, 0.5 * chx)
    cfg.update(more)
    return cfg


def _interface(cfg, rng):
    """c of a drop of radius R(theta) = R (1 + sum_{k=2..8} a_k cos(k theta + phi_k)), a_k = 0.02 U(-1, 1)."""
    nx, ny = cfg["nx"], cfg["ny"]
    x = (np.arange(nx) + 0.5) * (cfg["lx"] / nx) - cfg["interface_center_x"]
    y = (np.arange(ny) + 0.5) * (cfg["ly"] / ny) - cfg["interface_center_y"]
    z = x[:, None] + 1j * y[None, :]
    r = np.abs(z)
    e = z / np.maximum(r, 1e-30)  # exp(i theta)
    R = np.full((nx, ny), 1.0)
    ek = e
    for _ in range(2, 9):
        ek = ek * e
        R += 0.02 * rng.uniform(-1, 1) * (ek * np.exp(1j * rng.uniform(0, 2 * np.pi))).real
    return 0.5 - 0.5 * np.tanh((r - cfg["interface_radius"] * R) / (2.0 * math.sqrt(2.0) * cfg["cn"]))


def _ghosted(a, g):
    return np.pad(a, g, mode="edge")


def _start(solver, cfg, rng):
    """The reference's own start (velocity profile, materials) with the seeded interface as its phase."""
    solver.initialize()
    c = _ghosted(_interface(cfg, rng), cfg["ghost"])
    for n in ("c", "c_prev", "c_prev2"):
        solver.set_field(n, c)
    solver.refresh_derived()
    solver.set_initial_mass(solver.compute_mass("c"))


class _DeviceField:
    """A solver's device field as an object that torch can look into; the solver lives as long as the views
    do (a tensor made from this object holds a reference to it)."""

    def __init__(self, solver, name):
        self.owner = solver
        self.__cuda_array_interface__ = {"shape": solver.field_shape(name), "typestr": "<f8", "version": 3,
                                         "data": (solver.device_ptr(name), False), "strides": None}


def _views(solver, names=OUTPUTS):
    """The interior of the solver's fields, in place on the device."""
    g = solver.ghost
    out = {}
    for n in names:
        t = torch.as_tensor(_DeviceField(solver, n), device="cuda")
        out[n] = t[g:t.shape[0] - g, g:t.shape[1] - g]
    return out


# ---------------------------------------------------------------------------------------------------------
# what a user's program has in hand, and one pass
# ---------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    form = case["form"]
    if form == "ensemble":
        # a quarter of the instances' own time steps: their limits are those of a droplet at rest
        cfgs = [dict(c, dt=0.25 * c["dt"]) for c in droplet_cfgs(case["count"], seed=case["pick"])]
        shard = ShardedEnsemble(cfgs, step_graph=True)
        shard.initialize()
        for m, cfg in zip(shard.members, cfgs):
            _start(m, cfg, rng)
        for k in range(3):  # the starting step, then the steps that record
            shard.step(k)
        # (mu is a function of c)
        return dict(form=form, shard=shard, k=3, out=[_views(m, ("c", "u", "v", "p")) for m in shard.members])
    if form == "batch":
        cfg = _config(case, device_share=case["count"])
        members = []
        for _ in range(case["count"]):
            members.append(dn.Solver(cfg))
            _start(members[-1], cfg, rng)
            members[-1].set_step_graph(True)
        for k in range(3):
            capi.step_batch(members, [k] * len(members))
        return dict(form=form, members=members, k=3, out=[_views(m) for m in members])
    if form == "backends":
        return _prepare_backends(case, rng)
    cfg = _config(case, **(dict(precision="mixed") if form == "mixed_step" else {}))
    solver = dn.Solver(cfg)
    _start(solver, cfg, rng)
    if form == "mixed_step":
        solver.set_step_graph(True)
    first = 3 if form == "mixed_step" else 1
    for k in range(first):
        solver.step(k)
    state = dict(form=form, solver=solver, k=first)
    if form == "host_step":
        state["host"] = {n: torch.from_numpy(solver.get_field(n)).pin_memory().numpy() for n in RESTART}
    elif form == "gradient":
        g = cfg["ghost"]
        state["in"] = {}
        for k, n in GRADIENT_STATE.items():
            a = solver.get_field(n)
            state["in"][k] = torch.tensor(a[g:a.shape[0] - g, g:a.shape[1] - g].copy(), device="cuda")
        # cotangents of the next state: a smooth functional of c, u, v and p
        nx, ny = cfg["nx"], cfg["ny"]
        state["cot"] = {k: torch.from_numpy(_smooth(rng, *s)).cuda()
                        for k, s in (("c", (nx, ny)), ("u", (nx + 1, ny)), ("v", (nx, ny + 1)), ("p", (nx, ny)))}
    else:
        state["out"] = _views(solver)
    return state


def _smooth(rng, nx, ny):
    """A smooth seeded field: a few low modes and a little noise."""
    x, y = (np.arange(nx) + 0.5) / nx, (np.arange(ny) + 0.5) / ny
    f = 0.01 * rng.standard_normal((nx, ny))
    for _ in range(6):
        kx, ky = rng.integers(0, 5, size=2)
        f += rng.standard_normal() * np.cos(np.pi * kx * x + rng.uniform(0, 6.28))[:, None] * np.cos(
            np.pi * ky * y + rng.uniform(0, 6.28))[None, :]
    return f


def _backend_inputs(case, rng):
    cfg = _config(case)
    nx, ny, g, dt = cfg["nx"], cfg["ny"], cfg["ghost"], cfg["dt"]
    c = _interface(cfg, rng)
    alpha0 = 3.0 / (2.0 * dt)
    rhs = alpha0 * c + 20.0 * _smooth(rng, nx, ny)
    rho_mid = c + (1.0 - c) * cfg["density_ratio"]
    u, v = 0.1 * _smooth(rng, nx + 1, ny), 0.1 * _smooth(rng, nx, ny + 1)
    u[0] = u[-1] = 0.0
    v[:, 0] = v[:, -1] = 0.0
    p = _smooth(rng, nx, ny)
    p_prev = p + 0.01 * _smooth(rng, nx, ny)
    return cfg, alpha0, {k: _ghosted(a, g) for k, a in
                         dict(rhs=rhs, c=c, u=u, v=v, rho_mid=rho_mid, p=p, p_prev=p_prev).items()}


def _prepare_backends(case, rng):
    cfg, alpha0, host = _backend_inputs(case, rng)
    solver = dn.Solver(cfg)
    solver.initialize()
    return dict(form="backends", solver=solver, alpha0=alpha0, host=host)


def run(state):
    form = state["form"]
    if form == "backends":
        s, a, g = state["solver"], state["host"], state["solver"].ghost
        c = s.ch_linear_solve(a["rhs"], state["alpha0"], a["c"])[0]
        p = s.pressure_solve(1, a["u"], a["v"], a["rho_mid"], a["p"], a["p_prev"])[0]
        return {"c": c[g:-g, g:-g], "p": p[g:-g, g:-g]}
    if form == "gradient":
        st = {k: t.detach().requires_grad_(True) for k, t in state["in"].items()}
        new = autograd.full_step(state["solver"], state["k"], st)
        loss = sum((new[k] * w).sum() for k, w in state["cot"].items())
        names = ("c", "u", "v", "p")
        grads = torch.autograd.grad(loss, [st[n] for n in names])
        return {"new": {n: new[n].detach() for n in names}, "grad": dict(zip(names, grads))}
    k = state["k"]
    state["k"] = k + 1
    if form == "ensemble":
        state["shard"].step(k)
        return state["out"]
    if form == "batch":
        capi.step_batch(state["members"], [k] * len(state["members"]))
        return state["out"]
    solver = state["solver"]
    if form == "host_step":
        host = state["host"]
        for n, a in host.items():
            solver.set_field(n, a)
        solver.refresh_derived()
        solver.step(k)
        for n, a in host.items():
            solver.get_field(n, out=a)
        g = solver.ghost
        return {n: a[g:-g, g:-g] for n, a in host.items()}
    solver.step(k)
    return state["out"]


# ---------------------------------------------------------------------------------------------------------
# what the path cannot do without, and its values in 64 bits
# ---------------------------------------------------------------------------------------------------------
def work(case):
    """Each state field read and written once per pass; about 600 operations a cell for the stencils of a step,
    and 60 a cell for each of the solves' iterations, whose number grows with the extent (one per four cells
    of the longer side, in the plain form) or does not (multigrid)."""
    form = case["form"]
    if form == "ensemble":
        cells = sum(c["nx"] * c["ny"] for c in droplet_cfgs(case["count"], seed=case["pick"]))
        return {"bytes": 8.0 * 24 * cells, "flops": 3000.0 * cells}
    n = case["nx"] * case["ny"]
    its = max(case["nx"], case["ny"]) / 4.0
    if form == "backends":
        return {"bytes": 8.0 * 9 * n, "flops": (100.0 + 60.0 * its) * n}
    if form == "gradient":
        return {"bytes": 8.0 * 21 * n, "flops": 2 * (600.0 + 60.0 * its) * n}
    flops = 3000.0 if form == "mixed_step" else 600.0 + 60.0 * its
    return {"bytes": 8.0 * 24 * n * case.get("count", 1), "flops": flops * n * case.get("count", 1)}


def _cosines(n):
    """The orthonormal eigenvectors (rows) of the cell-centred Neumann Laplacian, and its eigenvalues h^2 L."""
    k, i = np.arange(n)[:, None], np.arange(n)[None, :]
    m = np.cos(np.pi * k * (i + 0.5) / n) * math.sqrt(2.0 / n)
    m[0] = math.sqrt(1.0 / n)
    return m, 2.0 * np.cos(np.pi * np.arange(n) / n) - 2.0


def exact(case, seed):
    """The backends' solutions by diagonalisation: both operators are polynomials of the constant Neumann
    Laplacian.  The other cases are whole non-linear steps; plain torch or numpy has no value for them short
    of the whole solver written once more."""
    if case["form"] != "backends":
        return None
    cfg, alpha0, host = _backend_inputs(case, np.random.default_rng(seed))
    g, nx, ny, dt = cfg["ghost"], cfg["nx"], cfg["ny"], cfg["dt"]
    dx, dy = cfg["lx"] / nx, cfg["ly"] / ny
    f = {k: a[g:a.shape[0] - g, g:a.shape[1] - g] for k, a in host.items()}
    mx, ex = _cosines(nx)
    my, ey = _cosines(ny)
    lap = ex[:, None] / dx ** 2 + ey[None, :] / dy ** 2
    # CH: alpha0 I - beta1 L + beta2 L^2
    beta1 = 3.0 * math.sqrt(2.0) / (16.0 * cfg["cn"]) / cfg["pe"]
    beta2 = 3.0 * math.sqrt(2.0) * cfg["cn"] / 4.0 / cfg["pe"]
    c = mx.T @ ((mx @ f["rhs"] @ my.T) / (alpha0 - beta1 * lap + beta2 * lap ** 2)) @ my
    # split pressure: -L p = -(div((1 - rho_ref / rho) grad(2 p - p_prev)) + rho_ref div(u) / dt), zero mean
    rho_ref = min(1.0, cfg["density_ratio"])
    pe, rm = 2.0 * f["p"] - f["p_prev"], f["rho_mid"]
    fx, fy = np.zeros((nx + 1, ny)), np.zeros((nx, ny + 1))
    fx[1:-1] = (1.0 - rho_ref / (0.5 * (rm[:-1] + rm[1:]))) * (pe[1:] - pe[:-1]) / dx
    fy[:, 1:-1] = (1.0 - rho_ref / (0.5 * (rm[:, :-1] + rm[:, 1:]))) * (pe[:, 1:] - pe[:, :-1]) / dy
    div = lambda a, b: (a[1:] - a[:-1]) / dx + (b[:, 1:] - b[:, :-1]) / dy  # noqa: E731
    b = mx @ -(div(fx, fy) + rho_ref * div(f["u"], f["v"]) / dt) @ my.T
    lap[0, 0] = -1.0
    b[0, 0] = 0.0
    return {"c": c, "p": mx.T @ (b / -lap) @ my}
