"""Performance cases of the SISL and split-explicit cores.

A case is one call that a program built on this package makes: a time step, a
captured step of an ensemble, a gradient through steps, an implicit solve, a
semi-Lagrangian interpolation or a flux-form transport, on the grids and with
the solver settings of the package's own workloads (``suetes_b200.workloads``):
the mountain wave (dx 500 m, 20 km lid, dt 8 s), the dry warm bubble (dx 50 m,
dt 1 s; split-explicit dt 0.5 s with 12 acoustic steps).

Every input is a seeded smooth perturbation of the workload's state (cosine
modes of random wave number and phase), as a run meets it after its first
steps; the implicit solve takes normally distributed right-hand sides.

``exact`` restates the implicit solve, the interpolation and the transport in
plain float64 torch over flat terrain, where every coefficient of the operator
depends on the level and the map factor alone.
"""

import math
import random

import torch

from suetes_b200 import SemiLagrangianAdvector3D, StepGraph, DeviceState
from suetes_b200.adjoint import trajectory_vjp
from suetes_b200.core import fortran
from suetes_b200.workloads import box_energy_objective, mountain_wave, rising_bubble, split_bubble

F32, F64 = torch.float32, torch.float64
DTYPES = {"f32": F32, "f64": F64}
STATE = ("u", "v", "w", "eta_dot", "pi", "th_v", "rho")
SOLVER = ("u", "v", "w", "pi", "eta_dot")
DEVICE = "cuda"


def listed():
    return [
        # one step of a small limited run, launch- and latency-bound: a few thousand columns, odd sizes, and the
        # solver variant that leaves a cycle early
        {"name": "bubble-48x41x33-f32", "kind": "step", "flow": "bubble", "nx": 48, "ny": 41, "nz": 33, "dtype": "f32",
         "method": "incremental", "tol": 1e-7, "restart": 30},
        # the warm-bubble verification run: float64, a long restart, a tight tolerance
        {"name": "bubble-64x64x48-f64", "kind": "step", "flow": "bubble", "nx": 64, "ny": 64, "nz": 48, "dtype": "f64",
         "method": "batched", "tol": 1e-10, "restart": 100},
        # the production step: the float32 mountain wave with lateral relaxation, batched solves
        {"name": "wave-256x256x80-f32", "kind": "step", "flow": "wave", "nx": 256, "ny": 256, "nz": 80,
         "dtype": "f32", "method": "batched", "tol": 1e-7, "restart": 30},
        # its float64 reference run on a ragged grid
        {"name": "wave-150x131x60-f64", "kind": "step", "flow": "wave", "nx": 150, "ny": 131, "nz": 60, "dtype": "f64",
         "method": "batched", "tol": 1e-8, "restart": 30},
        # an ensemble of uneven bubbles advanced by one captured graph
        {"name": "ensemble-8-f32", "kind": "ensemble", "members": 8, "nx": 96, "ny": 96, "nz": 48, "dtype": "f32",
         "method": "incremental", "tol": 1e-7, "restart": 30},
        # sensitivity of the lee-box energy after two steps to the initial theta'
        {"name": "gradient-128x128x64-f32", "kind": "gradient", "nx": 128, "ny": 128, "nz": 64, "dtype": "f32",
         "method": "batched", "tol": 1e-7, "restart": 30, "steps": 2},
        # the same in float64 on a small odd grid, as a gradient check runs it
        {"name": "gradient-61x47x40-f64", "kind": "gradient", "nx": 61, "ny": 47, "nz": 40, "dtype": "f64",
         "method": "incremental", "tol": 1e-8, "restart": 30, "steps": 2},
        # the implicit solver called on its own, the microbenchmark's right-hand side and grid
        {"name": "solve-384x384x96-f32", "kind": "solve", "nx": 384, "ny": 384, "nz": 96, "dtype": "f32",
         "method": "batched", "tol": 1e-7, "restart": 30},
        # the split-explicit core's step, float32
        {"name": "split-256x256x64-f32", "kind": "split", "nx": 256, "ny": 256, "nz": 64, "dtype": "f32", "ns": 12},
        # the split-explicit step and its reverse sweep, float64, odd sizes
        {"name": "split-grad-109x90x50-f64", "kind": "split-gradient", "nx": 109, "ny": 90, "nz": 50, "dtype": "f64",
         "ns": 6},
        # departure points and tricubic interpolation of a field at them
        {"name": "advect-384x384x96-f32", "kind": "advect", "nx": 384, "ny": 384, "nz": 96, "dtype": "f32"},
        # flux-form transport of a tracer
        {"name": "transport-201x160x64-f64", "kind": "transport", "nx": 201, "ny": 160, "nz": 64, "dtype": "f64"},
    ]


def _size(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "ensemble", "gradient", "solve", "split", "split-gradient", "advect",
                       "transport"])
    dtype = rng.choice(["f32", "f32", "f64"])
    method = rng.choice(["batched", "incremental"])
    big = 256 if dtype == "f32" else 160
    case = {"kind": kind, "dtype": dtype}
    if kind == "step":
        case["flow"] = rng.choice(["bubble", "wave"])
        nz = _size(rng, 33, 80 if case["flow"] == "wave" else 64)
        case.update(nx=_size(rng, 40, big), ny=_size(rng, 40, big), nz=nz, method=method)
        case["tol"], case["restart"] = (1e-7, 30) if dtype == "f32" else (1e-8, rng.choice([30, 30, 50, 100]))
    elif kind == "ensemble":
        case.update(members=rng.choice([4, 6, 8]), nx=_size(rng, 48, 112), ny=_size(rng, 48, 112),
                    nz=_size(rng, 33, 56), dtype="f32", method=method, tol=1e-7, restart=30)
    elif kind == "gradient":
        big = 160 if dtype == "f32" else 96
        case.update(nx=_size(rng, 48, big), ny=_size(rng, 40, big), nz=_size(rng, 36, 64), method=method,
                    tol=1e-7 if dtype == "f32" else 1e-8, restart=30, steps=rng.choice([1, 2, 3]))
    elif kind == "solve":
        case.update(nx=_size(rng, 48, big), ny=_size(rng, 48, big), nz=_size(rng, 40, 80), method=method,
                    tol=1e-7 if dtype == "f32" else 1e-8, restart=rng.choice([20, 30, 40]))
    elif kind == "split":
        case.update(nx=_size(rng, 48, big), ny=_size(rng, 40, big), nz=_size(rng, 40, 64),
                    ns=rng.choice([4, 6, 12]))
    elif kind == "split-gradient":
        case.update(nx=_size(rng, 40, 112), ny=_size(rng, 40, 96), nz=_size(rng, 40, 60), ns=rng.choice([3, 6]))
    elif kind == "advect":
        case.update(nx=_size(rng, 48, 384), ny=_size(rng, 48, 384), nz=_size(rng, 40, 96))
    else:
        case.update(nx=_size(rng, 40, 256), ny=_size(rng, 40, 256), nz=_size(rng, 40, 80))
    return case


# ---------------------------------------------------------------------------
# seeded inputs
# ---------------------------------------------------------------------------
def _modes(rnd, shape, count=4, top=4):
    """Sum of ``count`` separable cosine modes of a grid's unit cube, in [-1, 1]."""
    total = torch.zeros(shape, dtype=F64, device=DEVICE)
    for _ in range(count):
        axes = []
        for n in shape:
            k, phase = rnd.randint(1, top), rnd.uniform(0.0, 2.0 * math.pi)
            at = torch.arange(n, dtype=F64, device=DEVICE) / n
            axes.append(torch.cos(2.0 * math.pi * k * at + phase))
        total += axes[0][:, None, None] * axes[1][None, :, None] * axes[2][None, None, :] / count
    return total


def _rigid(t):
    """Zero at the ground and at the lid."""
    t[:, :, 0] = 0.0
    t[:, :, -1] = 0.0
    return t


def _perturbed(state, rnd, wind, theta):
    """The workload's state some steps into its run: smooth winds and theta', history set."""
    out = dict(state)
    for k, amp in (("u", wind), ("v", wind), ("w", 0.2 * wind)):
        t = amp * _modes(rnd, tuple(state[k].shape))
        out[k] = fortran(state[k].to(F64) + (_rigid(t) if k == "w" else t), dtype=state[k].dtype)
    out["th_v"] = fortran(state["th_v"] + theta * _modes(rnd, tuple(state["th_v"].shape)), dtype=F64)
    out["pi"] = fortran(state["pi"], dtype=F64)
    if "u_prev" in state:
        for k in ("u", "v", "w", "eta_dot"):
            out[k + "_prev"] = out[k]
        out["is_first_step"] = 0.0
    return out


def _flow(case, rnd):
    """(stepper, state, bc) of a step or gradient case."""
    dtype = DTYPES[case["dtype"]]
    solver = {"solver_tol": case["tol"], "solver_restart": case["restart"], "solve_method": case["method"],
              "solver_maxiter": 30, "dtype": dtype, "device": DEVICE}
    if case.get("flow", "wave") == "wave":
        stepper, state, bc = mountain_wave(case["nx"], case["ny"], case["nz"], **solver)
        return stepper, _perturbed(state, rnd, 0.5, 0.3), bc
    stepper, state, bc = rising_bubble(case["nx"], case["ny"], case["nz"], amp=rnd.uniform(1.0, 3.0),
                                       center=(rnd.uniform(-300, 300), rnd.uniform(-300, 300), 1200.0), **solver)
    return stepper, _perturbed(state, rnd, 0.5, 0.1), bc


def _winds(case, rnd, grid):
    """Winds of Courant numbers up to about 1.5 and no flow through ground and lid."""
    dtype = DTYPES[case["dtype"]]
    u = 30.0 + 60.0 * _modes(rnd, grid.shape_of("u"))
    v = 60.0 * _modes(rnd, grid.shape_of("v"))
    e = _rigid(0.15 * _modes(rnd, grid.shape_of("w")))
    return {"u": fortran(u, dtype=dtype), "v": fortran(v, dtype=dtype), "eta_dot": fortran(e, dtype=dtype)}


def _flat(case, rnd):
    """(stepper, inputs) of a solve, advect or transport case: the mountain-wave physics over flat terrain."""
    dtype = DTYPES[case["dtype"]]
    stepper, _, _ = mountain_wave(case["nx"], case["ny"], case["nz"], dtype=dtype, device=DEVICE, flat=True,
                                  solver_tol=case.get("tol", 1e-7), solver_restart=case.get("restart", 30),
                                  solve_method=case.get("method", "batched"))
    grid = stepper.physics.grid
    if case["kind"] == "solve":
        gen = torch.Generator(device=DEVICE).manual_seed(rnd.randrange(1 << 30))
        data = {}
        for k, loc in zip(SOLVER, ("u", "v", "w", "m", "w")):
            t = torch.randn(grid.shape_of(loc), generator=gen, device=DEVICE, dtype=dtype)
            data[k] = fortran(_rigid(t) if loc == "w" else t)
        return stepper, data
    data = _winds(case, rnd, grid)
    data["field"] = fortran(1.0 + 0.5 * _modes(rnd, grid.shape_of("m"), count=8, top=12), dtype=dtype)
    return stepper, data


def prepare(case, seed):
    rnd = random.Random(seed)
    kind = case["kind"]
    dtype = DTYPES[case["dtype"]]
    if kind == "step":
        stepper, state, bc = _flow(case, rnd)
        return {"kind": kind, "stepper": stepper, "state": state, "bc": bc}
    if kind == "ensemble":
        members, outs = [], []
        for m in range(case["members"]):
            # members differ in extent by up to a third, as the package's ensemble workload has them
            one = dict(case, flow="bubble", nx=case["nx"] - 8 * (m % 4), ny=case["ny"] - 5 * (m % 3),
                       nz=case["nz"] - 3 * (m % 5))
            stepper, state, _ = _flow(one, rnd)
            ds = stepper.to_device_state(state, dtype)
            out = DeviceState(ds.core)
            members.append((stepper, ds, out, None))
            outs.append(out)
        return {"kind": kind, "graph": StepGraph(members), "outs": outs}
    if kind == "gradient":
        stepper, state, bc = _flow(case, rnd)
        half = 500.0 * case["nx"] / 2.0
        objective = box_energy_objective(stepper, case["steps"], x_box=(0.1 * half, 0.8 * half))
        return {"kind": kind, "stepper": stepper, "state": stepper.to_device_state(state, dtype), "bc": bc,
                "objective": objective, "steps": case["steps"]}
    if kind in ("split", "split-gradient"):
        stepper, state = split_bubble(case["nx"], case["ny"], case["nz"], amp=rnd.uniform(1.0, 3.0), dtype=dtype,
                                      device=DEVICE, ns=case["ns"], radius=800.0,
                                      center=(rnd.uniform(-300, 300), rnd.uniform(-300, 300), 1200.0))
        out = {"kind": kind, "stepper": stepper, "state": _perturbed(state, rnd, 0.5, 0.1)}
        if kind == "split-gradient":
            out["cotangents"] = {k: fortran(_modes(rnd, tuple(state[k].shape)), dtype=dtype)
                                 for k in ("u", "v", "w", "pi", "th_v")}
        return out
    stepper, data = _flat(case, rnd)
    physics = stepper.physics
    state = {"kind": kind, "data": data, "stepper": stepper, "bg": physics.precompute_bg(physics.bg_state_ref())}
    if kind == "advect":
        state["advector"] = SemiLagrangianAdvector3D(physics.grid, physics, stepper.dt)
    return state


def run(s):
    kind = s["kind"]
    if kind == "step":
        out = s["stepper"].step(s["state"], 0.0, None, s["bc"])
        return {k: out[k] for k in STATE}
    if kind == "ensemble":
        s["graph"].launch()
        return [{k: o.t[k] for k in ("u", "v", "w", "eta_dot", "pi_p", "th_p", "rho")} for o in s["outs"]]
    if kind == "gradient":
        value, grads = trajectory_vjp(s["stepper"], s["state"], s["steps"], s["objective"], bc_fn=s["bc"],
                                      wrt=("u", "v", "w", "pi_p", "th_p"))
        return {"value": value, **grads}
    if kind == "split":
        out = s["stepper"].step(dict(s["state"]), 0.0, None, None)
        return {k: out[k] for k in STATE}
    if kind == "split-gradient":
        out, grads = s["stepper"].step_vjp(dict(s["state"]), s["cotangents"])
        return {"state": {k: out[k] for k in STATE}, "grads": {k: grads[k] for k in ("u", "v", "w", "pi", "th_v")}}
    d = s["data"]
    if kind == "solve":
        return s["stepper"].implicit_solver.solve({k: d[k] for k in SOLVER}, s["bg"])
    if kind == "advect":
        coords = s["advector"].compute_departure_indices(d, loc="m")
        return {"coords": coords, "values": s["advector"].advect_cubic(d["field"], coords)}
    return s["stepper"].ffsl_advector.advect_3d_split(d["field"], d, s["bg"])


def work(case):
    """Each input and output field once; the floating operations of one pass over the path's formulas."""
    size = 4 if case["dtype"] == "f32" else 8
    cells = case["nx"] * case["ny"] * case["nz"]
    kind = case["kind"]
    if kind == "step":  # 11 state and history fields in, 7 out; two solves of a few dozen operator applications
        return {"bytes": 18 * cells * size, "flops": 2 * 30 * 250 * cells}
    if kind == "ensemble":
        return {"bytes": 18 * cells * size * case["members"], "flops": 2 * 30 * 250 * cells * case["members"]}
    if kind == "gradient":
        return {"bytes": (18 + 11) * cells * size * case["steps"], "flops": 4 * 30 * 250 * cells * case["steps"]}
    if kind == "solve":
        return {"bytes": 10 * cells * size, "flops": 60 * 250 * cells}
    if kind in ("split", "split-gradient"):
        both = 3 if kind == "split-gradient" else 1
        return {"bytes": (14 if both == 1 else 26) * cells * size, "flops": both * (3 * 300 + 2 * case["ns"] * 150) * cells}
    if kind == "advect":  # three winds and the field in, three coordinates and the values out
        return {"bytes": 8 * cells * size, "flops": 400 * cells}
    return {"bytes": 5 * cells * size, "flops": 60 * cells}


# ---------------------------------------------------------------------------
# float64 restatements over flat terrain
# ---------------------------------------------------------------------------
EARTH, OMEGA, LAT = 6371229.0, 7.2921e-5, math.radians(45.0)
GRAV, CP, RD, CVD, P0, N_BV = 9.81, 1004.0, 287.0, 717.0, 100000.0, 0.01
DX, LID, DT, ALPHA, PI_SCALE = 500.0, 20000.0, 8.0, 0.5, 1000.0


def _levels(nz):
    """Heights of mass and w levels of the stretched coordinate and the two thicknesses."""
    def z(at):
        return LID * (torch.exp(2.5 * at / LID) - 1.0) / (math.exp(2.5) - 1.0)
    faces = torch.arange(nz + 1, dtype=F64, device=DEVICE) * (LID / nz)
    zw, zm = z(faces).clamp(0.0, LID), z(0.5 * (faces[1:] + faces[:-1])).clamp(0.0, LID)
    ends = torch.cat([(2 * zm[0] - zm[1])[None], zm, (2 * zm[-1] - zm[-2])[None]])
    return zm, zw, torch.diff(zw), torch.diff(ends)


def _points(n):
    faces = torch.arange(n + 1, dtype=F64, device=DEVICE) * DX - n * DX / 2.0
    return 0.5 * (faces[1:] + faces[:-1]), faces


def _map_factor(x, y):
    return (1.0 + (x[:, None] ** 2 + y[None, :] ** 2) / (4.0 * EARTH ** 2))[:, :, None]


def _coriolis(x, y):
    rho = torch.sqrt(x[:, None] ** 2 + y[None, :] ** 2)
    rho = torch.where(rho == 0, torch.full_like(rho, 1e-15), rho)
    c = 2.0 * torch.atan(rho / (2.0 * EARTH))
    lat = torch.asin(torch.cos(c) * math.sin(LAT) + y[None, :] * torch.sin(c) * math.cos(LAT) / rho)
    return (2.0 * OMEGA * torch.sin(lat))[:, :, None]


def _mean(f, axis):
    n = f.shape[axis]
    return 0.5 * (f.narrow(axis, 0, n - 1) + f.narrow(axis, 1, n - 1))


def _edges(f, axis):
    return torch.cat([f.narrow(axis, 0, 1), f, f.narrow(axis, f.shape[axis] - 1, 1)], dim=axis)


def _to_faces(f, axis):
    return _edges(_mean(f, axis), axis)


class _Flat:
    """The implicit operator A and the column preconditioner M of the flat mountain-wave physics, scaled as the
    solver has them: pi by 1000, eta_dot by the w-level thickness."""

    def __init__(self, nx, ny, nz):
        zm, zw, self.dzm, self.dzw = _levels(nz)
        self.th = 300.0 * torch.exp(N_BV ** 2 / GRAV * zm)
        top = 1.0 + GRAV ** 2 / (CP * 300.0 * N_BV ** 2) * (math.exp(-N_BV ** 2 * float(zm[-1]) / GRAV) - 1.0)
        step = -GRAV * torch.diff(zm) / (CP * 0.5 * (self.th[1:] + self.th[:-1]))
        rev = torch.flip(torch.cumsum(torch.flip(step, [0]), 0), [0])
        pi = torch.cat([top - rev, torch.full((1,), top, dtype=F64, device=DEVICE)])
        rho = P0 / (RD * self.th) * pi ** (CVD / RD)
        self.cpi = RD / CVD * pi / (rho * self.th)
        self.flux = rho * self.th * self.dzm
        self.thw, self.rhow = _to_faces(self.th, 0), _to_faces(rho, 0)
        self.tau = torch.where(zw > 12000.0, 0.25 * (1.0 + torch.tanh(math.pi * (zw - 12000.0) / (LID - 12000.0)
                                                                      - math.pi / 2)), torch.zeros_like(zw))
        self.damp = 1.0 + DT * self.tau
        (xm, xu), (ym, yv) = _points(nx), _points(ny)
        self.m, self.mu, self.mv = _map_factor(xm, ym), _map_factor(xu, ym), _map_factor(xm, yv)
        self.fu, self.fv = _coriolis(xu, ym), _coriolis(xm, yv)
        self.shapes = [(nx + 1, ny, nz), (nx, ny + 1, nz), (nx, ny, nz + 1), (nx, ny, nz), (nx, ny, nz + 1)]
        p = ALPHA * DT * CP * self.thw / (self.dzw * self.damp) * self.rhow * self.thw
        p[0] = p[-1] = 0.0
        self.lpi = ALPHA * DT * self.cpi / self.dzm
        lower, upper = -self.lpi * p[:-1], -self.lpi * p[1:]
        column = torch.diag(1.0 - lower - upper) + torch.diag(lower[1:], -1) + torch.diag(upper[:-1], 1)
        self.column = torch.linalg.inv(column)

    def fields(self, x):
        return [t.reshape(s) for t, s in zip(torch.split(x, [math.prod(s) for s in self.shapes]), self.shapes)]

    @staticmethod
    def flat(fields):
        return torch.cat([t.reshape(-1) for t in fields])

    def apply(self, x):
        u, v, w, pi, eta = self.fields(x)
        pi, adt = pi / PI_SCALE, ALPHA * DT
        gx = _edges(torch.diff(pi, dim=0) / DX, 0) * self.mu
        gy = _edges(torch.diff(pi, dim=1) / DX, 1) * self.mv
        gz = _edges(torch.diff(pi, dim=2), 2) / self.dzw
        lu = u - adt * (-CP * self.th * gx + self.fu * _to_faces(_mean(v, 1), 0))
        lv = v - adt * (-CP * self.th * gy - self.fv * _to_faces(_mean(u, 0), 1))
        lw = self.damp * w + adt * CP * self.thw * gz
        fx, fy = u * self.flux / self.mu, v * self.flux / self.mv
        fz = _rigid(eta * self.rhow * self.thw)
        div = self.m * (torch.diff(fx, dim=0) * self.m + torch.diff(fy, dim=1) * self.m) / DX + torch.diff(fz, dim=2)
        lp = pi + adt * self.cpi / self.dzm * div
        lu = torch.cat([u[:1], lu[1:-1], u[-1:]], dim=0)
        lv = torch.cat([v[:, :1], lv[:, 1:-1], v[:, -1:]], dim=1)
        lw = torch.cat([w[:, :, :1], lw[:, :, 1:-1], w[:, :, -1:]], dim=2)
        # an end level holds the unscaled eta_dot, the levels between the scaled one
        le = torch.cat([eta[:, :, :1] / self.dzw[0], (ALPHA * (eta - w))[:, :, 1:-1], eta[:, :, -1:] / self.dzw[-1]], 2)
        return self.flat([lu, lv, lw, lp * PI_SCALE, le])

    def precondition(self, x):
        u, v, w, pi, eta = self.fields(x)
        wt = _rigid(self.rhow * self.thw * (w / self.damp + eta / ALPHA))
        po = (pi / PI_SCALE - self.lpi * torch.diff(wt, dim=2)) @ self.column.T
        gz = _edges(torch.diff(po, dim=2), 2) / self.dzw
        wo = (w - ALPHA * DT * CP * self.thw * gz) / self.damp
        wo = torch.cat([w[:, :, :1], wo[:, :, 1:-1], w[:, :, -1:]], dim=2)
        eo = eta / ALPHA + wo
        eo = torch.cat([eta[:, :, :1] * self.dzw[0], eo[:, :, 1:-1], eta[:, :, -1:] * self.dzw[-1]], dim=2)
        return self.flat([u, v, wo, po * PI_SCALE, eo])

    def solve(self, rhs, tol=1e-12, restart=60, cycles=12):
        """Left-preconditioned GMRES with twice-orthogonalised bases."""
        b = self.flat([rhs[0], rhs[1], rhs[2], rhs[3] * PI_SCALE, rhs[4]])
        x = b.clone()
        goal = tol * float(self.precondition(b).norm())
        for _ in range(cycles):
            r = self.precondition(b - self.apply(x))
            beta = float(r.norm())
            if beta <= goal:
                break
            basis = torch.empty((restart + 1, b.numel()), dtype=F64, device=b.device)
            hess = torch.zeros((restart + 1, restart), dtype=F64, device=b.device)
            basis[0] = r / beta
            used = restart
            for j in range(restart):
                w = self.precondition(self.apply(basis[j]))
                for _ in range(2):
                    h = basis[:j + 1] @ w
                    w -= basis[:j + 1].T @ h
                    hess[:j + 1, j] += h
                norm = w.norm()
                hess[j + 1, j] = norm
                if float(norm) <= 1e-14:
                    used = j + 1
                    break
                basis[j + 1] = w / norm
            first = torch.zeros((used + 1, 1), dtype=F64, device=b.device)
            first[0] = beta
            y = torch.linalg.lstsq(hess[:used + 1, :used], first).solution[:, 0]
            x = x + basis[:used].T @ y
            del basis
        u, v, w, pi, eta = self.fields(x)
        return {"u": u, "v": v, "w": w, "pi": pi / PI_SCALE, "eta_dot": eta / self.dzw}


def _linear(f, at):
    """Linear interpolation at index coordinates, indices clamped to the field."""
    lo = [torch.floor(c) for c in at]
    out = 0.0
    for corner in range(8):
        weight, index = 1.0, []
        for d in range(3):
            up = (corner >> (2 - d)) & 1
            frac = at[d] - lo[d]
            weight = weight * (frac if up else 1.0 - frac)
            index.append(torch.clamp(lo[d].long() + up, 0, f.shape[d] - 1))
        out = out + weight * f[tuple(index)]
    return out


def _cubic(f, at):
    """Catmull-Rom interpolation on the clamped 4x4x4 stencil."""
    weights, index = [], []
    for c, n in zip(at, f.shape):
        c = c.clamp(0, n - 1)
        base = torch.floor(c).long()
        t = c - base
        weights.append([-0.5 * t ** 3 + t ** 2 - 0.5 * t, 1.5 * t ** 3 - 2.5 * t ** 2 + 1.0,
                        -1.5 * t ** 3 + 2.0 * t ** 2 + 0.5 * t, 0.5 * t ** 3 - 0.5 * t ** 2])
        index.append([(base + q).clamp(0, n - 1) for q in (-1, 0, 1, 2)])
    out = torch.zeros_like(at[0])
    for a in range(4):
        for b in range(4):
            line = sum(weights[2][c] * f[index[0][a], index[1][b], index[2][c]] for c in range(4))
            out += weights[0][a] * weights[1][b] * line
    return out


def _exact_advect(case, d):
    (xm, _), (ym, _) = _points(case["nx"]), _points(case["ny"])
    m = _map_factor(xm, ym)
    vel = [_mean(d["u"], 0) * m / DX, _mean(d["v"], 1) * m / DX, _mean(d["eta_dot"], 2)]
    home = torch.meshgrid(*[torch.arange(n, dtype=F64, device=DEVICE) for n in vel[2].shape], indexing="ij")
    shift = [DT * q for q in vel]
    for _ in range(2):
        mid = [h - 0.5 * s for h, s in zip(home, shift)]
        shift = [DT * _linear(q, mid) for q in vel]
    coords = [h - s for h, s in zip(home, shift)]
    return {"coords": torch.stack(coords), "values": _cubic(d["field"], coords)}


def _swept(mass, courant):
    """One flux-form sweep along the last axis: mass between the departure points of the cells' faces."""
    n = mass.shape[-1]
    total = torch.nn.functional.pad(torch.cumsum(mass, dim=-1), (1, 0))
    at = (torch.arange(n + 1, dtype=F64, device=DEVICE) - courant).clamp(0.0, float(n))
    lo = torch.floor(at)
    part = at - lo
    low = torch.gather(total, -1, lo.long())
    high = torch.gather(total, -1, (lo.long() + 1).clamp(max=n))
    return torch.diff((1.0 - part) * low + part * high, dim=-1)


def _exact_transport(case, d):
    (xm, xu), (ym, yv) = _points(case["nx"]), _points(case["ny"])
    _, _, dzm, _ = _levels(case["nz"])
    volume = DX * DX / _map_factor(xm, ym) ** 2 * dzm
    mass = d["field"] * volume
    cx, cy = d["u"] * _map_factor(xu, ym) * DT / DX, d["v"] * _map_factor(xm, yv) * DT / DX
    mass = _swept(mass.permute(1, 2, 0), cx.permute(1, 2, 0)).permute(2, 0, 1)
    mass = _swept(mass.permute(0, 2, 1), cy.permute(0, 2, 1)).permute(0, 2, 1)
    return _swept(mass, d["eta_dot"] * DT) / volume


def exact(case, seed):
    """Steps and gradients have no value here: a restatement of the whole core would be a second package."""
    if case["kind"] not in ("solve", "advect", "transport"):
        return None
    _, data = _flat(case, random.Random(seed))
    d = {k: v.to(F64) for k, v in data.items()}
    if case["kind"] == "solve":
        return _Flat(case["nx"], case["ny"], case["nz"]).solve([d[k] for k in SOLVER])
    return _exact_advect(case, d) if case["kind"] == "advect" else _exact_transport(case, d)
