"""The work a program has this library do, as cases that can be timed and checked.

Every case starts a solver from an initial state that is already on the GPU,
advances it through the public calls a hom3 driver makes (set_state,
reset_time, solve / dt / cht_solve / adjoint, apply_bcs, state) and reads the
whole result back into a GPU tensor.  `exact` is the same step in plain torch
float64 on the same grid tables (the tables are the input of the calls).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import hom3_b200 as hb
from hom3_b200 import _ffi as F
from hom3_b200.solver import Condition, GridSpec, build_tables, edge, square
from hom3_b200.workloads import cht_setup, ensemble_member_tables, ensemble_members, rotation_velocity

_TI = {"fe": F.EULER_FORWARD, "rk2": F.RUNGE_KUTTA_2, "ssprk3": F.SSPRK3}
_FLUX = {"ausm": F.FLUX_AUSM, "llf": F.FLUX_LLF, "upwind": F.FLUX_UPWIND}
_PREC = {"fp64": F.FP64, "mixed": F.MIXED}
_STAGES = {"fe": 1, "rk2": 2, "ssprk3": 3}
_FOREVER = 1e30  # time_end: the runs are bounded by their step count


def listed():
    return [
        # the smallest call: hom3's own 2D Euler tests on a 64 x 64 grid, run by hom3's loop, which reads dt
        # after every step (launch and read-back latency is all there is)
        dict(name="euler2d_small_loop", kind="euler", nx=64, ny=64, nz=0, fine=0, flux="ausm", ti="fe", prec="fp64",
             steps=10, loop="dt"),
        # the headline: 3D Riemann problem on a 64^3 tree refined twice in a sphere (1,448,336 cells), RK2
        dict(name="euler3d_tree", kind="euler", nx=64, ny=64, nz=64, fine=2, flux="ausm", ti="rk2", prec="fp64",
             steps=10, loop="run"),
        # the same run with FP32 fluxes
        dict(name="euler3d_tree_mixed", kind="euler", nx=64, ny=64, nz=64, fine=2, flux="ausm", ti="rk2",
             prec="mixed", steps=10, loop="run"),
        # a ragged box without refinement, three-stage Runge-Kutta: no side a multiple of a tile
        dict(name="euler3d_box_ragged", kind="euler", nx=117, ny=75, nz=50, fine=0, flux="ausm", ti="ssprk3",
             prec="fp64", steps=10, loop="run"),
        # the second-order scheme: periodic isentropic vortex on 256 x 256, MUSCL, SSP-RK3
        dict(name="euler2d_muscl", kind="muscl", n=256, ti="ssprk3", prec="fp64", steps=30),
        # 3D Navier-Stokes Taylor-Green vortex, RK2
        dict(name="cns3d_tgv", kind="cns", nx=128, ny=128, nz=128, ti="rk2", prec="fp64", steps=4),
        # a coarser one with FP32 fluxes
        dict(name="cns3d_tgv_mixed", kind="cns", nx=64, ny=64, nz=64, ti="rk2", prec="mixed", steps=10),
        # conjugate heat transfer: a 512 x 128 channel over a 512 x 64 solid, coupled steps
        dict(name="cht_channel", kind="cht", level=9, fluid=128, solid=64, steps=48),
        # hom3's rotating disc, refined to 2048 x 2048
        dict(name="advection2d", kind="advection", n=2048, flux="llf", ti="fe", steps=10),
        # heat conduction in a 3D block between two plates
        dict(name="heat3d", kind="heat", nx=100, ny=100, nz=100, ti="fe", steps=20),
        # many small independent 2D grids of uneven size stepped together, FP32 fluxes
        dict(name="ensemble2d_mixed", kind="batch", count=24, nmax=512, ti="rk2", prec="mixed", steps=10),
        # gradient of a 10-step run with respect to its initial state, on a smaller tree
        dict(name="euler3d_adjoint", kind="adjoint", nx=32, ny=32, nz=32, fine=2, ti="rk2", steps=10),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["euler", "euler", "euler", "muscl", "cns", "cht", "advection", "heat", "batch", "adjoint"])
    steps = rng.randint(3, 12)
    ti = rng.choice(["fe", "rk2", "ssprk3"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "euler":
        flux = rng.choice(["ausm", "ausm", "ausm", "llf"])
        if flux == "llf":  # hom3's LLF flux grows in 2D and 3D: short runs only
            steps = 3
        loop = rng.choice(["run", "run", "dt"])
        if rng.random() < 0.5:
            return dict(kind="euler", nx=size(16, 800), ny=size(16, 800), nz=0, fine=rng.randint(0, 1), flux=flux,
                        ti=ti, prec=prec, steps=steps, loop=loop)
        return dict(kind="euler", nx=size(12, 100), ny=size(12, 100), nz=size(12, 100), fine=rng.randint(0, 1),
                    flux=flux, ti=ti, prec=prec, steps=min(steps, 6), loop=loop)
    if kind == "muscl":
        return dict(kind="muscl", n=size(48, 400), ti=ti, prec=prec, steps=steps)
    if kind == "cns":
        if rng.random() < 0.4:
            return dict(kind="cns", nx=size(24, 400), ny=size(24, 400), nz=0, ti=ti, prec=prec, steps=steps)
        return dict(kind="cns", nx=size(16, 110), ny=size(16, 110), nz=size(16, 110), ti=ti, prec=prec,
                    steps=min(steps, 4))
    if kind == "cht":
        return dict(kind="cht", level=rng.randint(6, 9), fluid=rng.randint(20, 60), solid=rng.randint(9, 40),
                    steps=8 * rng.randint(2, 5) + rng.randint(0, 7))
    if kind == "advection":
        return dict(kind="advection", n=size(64, 1500), flux=rng.choice(["llf", "upwind"]), ti=ti, steps=steps)
    if kind == "heat":
        return dict(kind="heat", nx=size(10, 100), ny=size(10, 100), nz=size(10, 100), ti=ti, steps=steps)
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(2, 20), nmax=rng.randint(60, 400), ti=rng.choice(["fe", "rk2"]),
                    prec=prec, steps=steps)
    return dict(kind="adjoint", nx=size(12, 40), ny=size(12, 40), nz=size(12, 40), fine=rng.randint(0, 1), ti=ti,
                steps=min(steps, 6))


# ---------------------------------------------------------------------------
# grids
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=3)
def _box(dims, side, fine):
    """Tables of a box of dims cells (its longest edge `side` long) with its low corner at the origin, refined
    `fine` levels in a sphere about its centre; conditions in the order -x, +x, -y, +y (, -z, +z)."""
    nd = len(dims)
    level = max(1, math.ceil(math.log2(max(dims))))
    h = side / max(dims)
    root = h * 2 ** level
    mid = [0.5 * n * h for n in dims]
    refine = [(mid, 0.25 * min(dims) * h, level + fine)] if fine else []
    spec = GridSpec(nd, [0.0] * nd, [root] * nd, level, refine=refine)
    if all(n == 2 ** level for n in dims):
        return build_tables(spec, spec.cube_boundaries(), device=True)
    eps = root * 1e-15
    geoms = []
    for d in range(nd):
        for at, sign in ((eps, 1.0), (dims[d] * h - eps, -1.0)):
            point, normal = [0.0] * nd, [0.0] * nd
            point[d], normal[d] = at, sign
            geoms.append(edge(point, normal))
    return build_tables(spec, geoms, square(mid, [n * h for n in dims]), 2, device=True)


@functools.lru_cache(maxsize=3)
def _wrap(dims, side):
    """The interior cell on the opposite face for every ghost of a uniform box (-1: none)."""
    t = _box(dims, side, 0)
    h = side / max(dims)
    nd, fg = len(dims), t["first_ghost"]
    ix = np.floor(t["x_center"] / h).astype(np.int64)
    key = np.zeros(t["ncells"], np.int64)
    for d in range(nd):
        key = key * dims[d] + ix[d] % dims[d]
    order = np.argsort(key[:fg])
    return order[np.searchsorted(key[:fg], key[fg:], sorter=order)]


@functools.lru_cache(maxsize=2)
def _members(count, nmax):
    return [(m, ensemble_member_tables(m)) for m in ensemble_members(count, seed=3, nmin=32, nmax=nmax)]


@functools.lru_cache(maxsize=2)
def _cht(level, fluid, solid):
    return cht_setup(level=level, side=4.0, fluid_rows=fluid, solid_rows=solid)


def _dims(case):
    return tuple(n for n in (case["nx"], case["ny"], case["nz"]) if n > 0)


_PI2 = 2 * math.pi


def _grid(case):
    """(tables, conditions, periodic partners or None) of a single-grid case."""
    k = case["kind"]
    if k in ("euler", "adjoint"):
        dims = _dims(case)
        return _box(dims, 1.0, case["fine"]), [Condition(F.BC_EULER_NEUMANN) for _ in range(2 * len(dims))], None
    if k == "muscl":
        dims = (case["n"], case["n"])
        return _box(dims, 10.0, 0), [Condition(F.BC_PERIODIC)] * 4, _wrap(dims, 10.0)
    if k == "cns":
        dims = _dims(case)
        if len(dims) == 3:
            return _box(dims, _PI2, 0), [Condition(F.BC_PERIODIC)] * 6, _wrap(dims, _PI2)
        fs = [0.2, 0.0, 1.0, 1.0 / 1.4]
        return _box(dims, 1.0, 0), [Condition(F.BC_CNS_INFLOW, fs), Condition(F.BC_CNS_OUTFLOW, fs),
                                    Condition(F.BC_CNS_ADIABATIC_NOSLIP), Condition(F.BC_CNS_ADIABATIC_SLIP)], None
    if k == "advection":
        return _box((case["n"], case["n"]), 1.0, 0), [Condition(F.BC_ADV_CHARACTERISTIC)] * 4, None
    dims = _dims(case)
    conds = [Condition(F.BC_HEAT_DIRICHLET, [1.0]), Condition(F.BC_HEAT_DIRICHLET, [0.5])]
    return _box(dims, 1.0, 0), conds + [Condition(F.BC_HEAT_NEUMANN, [0.0])] * (2 * len(dims) - 2), None


# ---------------------------------------------------------------------------
# initial states (on the GPU, from the seed)
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _waves(x, seed, side, n=8):
    """A smooth seeded field in [-1, 1]: n random Fourier modes."""
    rng = np.random.Generator(np.random.PCG64(seed))
    k = rng.integers(1, 5, size=(n, x.shape[0])) * (_PI2 / side)
    ph = rng.uniform(0, _PI2, n)
    f = torch.zeros_like(x[0])
    for m in range(n):
        arg = torch.full_like(f, float(ph[m]))
        for d in range(x.shape[0]):
            arg = arg + float(k[m, d]) * x[d]
        f = f + torch.sin(arg)
    return f / n


def _conserved(u, rho, p):
    ke = sum(v * v for v in u)
    return torch.stack([rho * v for v in u] + [rho, p / 0.4 + 0.5 * rho * ke])


def _vortex(x, cx, cy, beta):
    dx, dy = x[0] - cx, x[1] - cy
    e1 = torch.exp(1 - dx * dx - dy * dy)
    u = [1.0 - beta * e1 * dy / _PI2, 1.0 + beta * e1 * dx / _PI2]
    rho = (1 - 0.4 * beta ** 2 * e1 * e1 / (16 * 1.4 * math.pi ** 2)) ** 2.5
    return u, rho, rho ** 1.4


def _initial(case, t, seed):
    """State [nv][ncells] of a single-grid case; ghosts are zero (the conditions fill them)."""
    fg = t["first_ghost"]
    x = torch.as_tensor(t["x_center"][:, :fg], device=_device())
    k = case["kind"]
    if k in ("euler", "adjoint"):
        left = x[0] < 0.5 * case["nx"] / max(_dims(case))
        one = torch.ones_like(x[0])
        rho = torch.where(left, one, 0.125 * one) * (1 + 0.01 * _waves(x, seed, 1.0, 16))
        p = torch.where(left, one, 0.1 * one) * (1 + 0.01 * _waves(x, seed + 1000, 1.0, 16))
        drift = [0.3, 0.1, 0.05] if k == "adjoint" else [0.0, 0.0, 0.0]  # off the flux's switch at rest
        q = _conserved([d * one for d in drift[:x.shape[0]]], rho, p)
    elif k == "muscl":
        rng = np.random.Generator(np.random.PCG64(seed))
        u, rho, p = _vortex(x, *rng.uniform(4.0, 6.0, 2), rng.uniform(2.0, 5.0))
        q = _conserved(u, rho, p)
    elif k == "cns" and x.shape[0] == 3:
        v0 = 0.1 * (1 + 0.05 * _waves(x, seed, _PI2))
        u = [v0 * torch.sin(x[0]) * torch.cos(x[1]) * torch.cos(x[2]),
             -v0 * torch.cos(x[0]) * torch.sin(x[1]) * torch.cos(x[2]), torch.zeros_like(x[0])]
        p = 1 / 1.4 + 0.01 / 16 * (torch.cos(2 * x[0]) + torch.cos(2 * x[1])) * (torch.cos(2 * x[2]) + 2)
        q = _conserved(u, 1.4 * p, p)
    elif k == "cns":
        w = 1 + 0.02 * _waves(x, seed, 1.0)
        q = _conserved([0.2 * w, 0.01 * _waves(x, seed + 1, 1.0)], w, w / 1.4)
    elif k == "advection":
        rng = np.random.Generator(np.random.PCG64(seed))
        cx, cy = rng.uniform(0.2, 0.3), rng.uniform(0.45, 0.55)
        inside = (x[0] - cx) ** 2 + (x[1] - cy) ** 2 < 0.08 ** 2
        q = torch.where(inside, torch.ones_like(x[0]), 0.1 * torch.ones_like(x[0]))[None]
    else:
        q = (0.75 + 0.2 * _waves(x, seed, 1.0))[None]
    full = torch.zeros((q.shape[0], t["ncells"]), dtype=torch.float64, device=x.device)
    full[:, :fg] = q
    return full


def _batch_initial(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    parts = []
    for m, t in _members(case["count"], case["nmax"]):
        fg = t["first_ghost"]
        x = torch.as_tensor(t["x_center"][:, :fg], device=_device())
        c, beta = rng.uniform(0, 1, 2), rng.uniform(1.0, 5.0)
        q = torch.zeros((4, t["ncells"]), dtype=torch.float64, device=x.device)
        q[:, :fg] = _conserved(*_vortex(x, c[0] * m["nx"] * m["h"], c[1] * m["ny"] * m["h"], beta))
        parts.append(q)
    return torch.cat(parts, dim=1)


def _cht_initial(case, seed):
    d = _cht(case["level"], case["fluid"], case["solid"])
    qf = torch.as_tensor(d["q_fluid"], device=_device()).clone()
    qs = torch.as_tensor(d["q_solid"], device=_device()).clone()
    for key, q in (("tables_fluid", qf), ("tables_solid", qs)):
        fg = d[key]["first_ghost"]
        x = torch.as_tensor(d[key]["x_center"][:, :fg], device=_device())
        if q is qs:
            q[0, :fg] = d["T_inf"] * (1 + 0.1 * _waves(x, seed, 4.0))
        else:  # density, momentum and energy together: the free stream's velocity and temperature
            q[:, :fg] *= 1 + 0.01 * _waves(x, seed + 1, 4.0)
    return qf, qs


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
_TGV = dict(cfl=0.5, cfl_viscous=0.4, Minfty=0.1, ReInfty=1600.0, Pr0=0.71)
_CHANNEL = dict(cfl=0.4, cfl_viscous=0.4, Minfty=0.2, ReInfty=200.0, Pr0=0.72)
_TR0 = 1.0


def _spec(case):
    """(physics, flux, reconstruction, properties) of a single-grid case."""
    k = case["kind"]
    if k == "muscl":
        return F.EULER, F.FLUX_AUSM, F.RECON_MUSCL, dict(cfl=0.5, limiter_k=1.0)
    if k == "cns":
        return F.CNS, F.FLUX_AUSM, F.RECON_NONE, _TGV if case["nz"] else _CHANNEL
    if k == "advection":
        return F.ADVECTION, _FLUX[case["flux"]], F.RECON_NONE, dict(cfl=0.5)
    if k == "heat":
        return F.HEAT, F.FLUX_AUSM, F.RECON_NONE, dict(cfl=0.3)
    return F.EULER, _FLUX[case.get("flux", "ausm")], F.RECON_NONE, dict(cfl=0.4)


def prepare(case, seed):
    if case["kind"] == "cht":
        d = _cht(case["level"], case["fluid"], case["solid"])
        cns = hb.Solver(2, F.CNS, time_end=_FOREVER, **d["props"])
        heat = hb.Solver(2, F.HEAT, time_end=_FOREVER, cfl=0.5)
        for s, w in ((cns, "fluid"), (heat, "solid")):
            t = d["tables_" + w]
            s.set_grid(t["neighbors"], t["x_center"], t["length"], t["bc_idx"], t["first_ghost"],
                       d["conditions_" + w])
        cns.set_partner(heat, d["partners_fluid"])
        heat.set_partner(cns, d["partners_solid"])
        qf, qs = _cht_initial(case, seed)
        return dict(case=case, cns=cns, heat=heat, qf=qf, qs=qs, of=torch.empty_like(qf), os=torch.empty_like(qs))
    if case["kind"] == "batch":
        tables = [t for _, t in _members(case["count"], case["nmax"])]
        s = hb.Batch(2, F.EULER, F.FLUX_AUSM, _TI[case["ti"]], _PREC[case["prec"]], cfl=0.4, time_end=_FOREVER)
        s.set_grids(tables, [[Condition(F.BC_EULER_NEUMANN) for _ in range(4)] for _ in tables])
        q = _batch_initial(case, seed)
        return dict(case=case, solver=s, q=q, out=torch.empty_like(q))
    t, conds, wrap = _grid(case)
    physics, flux, recon, props = _spec(case)
    s = hb.Solver(t["x_center"].shape[0], physics, flux, _TI[case["ti"]], _PREC[case.get("prec", "fp64")],
                  reconstruction=recon, time_end=_FOREVER, **props)
    s.set_grid(t["neighbors"], t["x_center"], t["length"], t["bc_idx"], t["first_ghost"], conds, t["subface_cells"])
    if wrap is not None:
        s.set_periodic(wrap)
    if physics == F.ADVECTION:
        s.set_velocity(rotation_velocity(t["x_center"]))
    q = _initial(case, t, seed)
    state = dict(case=case, solver=s, q=q, out=torch.empty_like(q))
    if case["kind"] == "adjoint":
        state["lam"] = _cotangent(t, q, seed)
    return state


def _cotangent(t, q, seed):
    x = torch.as_tensor(t["x_center"], device=q.device)
    return torch.stack([_waves(x, seed + 77 + v, 1.0) for v in range(q.shape[0])])


def run(state):
    case = state["case"]
    if case["kind"] == "cht":
        cns, heat = state["cns"], state["heat"]
        cns.set_state(state["qf"])
        heat.set_state(state["qs"])
        cns.reset_time()
        heat.reset_time()
        hb.cht_solve(_TR0, cns, heat, case["steps"])
        return dict(fluid=cns.state(out=state["of"])[:, :cns.first_ghost],
                    solid=heat.state(out=state["os"])[:, :heat.first_ghost], time=cns.time())
    s = state["solver"]
    s.set_state(state["q"])
    s.reset_time()
    if case["kind"] == "adjoint":
        grad, dts = s.adjoint(case["steps"], state["lam"], out=state["out"])
        return dict(grad=grad, dts=dts)
    if case.get("loop") == "dt":  # hom3's run loop: the driver looks at dt after every step
        for _ in range(case["steps"]):
            s.solve(1)
            s.dt()
    else:
        s.solve(case["steps"])
    s.apply_bcs()  # as hom3's output does: the ghosts of the state that is read
    q = s.state(out=state["out"])
    if case["kind"] == "batch":
        dt, time, _ = s.instances()
        return dict(q=q, dt=dt, time=time)
    return dict(q=q, time=s.time())


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _cells(case):
    k = case["kind"]
    if k == "cht":
        n = 2 ** case["level"]
        return n * case["fluid"], n * case["solid"]
    if k == "batch":
        return sum(t["first_ghost"] for _, t in _members(case["count"], case["nmax"]))
    return _grid(case)[0]["first_ghost"]


def work(case):
    """Bytes: the state in and out once per stage (the later stages also read the step's start state), the
    neighbour links and levels once per stage, the caller's state in and out once.  Flops: primitive variables
    once per cell, each face's flux once, the update; twice that and the reverse for the adjoint."""
    k, steps = case["kind"], case["steps"]
    if k == "cht":
        nf, ns = _cells(case)
        return {"bytes": steps * (nf * (64 + 17) + ns * (16 + 17)) + 64 * nf + 16 * ns,
                "flops": steps * (nf * (60 + 2 * 160) + ns * 12)}
    n = _cells(case)
    nd = 2 if k in ("batch", "muscl", "advection") or not case.get("nz", 0) else 3
    nv = 1 if k in ("advection", "heat") else nd + 2
    st = _STAGES[case["ti"]]
    cols = 2 * st + (st - 1)
    links = st * (8 * nd + 1) + (st * 8 * nd if k == "advection" else 0)
    per_cell = {"advection": 12 * nd, "heat": 4 * nd, "cns": 60 + nd * (45 + 70 * nd), "muscl": 120 + nd * 220}
    flops = st * per_cell.get(k, 40 + nd * 35)
    if k == "adjoint":
        return {"bytes": n * (steps * 3 * (8 * nv * cols + links) + 24 * nv), "flops": 4 * n * steps * flops}
    return {"bytes": n * (steps * (8 * nv * cols + links) + 16 * nv), "flops": n * steps * flops}


# ---------------------------------------------------------------------------
# the same steps in plain torch, float64
# ---------------------------------------------------------------------------
class _Ref:
    """hom3's finite-volume step on a table grid: first-order AUSM / LLF, MUSCL, Navier-Stokes, heat, advection."""

    def __init__(self, tables, conditions, physics, flux, recon, ti, props, wrap=None, partner=None, kappa=0.0):
        dev = _device()
        self.nd = tables["x_center"].shape[0]
        self.n, self.fg = tables["ncells"], tables["first_ghost"]
        self.physics, self.flux, self.recon, self.ti = physics, flux, recon, ti
        self.p = dict(gamma=1.4, cfl=0.2, cfl_viscous=0.4, T0=273.15, Sutherland0=110.4, Minfty=0.1, ReInfty=100.0,
                      Pr0=0.72, limiter_k=1.0)
        self.p.update(props)
        nb = torch.as_tensor(tables["neighbors"], device=dev)
        self.x = torch.as_tensor(tables["x_center"], device=dev)
        self.h = torch.as_tensor(tables["length"], device=dev)
        self.nbr = nb[:, :self.fg]
        sub = tables.get("subface_cells")
        self.sub = torch.as_tensor(sub, device=dev) if sub is not None else None
        gn = nb[:, self.fg:]
        valid = (gn >= 0) & (gn < self.n)
        self.pos = valid.to(torch.int64).argmax(0)  # side on which a ghost's boundary cell lies
        self.bcell = gn.gather(0, self.pos[None])[0]
        self.gbc = torch.as_tensor(tables["bc_idx"][self.fg:].astype(np.int64), device=dev)
        self.conds = conditions
        self.gdx = (self.x[:, self.bcell] - self.x[:, self.fg:]).square().sum(0).sqrt()
        self.wrap = torch.as_tensor(np.asarray(wrap), device=dev) if wrap is not None else None
        self.partner = torch.as_tensor(np.asarray(partner), device=dev) if partner is not None else None
        self.kappa = kappa
        self.vel = None
        if physics == F.ADVECTION:
            self.vel = torch.as_tensor(rotation_velocity(tables["x_center"]), device=dev)
        g, gm1 = self.p["gamma"], self.p["gamma"] - 1
        M = self.p["Minfty"]
        T = 1 / (1 + 0.5 * gm1 * M * M)
        self.S = self.p["Sutherland0"] / self.p["T0"]
        mu = T ** 1.5 * (1 + self.S) / (T + self.S)
        self.Re0 = self.p["ReInfty"] * mu / (T ** (1 / gm1) * M * math.sqrt(T)) if physics == F.CNS else 1.0
        self.gamma, self.gm1 = g, gm1

    # -- primitive variables --
    def prim(self, q):
        nd = self.nd
        rho = q[nd]
        u = [q[d] / rho for d in range(nd)]
        p = self.gm1 * (q[nd + 1] - 0.5 * rho * sum(v * v for v in u))
        return u, rho, p

    def temperature(self, q):
        if self.physics == F.HEAT:
            return q[0]
        _, rho, p = self.prim(q)
        return self.gamma * p / rho

    def to_conserved(self, u, rho, p):
        return torch.stack([rho * v for v in u] + [rho, p / self.gm1 + 0.5 * rho * sum(v * v for v in u)])

    # -- conditions: the state with its ghosts filled --
    def fill(self, q, other_T=None):
        qi = q[:, :self.fg]
        ghosts = torch.zeros((q.shape[0], self.n - self.fg), dtype=q.dtype, device=q.device)
        for i, c in enumerate(self.conds):
            at = torch.nonzero(self.gbc == i)[:, 0]
            b = self.bcell[at]
            qb = qi[:, b]
            v = list(c.values) + [0.0] * 8
            if c.kind in (F.BC_EULER_NEUMANN, F.BC_HEAT_NEUMANN):
                g = qb - self.gdx[at] * torch.tensor(v[:q.shape[0]], dtype=q.dtype, device=q.device)[:, None]
            elif c.kind == F.BC_HEAT_DIRICHLET:
                g = 2 * v[0] - qb
            elif c.kind == F.BC_PERIODIC:
                g = qi[:, self.wrap[at]]
            elif c.kind == F.BC_ADV_CHARACTERISTIC:
                g = qb
            elif c.kind == F.BC_CPL_HEAT_CNS:
                Ts = (other_T[self.partner[at]] + self.kappa * qb[0]) / (1 + self.kappa)
                g = 2 * Ts[None] - qb
            else:
                u, rho, p = self.prim(qb)
                if c.kind == F.BC_CNS_INFLOW:
                    u, rho = [2 * v[d] - u[d] for d in range(self.nd)], 2 * v[self.nd] - rho
                elif c.kind == F.BC_CNS_OUTFLOW:
                    p = 2 * v[self.nd + 1] - p
                elif c.kind == F.BC_CNS_ADIABATIC_NOSLIP:
                    u = [-w for w in u]
                elif c.kind == F.BC_CNS_ADIABATIC_SLIP:
                    u = [torch.where(self.pos[at] // 2 == d, -u[d], u[d]) for d in range(self.nd)]
                elif c.kind == F.BC_CPL_CNS_HEAT:
                    Tf = self.gamma * p / rho
                    Ts = (Tf + self.kappa * other_T[self.partner[at]]) / (1 + self.kappa)
                    u, rho = [-w for w in u], 2 * (p * self.gamma / Ts) - rho
                else:
                    raise ValueError(c.kind)
                g = self.to_conserved(u, rho, p)
            ghosts = ghosts.index_copy(1, at, g)
        return torch.cat([qi, ghosts], dim=1)

    # -- fluxes of the faces between cells l and r (index tensors) along d --
    def ausm(self, L, Rt, d):
        (uL, rL, pL), (uR, rR, pR) = L, Rt
        aL, aR = torch.sqrt(self.gamma * pL / rL), torch.sqrt(self.gamma * pR / rR)
        ML, MR = uL[d] / aL, uR[d] / aR

        def m(s, M):
            return torch.where(M.abs() > 1, 0.5 * (M + s * M.abs()), s * 0.25 * (M + s) ** 2)

        def pr(s, M):
            sup = torch.where(s * M > 0, torch.ones_like(M), torch.zeros_like(M))
            return torch.where(M.abs() > 1, sup, 0.25 * (M + s) ** 2 * (2 - s * M))

        mi = m(1, ML) + m(-1, MR)
        pi = pr(1, ML) * pL + pr(-1, MR) * pR

        def theta(u, r, p, a):
            ke = sum(w * w for w in u)
            return torch.stack([r * w for w in u] + [r, p / self.gm1 + 0.5 * r * ke + p]) * a

        f = torch.where(mi >= 0, theta(uL, rL, pL, aL), theta(uR, rR, pR, aR)) * mi
        pres = torch.zeros_like(f)
        pres[d] = pi
        return f + pres

    def face(self, S, l, r, c, d, dt):
        q = S["q"]
        if self.physics == F.HEAT:
            return (q[:, l] - q[:, r]) / self.h[c]
        if self.physics == F.ADVECTION:
            ul, ur = self.vel[d, l], self.vel[d, r]
            if self.flux == F.FLUX_LLF:
                lam = torch.maximum(ul.abs(), ur.abs())
                return 0.5 * (q[:, l] * ul + q[:, r] * ur + lam * (q[:, l] - q[:, r]))
            f = ul * q[:, l]
            return torch.where(0.5 * (ul + ur) < 0, -f, f)
        u, rho, p = S["prim"]
        if self.recon == F.RECON_MUSCL:
            G = S["grad"]
            small = torch.where(self.h[r] < self.h[l], r, l)
            xf = self.x[:, small].clone()
            xf[d] = self.x[d, l] + 0.5 * self.h[l]
            w = torch.stack(list(u) + [rho, p])
            L = w[:, l] + sum(G[:, k, l] * (xf[k] - self.x[k, l]) for k in range(self.nd))
            R = w[:, r] + sum(G[:, k, r] * (xf[k] - self.x[k, r]) for k in range(self.nd))
            nd = self.nd
            ok = (L[nd] > 0) & (L[nd + 1] > 0) & (R[nd] > 0) & (R[nd + 1] > 0)
            L, R = torch.where(ok, L, w[:, l]), torch.where(ok, R, w[:, r])
            return self.ausm((L[:nd], L[nd], L[nd + 1]), (R[:nd], R[nd], R[nd + 1]), d)
        if self.flux == F.FLUX_LLF:
            def ef(i):
                f = torch.stack([q[k, i] * u[d][i] for k in range(self.nd)] + [q[d, i], u[d][i] * (q[-1, i] + p[i])])
                add = torch.zeros_like(f)
                add[d] = p[i]
                return f + add
            return 0.5 * (ef(l) + ef(r) + self.h[c] / dt * (q[:, l] - q[:, r]))
        f = self.ausm(([w[l] for w in u], rho[l], p[l]), ([w[r] for w in u], rho[r], p[r]), d)
        if self.physics == F.CNS:
            f = f + self.viscous(S, l, r, d)
        return f

    def viscous(self, S, l, r, d):
        q, sl, nd = S["q"], S["slope"], self.nd
        mean = 0.5 * (q[:, l] + q[:, r])
        rho = mean[nd]
        u = [mean[k] / rho for k in range(nd)]
        ke = sum(w * w for w in u)
        p = self.gm1 * (mean[nd + 1] - 0.5 * rho * ke)
        along = (q[:, r] - q[:, l]) / self.h[r]

        def g(v, k):
            return along[v] if k == d else 0.5 * (sl[k, v, l] + sl[k, v, r])

        gu = [[(g(c, k) * rho - g(nd, k) * mean[c]) / rho ** 2 for k in range(nd)] for c in range(nd)]
        pp = S["prim"][2]
        T = self.gamma * 0.5 * (pp[l] + pp[r]) / rho
        mu = T ** 1.5 * (1 + self.S) / (T + self.S)
        gke = g(nd, d) * ke + sum(2 * rho * u[k] * gu[k][d] for k in range(nd))
        gp = self.gm1 * (g(nd + 1, d) - 0.5 * gke)
        heat = -mu * self.gamma / (self.gm1 * self.p["Pr0"] * rho) * (gp - p / rho * g(nd, d))
        div = sum(gu[k][k] for k in range(nd)) * (2.0 / 3.0)
        tau = [-mu * (gu[d][k] + gu[k][d] - (div if k == d else 0.0)) for k in range(nd)]
        return torch.stack(tau + [torch.zeros_like(rho), sum(u[k] * tau[k] for k in range(nd)) + heat]) / self.Re0

    # -- per-stage data --
    def slopes(self, q):
        h2 = 2 * self.h[:self.fg]
        s = torch.stack([(q[:, self.nbr[2 * k + 1]] - q[:, self.nbr[2 * k]]) / h2 for k in range(self.nd)])
        src = self.bcell if self.wrap is None else self.wrap
        g = s[:, :, src]
        for i, c in enumerate(self.conds):
            if c.kind in (F.BC_CNS_ADIABATIC_NOSLIP, F.BC_CNS_ISOTHERMAL_NOSLIP, F.BC_CPL_CNS_HEAT):
                sign = torch.ones_like(g)
                for k in range(self.nd):
                    sign[k, :self.nd] = torch.where((self.gbc == i) & (self.pos // 2 != k), -1.0, 1.0)
                g = g * sign
        return torch.cat([s, g], dim=2)

    def gradients(self, S):
        nd, fg = self.nd, self.fg
        u, rho, p = S["prim"]
        w = torch.stack(list(u) + [rho, p])
        wc, xc = w[:, :fg], self.x[:, :fg]
        M = [[0.0] * nd for _ in range(nd)]
        b = [0.0] * nd
        hi, lo = wc, wc
        for pos in range(2 * nd):
            n = self.nbr[pos]
            dx = self.x[:, n] - xc
            wt = 1 / dx.square().sum(0)
            dw = w[:, n] - wc
            for i in range(nd):
                b[i] = b[i] + wt * dx[i] * dw
                for j in range(nd):
                    M[i][j] = M[i][j] + wt * dx[i] * dx[j]
            hi, lo = torch.maximum(hi, w[:, n]), torch.minimum(lo, w[:, n])
        A = torch.stack([torch.stack(r) for r in M]).permute(2, 0, 1)
        G = torch.linalg.solve(A[:, None], torch.stack(b).permute(2, 1, 0)[..., None])[..., 0].permute(1, 2, 0)
        e2 = (self.p["limiter_k"] * self.h[:fg]) ** 3
        psi = torch.ones_like(wc)
        for pos in range(2 * nd):
            n, d = self.nbr[pos], pos // 2
            small = torch.where(self.h[n] < self.h[:fg], n, torch.arange(fg, device=n.device))
            xf = self.x[:, small].clone()
            xf[d] = xc[d] + 0.5 * self.h[:fg] if pos % 2 else self.x[d, n] + 0.5 * self.h[n]
            d2 = sum(G[:, k] * (xf[k] - xc[k]) for k in range(nd))
            a = torch.where(d2 > 0, hi - wc, lo - wc)
            den = d2 * (a * a + 2 * d2 * d2 + a * d2 + e2)
            phi = ((a * a + e2) * d2 + 2 * d2 * d2 * a) / torch.where(d2 == 0, torch.ones_like(den), den)
            psi = torch.minimum(psi, torch.where(d2 == 0, torch.ones_like(phi), phi))
        lim = psi[:, None] * G
        ghost = torch.zeros(lim.shape[:2] + (self.n - fg,), dtype=lim.dtype, device=lim.device)
        if self.wrap is not None:
            ghost = lim[:, :, self.wrap]
        return torch.cat([lim, ghost], dim=2)

    # -- residual (sum of minus-side less plus-side fluxes) of a ghost-filled state --
    def residual(self, q, dt):
        S = {"q": q}
        if self.physics in (F.EULER, F.CNS):
            S["prim"] = self.prim(q)
        if self.physics == F.CNS:
            S["slope"] = self.slopes(q)
        if self.recon == F.RECON_MUSCL:
            S["grad"] = self.gradients(S)
        cells = torch.arange(self.fg, device=q.device)
        acc = 0.0
        for d in range(self.nd):
            for side in (0, 1):
                nb = self.nbr[2 * d + side]

                def flux(c, n):
                    return self.face(S, n, c, c, d, dt) if side == 0 else self.face(S, c, n, c, d, dt)

                f = flux(cells, nb.clamp(min=0))
                at = torch.nonzero(nb < 0)[:, 0] if self.sub is not None else cells[:0]
                if at.numel():
                    members = self.sub[:, -nb[at] - 2]
                    f = f.index_copy(1, at, sum(flux(at, m) for m in members) / members.shape[0])
                acc = acc + f if side == 0 else acc - f
        return acc

    def min_dt(self, q):
        q = q[:, :self.fg].detach()
        h = self.h[:self.fg]
        if self.physics == F.HEAT:
            return (self.p["cfl"] * 0.5 * h * h).min()
        if self.physics == F.ADVECTION:
            return (self.p["cfl"] * h / self.vel[:, :self.fg].abs().amax(0)).min()
        u, rho, p = self.prim(q)
        a = torch.sqrt(self.gamma * p / rho)
        dt = self.p["cfl"] * h / torch.stack([v.abs() + a for v in u]).amax(0)
        if self.physics == F.CNS:
            T = self.gamma * p / rho
            coeff = T ** 1.5 * (1 + self.S) / (T + self.S) / (rho * h)
            visc = torch.maximum(coeff / self.Re0, coeff / (self.Re0 * self.p["Pr0"] * self.gm1))
            dt = torch.minimum(dt, self.p["cfl_viscous"] * h / (2 * visc))
        return dt.min()

    def step(self, q, dt, other_T=None):
        """q: interior columns (ghost columns ignored); returns the next interior state."""
        k = dt / self.h[:self.fg]

        def stage(v):
            f = self.fill(v, other_T)
            return f[:, :self.fg] + k * self.residual(f, dt)

        q0 = q[:, :self.fg]
        q1 = stage(q0)
        if self.ti == "fe":
            return q1
        q2 = stage(q1)
        if self.ti == "rk2":
            return 0.5 * (q0 + q2)
        q2 = 0.75 * q0 + 0.25 * q2
        return q0 / 3 + 2.0 / 3.0 * stage(q2)


def _reference(case, t=None):
    if t is not None:  # one instance of a batch
        return _Ref(t, [Condition(F.BC_EULER_NEUMANN)] * 4, F.EULER, F.FLUX_AUSM, F.RECON_NONE, case["ti"],
                    dict(cfl=0.4))
    t, conds, wrap = _grid(case)
    physics, flux, recon, props = _spec(case)
    return _Ref(t, conds, physics, flux, recon, case["ti"], props, wrap)


def _advance(ref, q, steps):
    time, dt = 0.0, 0.0
    with torch.no_grad():
        for _ in range(steps):
            dt = ref.min_dt(q)
            q = ref.step(q, dt)
            time = time + dt
        return ref.fill(q), float(time), float(dt)


def exact(case, seed):
    if case["kind"] == "cht":
        return _exact_cht(case, seed)
    if case["kind"] == "batch":
        q0, parts, dts, times, at = _batch_initial(case, seed), [], [], [], 0
        for _, t in _members(case["count"], case["nmax"]):
            q, time, dt = _advance(_reference(case, t), q0[:, at:at + t["ncells"]], case["steps"])
            at += t["ncells"]
            parts.append(q)
            dts.append(dt)
            times.append(time)
        return dict(q=torch.cat(parts, dim=1), dt=np.array(dts), time=np.array(times))
    ref = _reference(case)
    t = _grid(case)[0]
    q0 = _initial(case, t, seed)
    if case["kind"] != "adjoint":
        q, time, _ = _advance(ref, q0, case["steps"])
        return dict(q=q, time=time)
    fg, dts = t["first_ghost"], []
    q = start = q0[:, :fg].clone().requires_grad_(True)
    states = [start]
    for _ in range(case["steps"]):  # forward: the states and time steps; each step is differentiated by itself below
        with torch.no_grad():
            dt = ref.min_dt(q)
            q = ref.step(q, dt)
        dts.append(dt)
        states.append(q)
    lam = _cotangent(t, q0, seed)[:, :fg]
    for q, dt in zip(reversed(states[:-1]), reversed(dts)):
        q = q.detach().requires_grad_(True)
        lam = torch.autograd.grad((ref.step(q, dt) * lam).sum(), q)[0]
    grad = torch.zeros_like(q0)
    grad[:, :fg] = lam
    return dict(grad=grad, dts=np.array([float(v) for v in dts]))


def _exact_cht(case, seed):
    d = _cht(case["level"], case["fluid"], case["solid"])
    kappa = d["conditions_fluid"][3].values[0]
    cns = _Ref(d["tables_fluid"], d["conditions_fluid"], F.CNS, F.FLUX_AUSM, F.RECON_NONE, "fe", d["props"],
               partner=d["partners_fluid"], kappa=kappa)
    heat = _Ref(d["tables_solid"], d["conditions_solid"], F.HEAT, F.FLUX_AUSM, F.RECON_NONE, "fe", dict(cfl=0.5),
                partner=d["partners_solid"], kappa=kappa)
    scale = _TR0 * cns.p["Pr0"] * cns.Re0
    qf, qs = _cht_initial(case, seed)
    qf, qs = qf[:, :cns.fg], qs[:, :heat.fg]
    time = 0.0
    with torch.no_grad():
        for _ in range(case["steps"]):
            dt = torch.minimum(cns.min_dt(qf), heat.min_dt(qs) / scale)
            qf = cns.step(qf, dt, qs[0])
            qs = heat.step(qs, dt * scale, cns.temperature(qf))
            time = time + dt
    return dict(fluid=qf, solid=qs, time=float(time))
