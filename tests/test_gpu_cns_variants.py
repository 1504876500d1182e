"""Both variants of the CNS tile stage (brick grids with a border list, and the general one) and both ways its fused
time step is decided, against the per-cell kernel: ragged boxes whose tiles are no bricks and partial last tiles,
walls, slip and isothermal walls, periodic ragged boxes, every time integration, persistent grids, supersonic cells
(the splits' general branches), and a time step limited by viscosity, by convection, and by one in some warps and the
other in others.

Both kernels evaluate the same F(l, r) and round products and sums in different places: a step adds some fifty terms
of the state's size per cell, so two steps stay within 1e-13 of the largest value (FP64; FP32 face fluxes: 1e-5)."""
import numpy as np
import pytest

import hom3_b200 as hb
from hom3_b200 import _ffi as F
from hom3_b200.solver import Condition
from test_gpu_split import TOL, _state, _tables

pytestmark = pytest.mark.gpu
GAMMA, CFL, CFLV = 1.4, 0.2, 0.3
# dims -> whether every tile is a brick
GRIDS = {(32, 32): 1, (48, 32): 1, (37, 23): 0, (100, 60): 0, (16, 16, 16): 1, (24, 16, 12): 1, (20, 12, 9): 0,
         (33, 31, 29): 0, (9, 7, 5): 0}


def _mild(t, mach):
    """Densities and pressures within 0.8 .. 1.25: an isothermal wall's ghost takes 2 T_wall - T, so T stays below 2.6."""
    nd, fg = t["x_center"].shape[0], t["first_ghost"]
    rng = np.random.default_rng(0)
    rho, p = rng.uniform(0.8, 1.25, fg), rng.uniform(0.8, 1.25, fg)
    u = rng.uniform(-mach, mach, (nd, fg)) * np.sqrt(GAMMA * p / rho)
    q = np.zeros((nd + 2, t["ncells"]))
    q[:nd, :fg], q[nd, :fg] = rho * u, rho
    q[nd + 1, :fg] = p / (GAMMA - 1) + 0.5 * rho * (u * u).sum(0)
    return q


def _partners(t, dims):
    """For each ghost of a box the interior cell across the box."""
    fg, h = t["first_ghost"], 1.0 / max(dims)
    key = np.floor(t["x_center"] / h + 1e-9).astype(np.int64)
    cell = {tuple(k): i for i, k in enumerate(key[:, :fg].T)}
    return np.array([cell[tuple(np.mod(k, dims))] for k in key[:, fg:].T], np.int64)


def _run(t, dims, q, ti, precision, halo, re=50.0, periodic=False, blocks=0, steps=2):
    nd = len(dims)
    s = hb.Solver(nd, F.CNS, F.FLUX_AUSM, ti, precision, cfl=CFL, cfl_viscous=CFLV, ReInfty=re, gamma=GAMMA,
                  time_end=1e30)
    walls = [Condition(F.BC_CNS_ADIABATIC_NOSLIP), Condition(F.BC_CNS_ADIABATIC_SLIP),
             Condition(F.BC_CNS_ISOTHERMAL_NOSLIP, [1.3])]
    conds = [Condition(F.BC_PERIODIC)] * (2 * nd) if periodic else [walls[i % 3] for i in range(2 * nd)]
    s.set_grid(t["neighbors"], t["x_center"], t["length"], t["bc_idx"], t["first_ghost"], conds)
    if periodic:
        s.set_periodic(_partners(t, dims))
    s.set_option(F.OPT_HALO_KERNEL, halo)
    s.set_persistent_blocks(blocks)
    s.set_state(q)
    s.reset_time()
    s.solve(steps)
    return s.state()[:, :t["first_ghost"]], s.min_dt(), s.time(), s.kernel_info()


def _compare(t, dims, q, ti, precision, brick, **kw):
    blocks = kw.pop("blocks", 0)
    a, dta, ta, info = _run(t, dims, q, ti, precision, 1, blocks=blocks, **kw)
    b, dtb, tb, other = _run(t, dims, q, ti, precision, 0, **kw)
    assert info["kernel"] == "halo" and info["brick"] == brick and other["kernel"] == "per_cell"
    assert np.isfinite(a).all()
    assert np.abs(a - b).max() <= TOL[precision] * np.abs(b).max()
    assert abs(ta - tb) <= TOL[precision] * tb and abs(dta - dtb) <= TOL[precision] * dtb
    return info, tb


@pytest.mark.parametrize("precision", [F.FP64, F.MIXED])
@pytest.mark.parametrize("ti", [F.EULER_FORWARD, F.RUNGE_KUTTA_2, F.SSPRK3])
@pytest.mark.parametrize("dims", GRIDS)
def test_tile_equals_per_cell_on_boxes(dims, ti, precision):
    t = _tables(dims)
    _compare(t, dims, _mild(t, 0.3), ti, precision, GRIDS[dims])


@pytest.mark.parametrize("precision", [F.FP64, F.MIXED])
@pytest.mark.parametrize("dims", [(48, 32), (37, 23), (24, 16, 12), (20, 12, 9)])
@pytest.mark.parametrize("blocks", [1, 3, 0])
def test_periodic_boxes_and_persistent_grids(dims, blocks, precision):
    t = _tables(dims)
    info, _ = _compare(t, dims, _state(t, 0.5), F.RUNGE_KUTTA_2, precision, GRIDS[dims], periodic=True, blocks=blocks)
    assert not blocks or info["grid"] == blocks


@pytest.mark.parametrize("precision", [F.FP64, F.MIXED])
@pytest.mark.parametrize("dims", [(32, 32), (37, 23), (16, 16, 16), (20, 12, 9)])
def test_supersonic_cells(dims, precision):
    t = _tables(dims)
    _compare(t, dims, _state(t, 3.0), F.RUNGE_KUTTA_2, precision, GRIDS[dims], re=1e4, periodic=True)


def _convective_dt(t, q):
    """The least cfl h / max_d(|u_d| + a) over the cells."""
    nd, fg = t["x_center"].shape[0], t["first_ghost"]
    rho, u = q[nd, :fg], q[:nd, :fg] / q[nd, :fg]
    p = (GAMMA - 1) * (q[nd + 1, :fg] - 0.5 * rho * (u * u).sum(0))
    return float((CFL * t["length"][:fg] / (np.abs(u).max(0) + np.sqrt(GAMMA * p / rho))).min())


@pytest.mark.parametrize("precision", [F.FP64, F.MIXED])
@pytest.mark.parametrize("dims", [(48, 32), (37, 23), (16, 16, 16), (20, 12, 9)])
@pytest.mark.parametrize("limit", ["viscous", "both", "convective"])
def test_the_parts_that_decide_the_time_step(dims, limit, precision):
    t = _tables(dims)
    q = _mild(t, 0.3)
    dtc = _convective_dt(t, q)
    # the viscous limit is proportional to the Reynolds number: its value from a run it decides
    _, _, time, _ = _run(t, dims, q, F.EULER_FORWARD, F.FP64, 0, re=0.5, steps=1)
    assert time < 0.5 * dtc
    re = 0.5 * (0.25 if limit == "viscous" else 1.0 if limit == "both" else 8.0) * dtc / time
    _, tb = _compare(t, dims, q, F.EULER_FORWARD, precision, GRIDS[dims], re=re, steps=3)
    if limit == "viscous":
        assert tb < 0.9 * 3 * dtc
