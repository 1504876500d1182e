"""The two-cells-per-thread stage of heat and advection (grids of at least a wave of blocks) against numpy on the
grid tables: odd cell counts, pairs that are not neighbours (ragged boxes), every time integration and flux.

Tolerance: a step adds a dozen terms of the state's size, each rounded once: 1e-14 of the largest value per step
bounds both sides' rounding."""
import numpy as np
import pytest

import hom3_b200 as hb
from hom3_b200 import _ffi as F
from hom3_b200.solver import Condition, GridSpec, build_tables, edge, square

pytestmark = pytest.mark.gpu


def _box(dims):
    nd, level = len(dims), int(np.ceil(np.log2(max(dims))))
    h = 1.0 / max(dims)
    root, eps, geoms = h * 2 ** level, h * 2 ** level * 1e-15, []
    for d in range(nd):
        for at, sign in ((eps, 1.0), (dims[d] * h - eps, -1.0)):
            p, n = [0.0] * nd, [0.0] * nd
            p[d], n[d] = at, sign
            geoms.append(edge(p, n))
    return build_tables(GridSpec(nd, [0.0] * nd, [root] * nd, level), geoms,
                        square([0.5 * n * h for n in dims], [n * h for n in dims]), 2, device=True)


def _stage(t, q, k, flux, u):
    """q + k R(q) on the interior cells, zero-gradient ghosts (both physics' conditions here)."""
    fg, nb = t["first_ghost"], t["neighbors"]
    ghosts = np.arange(fg, t["ncells"])
    gn = nb[:, fg:]
    b = np.where((gn >= 0) & (gn < fg), gn, -1).max(0)
    q = q.copy()
    q[ghosts] = q[b]
    r = np.zeros(fg)
    for d in range(nb.shape[0] // 2):
        m, p = nb[2 * d, :fg], nb[2 * d + 1, :fg]

        def f(L, R):
            if flux == "heat":
                return (q[L] - q[R]) / t["length"][:fg]
            uL, uR = u[d][L], u[d][R]
            if flux == F.FLUX_LLF:
                return 0.5 * (q[L] * uL + q[R] * uR + np.maximum(abs(uL), abs(uR)) * (q[L] - q[R]))
            return np.where(0.5 * (uL + uR) < 0, -uL * q[L], uL * q[L])

        c = np.arange(fg)
        r += f(m, c) - f(c, p)
    return q[:fg] + k * r


@pytest.mark.parametrize("ti", [F.EULER_FORWARD, F.RUNGE_KUTTA_2, F.SSPRK3])
@pytest.mark.parametrize("dims,flux", [((513, 451), F.FLUX_LLF), ((513, 451), F.FLUX_UPWIND), ((512, 512), F.FLUX_LLF),
                                       ((67, 61, 59), "heat"), ((64, 64, 64), "heat"), ((67, 61, 59), F.FLUX_LLF)])
def test_scalar_stage_against_numpy(dims, flux, ti):
    t = _box(dims)
    fg, nd = t["first_ghost"], len(dims)
    assert fg >= 6 * 256 * 148
    rng = np.random.default_rng(3)
    q = np.zeros((1, t["ncells"]))
    q[0, :fg] = rng.random(fg)
    heat = flux == "heat"
    u = None if heat else rng.uniform(-1, 1, (nd, t["ncells"]))
    s = hb.Solver(nd, F.HEAT if heat else F.ADVECTION, F.FLUX_AUSM if heat else flux, ti, cfl=0.2, time_end=1e30)
    kind = F.BC_HEAT_NEUMANN if heat else F.BC_ADV_NEUMANN
    s.set_grid(t["neighbors"], t["x_center"], t["length"], t["bc_idx"], fg, [Condition(kind, [0.0])] * (2 * nd))
    if not heat:
        s.set_velocity(u)
    s.set_state(q)
    s.reset_time()
    h = t["length"][0]
    dt = 0.2 * 0.5 * h * h if heat else (0.2 * h / np.abs(u[:, :fg]).max(0)).min()
    assert abs(s.dt() - dt) <= 1e-15 * dt
    want, k = q[0].copy(), s.dt() / h
    full = lambda v: np.concatenate([v, np.zeros(t["ncells"] - fg)])  # noqa: E731
    s.solve(2)
    for _ in range(2):
        q0 = want[:fg]
        q1 = _stage(t, want, k, flux, u)
        if ti == F.EULER_FORWARD:
            out = q1
        else:
            q2 = _stage(t, full(q1), k, flux, u)
            if ti == F.RUNGE_KUTTA_2:
                out = 0.5 * (q0 + q2)
            else:
                q2 = 0.75 * q0 + 0.25 * q2
                out = q0 / 3 + 2 / 3 * _stage(t, full(q2), k, flux, u)
        want = full(out)
    got = s.state()[0, :fg]
    assert np.abs(got - want[:fg]).max() <= 2e-14 * max(1.0, np.abs(want).max())
    assert abs(s.min_dt() - dt) <= 1e-15 * dt
