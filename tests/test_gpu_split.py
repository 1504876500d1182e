"""The default Euler/AUSM tile stage (flux splits computed once per cell) against the per-cell stage kernel,
where its dispatch and its tables can go wrong: ragged boxes (partial tiles), one-cell-thick sheets (a tile's
halo exceeds its shared-memory slots, so faces read entries from global memory), refined trees (coarse/fine
groups in tiles and halos), supersonic states (the general split), batches and persistent grids.

Both kernels evaluate the same F(l, r); products and sums are rounded in different places, so after a few steps
the states agree to a few ulps of the largest terms (FP64: 1e-13 relative, FP32 face fluxes: 1e-5, as for the
other stage kernels)."""
import numpy as np
import pytest

import hom3_b200 as hb
from hom3_b200 import _ffi as F
from hom3_b200.solver import Condition, GridSpec, build_tables, edge, square

pytestmark = pytest.mark.gpu
TOL = {F.FP64: 1e-13, F.MIXED: 1e-5}


def _tables(dims, fine=0):
    nd, level = len(dims), max(1, int(np.ceil(np.log2(max(dims)))))
    h = 1.0 / max(dims)
    root = h * 2 ** level
    mid = [0.5 * n * h for n in dims]
    refine = [(mid, 0.3 * max(dims) * h, level + fine)] if fine else []
    eps, geoms = root * 1e-15, []
    for d in range(nd):
        for at, sign in ((eps, 1.0), (dims[d] * h - eps, -1.0)):
            p, n = [0.0] * nd, [0.0] * nd
            p[d], n[d] = at, sign
            geoms.append(edge(p, n))
    return build_tables(GridSpec(nd, [0.0] * nd, [root] * nd, level, refine=refine), geoms,
                        square(mid, [n * h for n in dims]), 2)


def _state(t, mach, seed=0):
    nd, fg = t["x_center"].shape[0], t["first_ghost"]
    rng = np.random.default_rng(seed)
    rho, p = rng.uniform(0.5, 2.0, fg), rng.uniform(0.5, 2.0, fg)
    u = rng.uniform(-mach, mach, (nd, fg)) * np.sqrt(1.4 * p / rho)
    q = np.zeros((nd + 2, t["ncells"]))
    q[:nd, :fg], q[nd, :fg] = rho * u, rho
    q[nd + 1, :fg] = p / 0.4 + 0.5 * rho * (u * u).sum(0)
    return q


def _run(t, q, kernel, ti, precision, steps, blocks=0):
    nd = t["x_center"].shape[0]
    s = hb.Solver(nd, F.EULER, F.FLUX_AUSM, ti, precision, cfl=0.2, time_end=1e30)
    s.set_grid(t["neighbors"], t["x_center"], t["length"], t["bc_idx"], t["first_ghost"],
               [Condition(F.BC_EULER_NEUMANN)] * (2 * nd), t["subface_cells"])
    s.set_option(F.OPT_EULER_KERNEL, kernel)
    s.set_persistent_blocks(blocks)
    s.set_state(q)
    s.reset_time()
    s.solve(steps)
    return s.state()[:, :t["first_ghost"]], s.time(), s.kernel_info()


@pytest.mark.parametrize("precision", [F.FP64, F.MIXED])
@pytest.mark.parametrize("dims,fine,ti", [
    ((17, 5), 0, F.EULER_FORWARD), ((37, 23), 1, F.RUNGE_KUTTA_2), ((64, 48), 0, F.SSPRK3),
    ((17, 13, 1), 0, F.RUNGE_KUTTA_2), ((40, 33, 1), 0, F.SSPRK3), ((9, 7, 5), 1, F.EULER_FORWARD),
    ((16, 16, 16), 1, F.RUNGE_KUTTA_2), ((20, 12, 9), 1, F.SSPRK3), ((2, 2, 2), 0, F.RUNGE_KUTTA_2)])
@pytest.mark.parametrize("mach", [0.5, 3.0])
def test_split_kernel_equals_per_cell_kernel(dims, fine, ti, precision, mach):
    t = _tables(dims, fine)
    q = _state(t, mach)
    a, ta, info = _run(t, q, 1, ti, precision, 2)
    b, tb, _ = _run(t, q, 2, ti, precision, 2)
    assert info["kernel"] == "tile"
    assert np.isfinite(a).all()
    assert np.abs(a - b).max() <= TOL[precision] * np.abs(b).max()
    assert abs(ta - tb) <= TOL[precision] * tb
    if dims == (40, 33, 1):
        assert info["max_halo"] > 384  # more than the slots a tile keeps in shared memory


@pytest.mark.parametrize("blocks", [1, 5])
def test_split_kernel_persistent_grid(blocks):
    t = _tables((24, 20, 11), 1)
    q = _state(t, 1.5)
    a, ta, _ = _run(t, q, 1, F.RUNGE_KUTTA_2, F.FP64, 3)
    b, tb, _ = _run(t, q, 1, F.RUNGE_KUTTA_2, F.FP64, 3, blocks)
    assert ta == tb and np.array_equal(a, b)


def test_split_kernel_keeps_a_uniform_flow():
    """Equal states on both sides of every face, coarse/fine faces included: the fluxes cancel exactly."""
    t = _tables((16, 16, 16), 1)
    q = np.zeros((5, t["ncells"]))
    q[:, :t["first_ghost"]] = np.array([0.3, 0.2, -0.1, 1.0, 2.5])[:, None]
    a, _, _ = _run(t, q, 1, F.RUNGE_KUTTA_2, F.FP64, 3)
    assert np.array_equal(a, q[:, :t["first_ghost"]])
