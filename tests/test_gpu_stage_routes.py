"""Which stage kernel runs and what h3c_kernel_info says of it, and the per-lane tile kernel on 256-cell tiles (the
route of grids beyond the halo tables' 2^29 cells, taken here by kernel 0 with the halo tables off) against the
per-cell kernel: ragged boxes, coarse/fine faces, supersonic states, persistent grids.  Both evaluate the same
F(l, r); the states agree to a few ulps (FP64: 1e-13 relative, FP32 face fluxes: 1e-5, as the other stage kernels)."""
import numpy as np
import pytest

import hom3_b200 as hb
from hom3_b200 import _ffi as F
from hom3_b200.solver import Condition
from test_gpu_split import TOL, _state, _tables

pytestmark = pytest.mark.gpu


def _solver(t, q, ti, precision, kernel, halo=1, blocks=0, flux=F.FLUX_AUSM):
    nd = t["x_center"].shape[0]
    s = hb.Solver(nd, F.EULER, flux, ti, precision, cfl=0.2, time_end=1e30)
    s.set_grid(t["neighbors"], t["x_center"], t["length"], t["bc_idx"], t["first_ghost"],
               [Condition(F.BC_EULER_NEUMANN)] * (2 * nd), t["subface_cells"])
    s.set_option(F.OPT_EULER_KERNEL, kernel)
    s.set_option(F.OPT_HALO_KERNEL, halo)
    s.set_persistent_blocks(blocks)
    s.set_state(q)
    s.reset_time()
    return s


@pytest.mark.parametrize("precision", [F.FP64, F.MIXED])
@pytest.mark.parametrize("dims,fine,ti,blocks", [
    ((17, 5), 0, F.EULER_FORWARD, 0), ((37, 23), 1, F.RUNGE_KUTTA_2, 2), ((16, 16), 0, F.SSPRK3, 0),
    ((17, 13, 1), 0, F.RUNGE_KUTTA_2, 0), ((9, 7, 5), 1, F.EULER_FORWARD, 1), ((20, 12, 9), 1, F.SSPRK3, 5)])
@pytest.mark.parametrize("mach", [0.5, 3.0])
def test_per_lane_kernel_equals_per_cell_kernel(dims, fine, ti, blocks, precision, mach):
    t = _tables(dims, fine)
    q = _state(t, mach)
    a = _solver(t, q, ti, precision, 0, halo=0, blocks=blocks)
    b = _solver(t, q, ti, precision, 2)
    assert a.kernel_info()["kernel"] == "lane" and b.kernel_info()["kernel"] == "cell"
    a.solve(2)
    b.solve(2)
    qa, qb = a.state()[:, :t["first_ghost"]], b.state()[:, :t["first_ghost"]]
    assert np.isfinite(qa).all()
    assert np.abs(qa - qb).max() <= TOL[precision] * np.abs(qb).max()
    assert abs(a.time() - b.time()) <= TOL[precision] * b.time()


@pytest.mark.parametrize("nd,precision,slots,smem", [(2, F.FP64, 256, 36864), (2, F.MIXED, 256, 20480),
                                                     (3, F.FP64, 384, 56320), (3, F.MIXED, 384, 30720)])
def test_the_split_kernel_reports_its_own_launch(nd, precision, slots, smem):
    """Rows: four thetas per slot, the extra row (3D: theta_E; FP32: p), a split pair per tile cell and direction and
    side and per halo slot."""
    t = _tables((24, 20, 11)[:nd], 1)
    s = _solver(t, _state(t, 0.5), F.RUNGE_KUTTA_2, precision, 1)
    size, extra = (4, 1) if precision == F.MIXED else (8, 0)
    extra += nd == 3
    assert smem == size * ((4 + extra) * (256 + slots) + 2 * (2 * nd * 256 + slots))
    info = s.kernel_info()
    assert info["kernel"] == "tile" and info["halo_slots"] == slots and info["smem_bytes"] == smem
    assert info["grid"] == info["tiles"] and info["blocks_per_sm"] == 0
    s.set_persistent_blocks(3)
    assert s.kernel_info()["grid"] == 3


@pytest.mark.parametrize("kernel,halo,flux,name", [
    (0, 1, F.FLUX_AUSM, "halo"), (0, 0, F.FLUX_AUSM, "lane"), (1, 1, F.FLUX_AUSM, "tile"), (1, 0, F.FLUX_AUSM, "tile"),
    (2, 1, F.FLUX_AUSM, "cell"), (3, 1, F.FLUX_AUSM, "warp"), (4, 1, F.FLUX_AUSM, "tile512"), (1, 1, F.FLUX_LLF, "llf_tile")])
def test_each_route_has_a_name_of_its_own(kernel, halo, flux, name):
    t = _tables((12, 10, 9))
    s = _solver(t, _state(t, 0.5), F.RUNGE_KUTTA_2, F.FP64, kernel, halo, flux=flux)
    info = s.kernel_info()
    assert info["kernel"] == name
    assert (info["halo_slots"] > 0) == (name in ("halo", "tile"))
    # one step, against the generic per-cell kernels (the LLF flux takes a random state out of the physical range;
    # both report that)
    g = _solver(t, _state(t, 0.5), F.RUNGE_KUTTA_2, F.FP64, kernel, halo, flux=flux)
    g.set_option(F.OPT_TILE_KERNEL, 0)
    assert g.kernel_info()["kernel"] == "per_cell"
    s.solve(1)
    g.solve(1)
    qs, qg = s.state()[:, :t["first_ghost"]], g.state()[:, :t["first_ghost"]]
    assert np.abs(qs - qg).max() <= TOL[F.FP64] * np.abs(qg).max()
    assert s.status() == g.status()
