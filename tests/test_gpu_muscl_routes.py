"""2D MUSCL with two threads per cell (grids of less than two blocks of them per SM) and with one, on refined trees
(coarse/fine groups in both) against the oracle, with the tolerances of the other MUSCL parity tests: small, just
under the line, and above it."""
import pytest

import cases
from oracle import h3o
from test_gpu_parity import MUSCL, run_single

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ti", [h3o.EULER_FORWARD, h3o.RK2, h3o.SSPRK3])
@pytest.mark.parametrize("level,fine,threads", [(5, 6, 2), (7, 8, 2), (7, 9, 1)])
def test_muscl_2d_refined(level, fine, threads, ti):
    import torch
    w = h3o.World(2, [0, 0], [1, 1], level=level)
    w.refine_sphere([0.45, 0.55], 0.3, fine)
    o = w.add_solver(h3o.EULER, h3o.AUSM, ti, bcs=cases.neumann_cube(w), ic_kind=h3o.IC_SHOCK_TUBE,
                     ic=[0, 0, 0.5, 1.0, 0.0, 1.0, 0.125, 0.0, 0.1], time_end=1.0, cfl=0.4, **MUSCL)
    o.initialize()
    n = o.first_ghost
    assert (n < 256 * torch.cuda.get_device_properties(0).multi_processor_count) == (threads == 2)
    run_single(o, nsteps=(1, 3))
    s = cases.gpu_solver_from_oracle(o)
    assert s.kernel_info()["grid"] == (threads * n + 255) // 256
