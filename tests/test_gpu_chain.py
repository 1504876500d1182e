"""The step as one chain: scalar work inside the conditions' kernel, the host's mirror of the scalars, third
Runge-Kutta buffers written out of place, coupled steps with both solvers' scalars set at once -- against the
same run by parts or by single calls, which take the separate kernels."""
import numpy as np
import pytest

import cases
import hom3_b200 as hb
from hom3_b200 import _ffi as F
from oracle import h3o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ti", [h3o.EULER_FORWARD, h3o.RK2, h3o.SSPRK3])
@pytest.mark.parametrize("graphs", [0, 1])
def test_whole_steps_equal_steps_by_parts(ti, graphs):
    _, (o,) = cases.euler_case("sod", nd=2, level=5, ti=ti)
    a, b = cases.gpu_solver_from_oracle(o), cases.gpu_solver_from_oracle(o)
    a.set_option(F.OPT_GRAPHS, graphs)
    for n in (1, 1, 3, 11):
        a.solve(n)
        for _ in range(n):
            for k in range(b.stages()):
                b.solve_stage(k)
        assert (a.dt(), a.time(), a.step()) == (b.dt(), b.time(), b.step())
        assert np.array_equal(a.state()[:, :o.first_ghost], b.state()[:, :o.first_ghost])


def test_mirror_follows_every_call():
    """dt / time / step after calls that change the scalars without a step in between."""
    _, (o,) = cases.euler_case("sod", nd=2, level=4)
    s = cases.gpu_solver_from_oracle(o)
    s.solve(3)
    t3, dt3 = s.time(), s.dt()
    assert s.step() == 3 and t3 > 0
    s.force_dt(0.5 * dt3)
    assert s.time() == t3 and s.dt() == dt3
    s.solve(1)
    assert s.dt() == 0.5 * dt3 and s.time() == t3 + 0.5 * dt3 and s.step() == 4
    s.solve_dt([0.25 * dt3] * 2)
    assert s.step() == 6 and s.dt() == 0.25 * dt3
    s.reset_time()
    assert s.time() == 0.0 and s.step() == 0
    s.solve(2)
    assert s.step() == 2
    q = s.state()
    q[2, 5] = np.nan
    s.set_state(q)
    with pytest.raises(hb.H3cError):  # the state check of set_state, not the last step's mirror
        s.dt()


def test_a_failing_step_is_seen_through_the_mirror():
    _, (o,) = cases.euler_case("sod", nd=2, level=4)
    s = cases.gpu_solver_from_oracle(o)
    s.solve(2)
    s.force_dt(1e3)  # far beyond the CFL limit: the step's result fails the state check
    s.solve(1)
    with pytest.raises(hb.H3cError):
        s.dt()
    assert s.status() & F.STATUS_STATE


def test_coupled_run_equals_single_coupled_steps():
    w, (cns, heat) = cases.cht_case(level=6, kappa=10.0)

    def pair():
        c, h = cases.gpu_solver_from_oracle(cns), cases.gpu_solver_from_oracle(heat)
        c.set_partner(h, cns.partner_cells())
        h.set_partner(c, heat.partner_cells())
        c.reset_time()
        h.reset_time()
        return c, h

    a, b = pair(), pair()
    hb.cht_solve(1.0, *a, 19)  # a plain step, graphs of 8, two single ones
    for _ in range(19):
        hb.couple_cht(1.0, *b)
        b[0].solve(1)
        b[1].solve(1)
    for x, y in zip(a, b):
        assert (x.dt(), x.time(), x.step()) == (y.dt(), y.time(), y.step())
        assert np.array_equal(x.state()[:, :x.first_ghost], y.state()[:, :y.first_ghost])
