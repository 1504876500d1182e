"""States and cotangents handed over in device memory (read and written in place), through host memory, with a
leading dimension of their own, as views of the solver's own buffers, and in a numbering of the caller's own:
the same states and the same first time step."""
import ctypes as C

import numpy as np
import pytest
import torch

import hom3_b200 as hb
from hom3_b200 import _ffi as F
from hom3_b200.solver import Condition, GridSpec, build_tables

pytestmark = pytest.mark.gpu


def _grid(shuffled):
    spec = GridSpec(2, [0.0, 0.0], [1.0, 1.0], 4, refine=[([0.5, 0.5], 0.2, 5)])
    t = build_tables(spec, spec.cube_boundaries())
    if shuffled:  # interior cells in an order of the caller's own
        n, fg = t["ncells"], t["first_ghost"]
        new = np.concatenate([np.random.default_rng(1).permutation(fg), np.arange(fg, n)])  # old cell of each new one
        back = np.empty(n, np.int64)
        back[new] = np.arange(n)
        nb = t["neighbors"][:, new]
        t.update(neighbors=np.where((nb >= 0) & (nb < n), back[np.clip(nb, 0, n - 1)], nb),
                 x_center=np.ascontiguousarray(t["x_center"][:, new]), length=t["length"][new],
                 bc_idx=t["bc_idx"][new], subface_cells=back[t["subface_cells"]])
    return t


def _solver(t, physics=F.EULER):
    s = hb.Solver(2, physics, cfl=0.3, time_end=1e30)
    kind = F.BC_HEAT_NEUMANN if physics == F.HEAT else F.BC_EULER_NEUMANN
    s.set_grid(t["neighbors"], t["x_center"], t["length"], t["bc_idx"], t["first_ghost"], [Condition(kind)] * 4,
               t["subface_cells"])
    return s


def _state(t, nv):
    q = 1.0 + 0.2 * np.random.default_rng(0).random((nv, t["ncells"]))
    if nv > 1:
        q[nv - 1] += 2.0
    return q


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("physics,nv", [(F.EULER, 4), (F.HEAT, 1)])
def test_device_and_host_states_agree(shuffled, physics, nv):
    t = _grid(shuffled)
    q = _state(t, nv)
    a, b = _solver(t, physics), _solver(t, physics)
    a.set_state(q)
    b.set_state(torch.as_tensor(q, device="cuda"))
    assert np.array_equal(a.state(), q)
    out = torch.full((nv, t["ncells"]), np.nan, dtype=torch.float64, device="cuda")
    assert np.array_equal(b.state(out=out).cpu().numpy(), q)
    for s in (a, b):
        s.reset_time()
        s.solve(3)
    assert (a.dt(), a.time()) == (b.dt(), b.time())
    assert np.array_equal(a.state(), b.state(out=out).cpu().numpy())
    assert a.min_dt() == b.min_dt()


def test_leading_dimension_and_own_buffers():
    t = _grid(True)
    q = _state(t, 4)
    n, ld = t["ncells"], t["ncells"] + 37
    wide = torch.full((4, ld), -7.0, dtype=torch.float64, device="cuda")
    wide[:, :n] = torch.as_tensor(q, device="cuda")
    s = _solver(t)
    lib = hb.lib()
    ptr = lambda x: C.cast(x, C.POINTER(C.c_double))  # noqa: E731
    assert lib.h3c_set_state(s.h, 0, ptr(wide.data_ptr()), ld) == 0
    assert np.array_equal(s.state(), q)
    assert lib.h3c_get_state(s.h, 0, ptr(wide.data_ptr()), ld) == 0
    assert bool((wide[:, n:] == -7.0).all()) and np.array_equal(wide[:, :n].cpu().numpy(), q)
    # the solver's own (internally numbered) columns as a source: read whole before they are overwritten
    p, own_ld = s.device_state(0)
    order = s.device_order()
    internal = np.empty_like(q)
    internal[:, order] = q
    assert lib.h3c_set_state(s.h, 0, ptr(p), own_ld) == 0
    assert np.array_equal(s.state(), internal)


@pytest.mark.parametrize("shuffled", [False, True])
def test_adjoint_of_device_and_host_cotangents(shuffled):
    t = _grid(shuffled)
    q = _state(t, 4)
    lam = np.random.default_rng(2).random(q.shape)
    grads = []
    for dev in (False, True):
        s = _solver(t)
        s.set_state(q)
        s.reset_time()
        g, _ = s.adjoint(4, torch.as_tensor(lam, device="cuda") if dev else lam)
        grads.append(g.cpu().numpy() if dev else g)
    assert np.array_equal(*grads)
    assert not grads[0][:, t["first_ghost"]:].any()
