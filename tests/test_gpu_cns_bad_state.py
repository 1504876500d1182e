"""Cells that are no physical state in the CNS tile kernel's warp-wise time step: the minimum is the per-cell
kernel's, cell by cell (a NaN state's time step is a negative denormal; a cell of negative density and pressure
has a sound speed and a negative viscous time step), and the state check reports them."""
import ctypes as C

import numpy as np
import pytest

import cases
from hom3_b200 import _ffi as F
from test_gpu_cns_tile import _pair

pytestmark = pytest.mark.gpu


def _dt(s):
    v = C.c_double()
    F.lib().h3c_dt(s.h, C.byref(v))  # the value is set although the call reports the state
    return v.value


@pytest.mark.parametrize("kind", ["nan", "negative"])
def test_bad_cell_pulls_the_tile_kernels_time_step_like_the_per_cell_kernels(kind):
    _, (o,) = cases.tgv_case(level=4)
    fg, nd = o.first_ghost, 3
    got = []
    for s in _pair(o):
        q = s.state(0)
        q[:, 5] = np.nan if kind == "nan" else [0.0] * nd + [-1.0, -2.5]
        s.set_state(q)
        s.reset_time()
        s.dt(1e-9)  # the first step runs with a time step of its own; its stages reduce the second's
        s.solve(1)
        assert s.status() & 2  # a failed state check
        s.solve(1)
        got.append((_dt(s), s.status()))
    (da, fa), (db, fb) = got
    assert db < 0 and fb & 1  # outside [1e-300, 1e300]
    assert fa == fb
    assert da == db if kind == "nan" else abs(da - db) <= 1e-12 * abs(db)
