"""h3c_adjoint and h3c_cht_adjoint allocate before they run: an allocation that fails after the forward run would
leave the solver at another step than its scalars say.  An allocation cannot be made to fail here, so the order is
checked on the source."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hom3_b200", "csrc", "h3c_solver.cu")


def _body(name):
    s = re.sub(r"//[^\n]*", "", open(SRC).read())
    i = s.index(f"int {name}(h3c_solver")
    return s[i:s.index("\n}\n", i)]


@pytest.mark.parametrize("name", ["h3c_adjoint", "h3c_cht_adjoint"])
def test_the_staging_buffer_is_allocated_before_the_forward_run(name):
    b = _body(name)
    run = min(i for i in (b.find("enqueue_step("), b.find("fwd_seg("), b.find("coupled_begin(")) if i >= 0)
    stage = b.find("ensure_stage(")
    assert 0 <= stage < run
    assert "cudaMalloc" not in b[run:] and "ensure_stage" not in b[run:]
    if name == "h3c_adjoint":  # both of the caller's arrays are looked at
        assert re.search(r"dJ_dqN,[^;{]*dJ_dq0[^;]*\bin_place\(", b[:run], re.S)
