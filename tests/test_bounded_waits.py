"""A block whose wait for its bulk copies ran out flags that and waits once more, with a limit, before it gives its
shared memory back to copies that may still land there.  No GPU is made to run into the limit: checked on the
sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hom3_b200", "csrc")


@pytest.mark.parametrize("name", ["stage_cns.cuh", "h3c_stage_halo.cu"])
def test_copies_in_flight_are_waited_for_after_a_timeout(name):
    s = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    gave_up = re.findall(r"if \(!__syncthreads_and\(ok\)\) \{(.*?)\n    \}", s, re.S)
    assert len(gave_up) == 1
    b = gave_up[0]
    assert 0 <= b.find("flag_timeout(") < b.find("mbar_wait_bounded(") < b.find("return;")


def test_every_wait_on_a_barrier_is_bounded():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")) and f != "async_copy.cuh":
            assert "mbar_try_wait" not in open(os.path.join(CSRC, f)).read(), f
