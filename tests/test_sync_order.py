"""Orderings between the lanes of a warp that no run can show to be missing: they are read off the
kernels' sources.  A vote orders no memory, so what one lane has acquired reaches another lane's
loads only through a warp barrier."""
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "wavedg_b200", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_resident_traces_are_read_behind_a_warp_barrier():
    stages = _code("stage_res.cu").split("const int nst = 5 * a.nsteps;")[1]
    wait, read = stages.index("res_wait("), stages.index("get(src")
    publish, release = stages.index("publish_row(dst"), stages.index("st_release(")
    assert wait < read < publish < release
    assert "__syncwarp()" in stages[wait:read]
    assert "__syncwarp()" in stages[publish:release]
