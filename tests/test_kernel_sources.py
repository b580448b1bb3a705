"""Orderings that a run cannot be relied on to show: what the kernels' sources have to contain."""
import glob
import os
import re

import flashkda_b200

CSRC = os.path.join(os.path.dirname(flashkda_b200.__file__), "csrc")


def _code(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_no_load_is_declared_invariant():
    """Inputs, states and tables may be written by a kernel that is still running when a dependent one starts, so no load of
    these kernels may be one that the compiler can move in front of the wait.  (The fold of context parallelism is launched
    normally.)"""
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        code = _code(path)
        if os.path.basename(path) == "fkda_cp.cu":
            assert "launch_dependent" not in code
            continue
        seen += code.count("grid_dep_wait();")
        for word in ("__ldg(", "__restrict__", "ld.global.nc"):
            assert word not in code, (path, word)
    assert seen >= 6   # decode, short, prefix, prepare, row-slice and one-kernel forms


def test_a_warp_barrier_between_the_chunks_of_a_pair():
    """The out tile of a walking warp is written by all lanes and read by all lanes in every chunk: a barrier lies between one
    chunk's reads and the next one's writes, also where two chunks share a stage."""
    code = _code(os.path.join(CSRC, "fkda_rows.cuh"))
    first, second = (m.start() for m in re.finditer(r"^\s+step\(", code, re.M))
    assert "__syncwarp();" in code[first:second] and "__syncwarp();" in code[second:]
    inside = code[code.index("w.chunk("):first]
    assert inside.index("stmatrix_x4_t(") < inside.index("__syncwarp();") < inside.index("lds_u4(")
