"""Kernels that start while the kernel in front of them still runs: what their sources may and may not do."""
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
