"""The device plan's launch lists, from the library's own planner (tests/cpp/plan_lists.cpp)."""
import functools
import json
import os
import subprocess
import tempfile

import numpy as np

from tensors_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FRONT, SOLVE, SUPER_DIAG, SUPER_REST = 12, 5, 9, 10          # launch kinds


@functools.lru_cache(maxsize=None)
def _exe():
    out = os.path.join(tempfile.mkdtemp(prefix="plan_lists"), "plan_lists")
    libdir = os.path.dirname(_lib.LIB_PATH)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "tensors_b200", "csrc"), os.path.join(ROOT, "tests", "cpp", "plan_lists.cpp"), "-o", out,
                    "-L", libdir, "-ltensors_b200", f"-Wl,-rpath,{libdir}"], check=True)
    return out


def plan_lists(outer, inner, perm=None):
    """Fronts [n0, n1, level, parent, taken whole], front tasks [n0, n1, children], solve tasks
    [n0, n1, r0, c0, c1] and the launch lists by name."""
    n = len(outer) - 1
    perm = np.arange(n) if perm is None else perm
    data = b"".join(np.ascontiguousarray(a, dtype=t).tobytes() for a, t in
                    (((n, len(inner)), np.int64), (outer, np.int64), (inner, np.int32), (perm, np.int32)))
    return json.loads(subprocess.run([_exe()], input=data, check=True, capture_output=True).stdout)
