"""Kernel attributes belong to a context: a process that solves on one and then on another
(another device, or the same one after its context was replaced) gets the same results on both."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes as C
import numpy as np
from mfix_b200 import leq
from mfix_b200 import systems as S

def solve():
    # odd FP64 lines: k_jline's staging exceeds the 48 KB a kernel has without asking, in k_iterate
    # (7 rows a lane, 8 warps) and, with long lines, launched by itself
    out = []
    for dims, graph in (((20, 51, 18), 1), ((4, 601, 3), 0)):
        s = S.conv_diff(*dims, seed=3)
        assert leq.set_option("use_graph", graph) == 0
        ier = leq.solve_system(s)
        assert ier == 0, (ier, leq.last_error())
        out.append(s.x)
    leq.finalize()
    return out

first = solve()
cu = C.CDLL("libcuda.so.1")
ctx, dev = C.c_void_p(), C.c_int()
assert cu.cuInit(0) == 0 and cu.cuDeviceGet(C.byref(dev), 0) == 0
assert cu.cuCtxCreate_v2(C.byref(ctx), 0, dev) == 0  # current from here on
assert all(np.array_equal(u, v) for u, v in zip(first, solve()))
"""


def test_solves_in_a_second_context():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
