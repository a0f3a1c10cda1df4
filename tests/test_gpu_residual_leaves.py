"""The residual kernel's shared memory (run on a GPU): leaves whose u, or two of them, take just under 48 KB,
where only the kernel's static share goes over the limit that needs an opt-in, and the largest leaf,
whose u leaves 96 bytes of an SM's 227 KB.  Each in a process of its own: a larger leaf solved before
would have raised the limit already."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = """
import sys
sys.path[:0] = [r"{root}", r"{root}/tests"]
import numpy as np
from robinsolver_b200 import workloads as W
from helpers import gpu_rhs, gpu_tree
a, b = {a}, {b}
h = 1.0 / 64.0
wl = W.make_workload(1, kinds="plane")
dom = np.array([[0.0, 0.0, 0.0], [4 * a * h, b * h, 0.0]]) if 2 * a >= b else np.array([[0.0, 0.0, 0.0], [a * h, 4 * b * h, 0.0]])
wl.L, wl.domain, wl.N = 2, dom, (1.0 - 1e-6) / h
for f in wl.rhs[0].g:
    f.domain = dom
out = []
for precision in ("mixed", "fp64"):
    T, op, opts = gpu_tree(wl)
    T.factor(wl.L, op, opts, precision)
    assert (T.info().leaf_a, T.info().leaf_b) == (a, b), (T.info().leaf_a, T.info().leaf_b)
    T.solve(gpu_rhs(wl.rhs))
    out.append(T.solution_array(0))
    T.close()
assert np.abs(out[0] - out[1]).max() < 1e-9 * np.abs(out[1]).max()      # the refinement's tolerance is 1e-10
"""


# n = 2 (a + b) + a b points of 16 bytes, two buffers up to 56 KB together: 49024, 49056, 49152 and 49152 bytes;
# one buffer of 232352
@pytest.mark.parametrize("a,b", [(30, 46), (27, 51), (33, 42), (26, 53), (16, 805)])
def test_mixed_solve_on_leaves_near_a_limit(a, b):
    r = subprocess.run([sys.executable, "-c", PROGRAM.format(root=ROOT, a=a, b=b)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
