"""Leaf factor over block widths and counts at the edges of its kernels (run on a GPU): every leaf's
RtR map and the solution against the oracle's dense leaf LU, at the bar the small configuration has
(1e-11, test_gpu_parity)."""
import numpy as np
import pytest

from oracle import hps_ref as H
from robinsolver_b200 import workloads as W
from helpers import gpu_rhs, gpu_tree, oracle_run, rel_err

pytestmark = pytest.mark.gpu


# (a, b): widths around 8, 16, 24 and 32 (tile edges, one warp or several per leaf, the wide-block
# kernel above 32), block counts from 3 up, boundary counts off the multiples of 8
@pytest.mark.parametrize("a,b", [(3, 3), (5, 9), (8, 8), (9, 5), (15, 16), (16, 3), (16, 29), (17, 10), (19, 25), (24, 12),
                                 (25, 4), (31, 17), (32, 32), (33, 9)])
def test_leaf_maps_and_solution_match_oracle(a, b):
    # two cuts along x of a (4 a h) x (b h) box, or one along each axis when the box is too tall
    h = 1.0 / 64.0
    L = 2
    wl = W.make_workload(1, kinds="plane")
    wl2 = W.make_workload(1, instance=1)
    dom = np.array([[0.0, 0.0, 0.0], [4 * a * h, b * h, 0.0]]) if 2 * a >= b else \
        np.array([[0.0, 0.0, 0.0], [a * h, 4 * b * h, 0.0]])
    wl.L, wl.domain, wl.N = L, dom, (1.0 - 1e-6) / h       # h_tgt a little above h: ceil gives a and b
    for f in wl.rhs[0].g:
        f.domain = dom
    rhs = wl.rhs + wl2.rhs
    O, U = oracle_run(wl, rhs)
    T, op, opts = gpu_tree(wl)
    T.factor(L, op, opts)
    assert (T.info().leaf_a, T.info().leaf_b) == (a, b)
    for i in range(2 ** L):
        assert rel_err(T.get_rtr(L, i), O.levels[L][i].rtr) < 1e-11, i
    T.solve(gpu_rhs(rhs))
    for r in range(len(rhs)):
        assert rel_err(T.solution_array(r), U[r]) < 1e-11, r
    T.close()
