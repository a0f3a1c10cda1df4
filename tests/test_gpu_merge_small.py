"""Merges of small interfaces (run on a GPU): the map of every node of every level against the oracle at
interface sizes around the kernels' tile edges (8, 16, 24, 32, 48, 64) and across the size from which
the levels run as separate products, at the bar the small configuration has (1e-11)."""
import numpy as np
import pytest

from robinsolver_b200 import workloads as W
from helpers import gpu_rhs, gpu_tree, oracle_run, rel_err

pytestmark = pytest.mark.gpu


# boxes of nx x ny cells cut L times, longest side first: interfaces of 7 to 64 points, and 66 and 128
# above them
@pytest.mark.parametrize("nx,ny,L", [(32, 7, 3), (32, 8, 2), (32, 15, 2), (36, 17, 2), (26, 24, 1), (64, 31, 2), (34, 33, 1),
                                     (84, 40, 2), (50, 49, 1), (128, 63, 2), (64, 64, 1), (66, 66, 2), (128, 128, 4)])
@pytest.mark.parametrize("graphs", [True, False])
def test_small_merges_match_oracle(nx, ny, L, graphs):
    h = 1.0 / 64.0
    wl = W.make_workload(1, kinds="plane")
    dom = np.array([[0.0, 0.0, 0.0], [nx * h, ny * h, 0.0]])
    wl.L, wl.domain, wl.N = L, dom, (1.0 - 1e-6) / h       # h_tgt a little above h
    for f in wl.rhs[0].g:
        f.domain = dom
    O, U = oracle_run(wl)
    T, op, opts = gpu_tree(wl, graphs=graphs)
    info = T.plan(L, op, opts)
    assert (info.root_a, info.root_b) == (nx, ny)
    for _ in range(3):                     # direct launches, then capture, then replay
        T.factor_samples(wl.potential(T.sample_points(0)))
    for l in range(L + 1):
        for i in range(2 ** l):
            assert rel_err(T.get_rtr(l, i), O.levels[l][i].rtr) < 1e-11, (l, i)
    T.solve(gpu_rhs(wl.rhs))
    assert rel_err(T.solution_array(0), U[0]) < 1e-11
    T.close()
