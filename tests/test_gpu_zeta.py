"""Merges with zeta != 0 in 2D (run on a GPU): Robin pairs other than the impedance one, whose zeta is 0.  There
B1 = -A2 T1_iN is formed from A2 = zeta I - T2_ii, the difference taken before the product, in every schedule.

Bars: the maps and the solution against the oracle at the small configuration's 1e-11 (test_gpu_parity); the
pipelined and the serial schedule bit for bit.  zeta close to the children's own reflection makes A2 small;
the oracle inverts it (condition about 1e2 there), so that pair has 1e-9."""
import numpy as np
import pytest

from robinsolver_b200 import workloads as W
from helpers import gpu_rhs, gpu_tree, oracle_run, rel_err

pytestmark = pytest.mark.gpu


def _pair(zeta, nu, b11):
    return np.array([[b11, 1.0], [(zeta + nu) * b11, zeta - nu]], dtype=np.complex128)


# interfaces of 16 to 64 points: columns of up to 16, the register interface of up to 32, separate launches above
@pytest.mark.parametrize("N,L", [(64, 4), (128, 4)])
@pytest.mark.parametrize("zeta,nu,bar", [(0.3 + 0.2j, -1.0, 1e-11), (-0.5j, 0.8 + 0.1j, 1e-11), ("reflection", -1.0, 1e-9)])
def test_merges_with_zeta_match_oracle(N, L, zeta, nu, bar):
    wl = W.make_workload(1, N=N, L=L)
    b11 = wl.bndry_params[0, 0]
    if zeta == "reflection":
        O, _ = oracle_run(wl)                          # a leaf's map does not depend on the pair
        r = O.levels[L][0].rtr
        zeta = np.mean(np.diag(r))
    wl.__class__ = type("Paired", (type(wl),), {"bndry_params": _pair(zeta, nu, b11)})
    O, U = oracle_run(wl)
    T, op, opts = gpu_tree(wl)
    T.plan(L, op, opts)
    k = wl.potential(T.sample_points(0))
    for _ in range(3):                                 # direct launches, capture, replay
        T.factor_samples(k)
    maps = [[np.array(T.get_rtr(l, i)) for i in range(2 ** l)] for l in range(L + 1)]
    for l in range(L + 1):
        for i in range(2 ** l):
            assert rel_err(maps[l][i], O.levels[l][i].rtr) < bar, (l, i)
    T.solve(gpu_rhs(wl.rhs))
    assert rel_err(T.solution_array(0), U[0]) < bar
    T.set_timing(2)                                    # the serial schedule
    T.factor_samples(k)
    for l in range(L + 1):
        for i in range(2 ** l):
            assert np.array_equal(np.array(T.get_rtr(l, i)), maps[l][i]), (l, i)
    T.close()
