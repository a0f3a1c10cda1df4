"""Which products of the FP64 factor run on the residue engine (run on a GPU), and what they are worth: parent
maps only, as exact as the FP64 tiles by every measure on the factor's own operands."""
import numpy as np
import pytest

from robinsolver_b200 import workloads as W
from helpers import gpu_tree
from test_gpu_tc5 import _run

pytestmark = pytest.mark.gpu


def _map_operands(T, level):
    """[(name, A, B)] of the two row blocks of a level's first map, and its interface points: T_Ni and [Y1; Y2]
    (K form, zeta = 0, nu = -1) formed on the host from the children's maps."""
    a, b, _ = T._level_grid(level + 1)
    r1, r2 = np.array(T.get_rtr(level + 1, 0)), np.array(T.get_rtr(level + 1, 1))
    pa, pb, _ = T._level_grid(level)
    off = np.cumsum([0, b, b, a, a])                      # faces x1 x2 y1 y2
    f1, f2 = (1, 0) if pa > a else (3, 2)
    i1, i2 = np.arange(off[f1], off[f1 + 1]), np.arange(off[f2], off[f2 + 1])
    N1, N2 = np.setdiff1d(np.arange(off[4]), i1), np.setdiff1d(np.arange(off[4]), i2)
    A1, A2 = -r1[np.ix_(i1, i1)], -r2[np.ix_(i2, i2)]
    T1iN, T2iN = r1[np.ix_(i1, N1)], r2[np.ix_(i2, N2)]
    Ki = np.linalg.inv(np.eye(len(i1)) - A2 @ A1)
    Y1 = Ki @ np.concatenate([-A2 @ T1iN, -T2iN], 1)
    Y2 = A1 @ Y1
    Y2[:, :len(N1)] -= T1iN
    return [("map1", r1[np.ix_(N1, i1)], Y1), ("map2", r2[np.ix_(N2, i2)], Y2)], len(i1)


@pytest.mark.parametrize("N,L", [(512, 10), (768, 10)])
def test_only_the_maps_run_on_the_residue_engine(N, L):
    wl = W.make_workload(2, N=N, L=L, nrhs=1)
    T, op, opts = gpu_tree(wl)
    T.plan(L, op, opts)
    k = wl.potential(T.sample_points(0))
    T.factor_samples(k)
    T.set_timing(2)
    T.clear_stage_times()
    T.factor_samples(k)
    flops = sum(f for name, _, f in T.stage_times(with_flops=True) if name == "zgemm_crt")
    want = 0.0
    for l in range(L):
        pa, pb, _ = T._level_grid(l)
        a, b, _ = T._level_grid(l + 1)
        m = b if pa > a else a
        n = 2 * (a + b) - m
        if m >= 256 and m * n >= 1 << 18:
            want += 2 ** l * 4 * 8.0 * n * n * m
    assert want > 0 and abs(flops - want) < 1e-9 * want, (flops, want)
    T.close()


@pytest.mark.parametrize("N,L", [(512, 10), (768, 10)])
def test_map_products_are_as_exact_as_the_fp64_tiles(N, L):
    """On a root's own operands, every element's error relative to (|A| |B|)_ij, largest and mean square, no
    larger than the tiles', whose own is at most 8 2^-53 (k + 4) (three real products and their sum)."""
    wl = W.make_workload(2, N=N, L=L, nrhs=1)
    T, op, opts = gpu_tree(wl)
    T.factor(L, op, opts)
    rng = np.random.default_rng(N)
    prods, m = _map_operands(T, 0)
    T.close()
    for name, A, B in prods:
        A, B = np.ascontiguousarray(A), np.ascontiguousarray(B)
        rows = np.sort(rng.choice(A.shape[0], 24, replace=False))
        cols = np.sort(rng.choice(B.shape[1], 60, replace=False))
        ref = A[rows].astype(np.clongdouble) @ B[:, cols].astype(np.clongdouble)
        sab = np.abs(A[rows]) @ np.abs(B[:, cols])
        C0 = np.zeros((1, A.shape[0], B.shape[1]), dtype=np.complex128)
        e = {eng: np.abs(_run(eng, A[None], B[None], C0, 1.0 + 0j, 0j)[0][np.ix_(rows, cols)] - ref).astype(float) / sab
             for eng in (0, 4)}
        assert e[0].max() < 8 * 2.0 ** -53 * (m + 4)
        assert e[4].max() <= e[0].max() and np.sqrt((e[4] ** 2).mean()) <= np.sqrt((e[0] ** 2).mean()), name


def _map_with(wl, factors=1, **kw):
    T, op, opts = gpu_tree(wl, **kw)
    T.plan(wl.L, op, opts)
    k = wl.potential(T.sample_points(0))
    for _ in range(factors):
        T.factor_samples(k)
    out = np.array(T.get_rtr(0, 0)), T.info().residue_maps, T.info().device_bytes
    T.close()
    return out


def test_a_caller_can_keep_the_fp64_products():
    """RB_FLAG_FP64_PRODUCTS: the bits of a tree whose budget has no room for the workspaces, and no workspaces
    held; the default differs from them by rounding only."""
    wl = W.make_workload(2, nrhs=1)
    ref, on, held = _map_with(wl)
    fp64, off, less = _map_with(wl, factors=3, fp64_products=True)
    assert (on, off) == (1, 0) and less < held
    tight, off2, _ = _map_with(wl, device_budget=less)
    assert off2 == 0 and np.array_equal(fp64, tight)
    assert not np.array_equal(ref, fp64) and np.abs(ref - fp64).max() < 1e-11 * np.abs(fp64).max()


def test_the_dfma_engine_reaches_every_product():
    """RB_GEMM_ENGINE=dfma (read once a process): no batched GEMM on any tensor core."""
    import os
    import subprocess
    import sys
    from pathlib import Path
    root = Path(__file__).resolve().parents[1]
    prog = ("import sys; sys.path[:0] = [r'%s', r'%s/tests']\n"
            "from robinsolver_b200 import workloads as W\nfrom helpers import gpu_tree\n"
            "wl = W.make_workload(2, nrhs=1)\nT, op, opts = gpu_tree(wl)\nT.plan(wl.L, op, opts)\n"
            "k = wl.potential(T.sample_points(0))\nT.factor_samples(k)\nT.set_timing(2)\nT.clear_stage_times()\nT.factor_samples(k)\n"
            "assert T.info().residue_maps == 0\n"
            "names = {e[0] for e in T.stage_times()}\nassert not {n for n in names if 'crt' in n or 'tc' in n}, names\n" % (root, root))
    r = subprocess.run([sys.executable, "-c", prog], env=dict(os.environ, RB_GEMM_ENGINE="dfma"), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


# one split level (768^2) and two (1024^2), and the largest cube: the parts of a workspace, the rule of 256 points
@pytest.mark.parametrize("case", ["768", "1024", "cube"])
def test_pipelined_and_serial_maps_agree_bit_for_bit(case):
    """The pipelined factor's face rows and other rows against the serial one's whole maps, on every level that
    uses the engine, direct and from a graph."""
    import robinsolver_b200 as rb
    if case == "cube":
        T = rb.robin_tree(skip_root_rtr=False)
        T.bndry_params = np.array([[1j, 1.0], [-1j, 1.0]], dtype=np.complex128)
        L = 9
        T.plan(L, rb.elliptic_operator(d=3, domain=np.array([[0.0, 0.0, 0.0], [1.0, 1.0, 1.0]])), rb.solve_opts(h_tgt=1.0 / 32, kb=1.0))
        X = T.sample_points(0)
        k = 1.0 + 0.3 * np.exp(-((X - 0.4) ** 2).sum(1) / 0.02) + 0.01j
    else:
        wl = W.make_workload(2 if case == "768" else 4, N=int(case), L={"768": 10, "1024": 12}[case], nrhs=1)
        T, op, opts = gpu_tree(wl)
        T.plan(wl.L, op, opts)
        k = wl.potential(T.sample_points(0))
    nodes = [(0, 0), (1, 0), (1, 1), (2, 1), (2, 2)]
    T.factor_samples(k)
    assert T.info().residue_maps == 1
    maps = [np.array(T.get_rtr(*v)) for v in nodes]
    for _ in range(2):                                    # captured, replayed
        T.factor_samples(k)
    for v, a in zip(nodes, maps):
        assert np.array_equal(np.array(T.get_rtr(*v)), a), v
    T.set_timing(2)                                       # the serial schedule
    T.factor_samples(k)
    for v, a in zip(nodes, maps):
        assert np.array_equal(np.array(T.get_rtr(*v)), a), v
    T.close()
