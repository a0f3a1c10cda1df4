"""The solve's GEMM (run on a GPU): its kernels for few and for many right-hand sides against a host
product, and bit for bit against each other -- a column's result may not depend on how many columns
there are."""
import numpy as np
import pytest

from test_gpu_tc5 import _run

pytestmark = pytest.mark.gpu


# rows and k around the tiles (8 rows, k-steps of 4, k ranges of a split batch), one problem (split
# 16 ways) to many (not split)
@pytest.mark.parametrize("m,k,cnt", [(16, 16, 700), (16, 96, 300), (17, 33, 5), (64, 256, 3), (100, 130, 2), (512, 512, 1),
                                     (129, 1000, 1), (3, 1024, 1), (1024, 2048, 1)])
def test_solve_gemm_columns_do_not_depend_on_their_number(m, k, cnt):
    rng = np.random.default_rng(m + 3 * k + cnt)
    N = 40
    A = rng.standard_normal((cnt, m, k)) + 1j * rng.standard_normal((cnt, m, k))
    B = rng.standard_normal((cnt, k, N)) + 1j * rng.standard_normal((cnt, k, N))
    C0 = rng.standard_normal((cnt, m, N)) + 1j * rng.standard_normal((cnt, m, N))
    alpha, beta = 0.7 - 0.2j, -0.5 + 0.25j
    ref = alpha * (A @ B) + beta * C0
    scale = np.abs(A).max() * np.abs(B).max() * k
    full = _run(3, A, B, C0, alpha, beta)
    assert np.abs(full - ref).max() / scale < 1e-13          # the FP64 engines' bar (test_gpu_tc5)
    for n in (1, 3, 8, 9, 16, 17, 32):
        assert np.array_equal(_run(3, A, B[:, :, :n], C0[:, :, :n], alpha, beta), full[:, :, :n]), n


@pytest.mark.parametrize("cells,L", [(112, 6), (96, 5)])
def test_a_column_does_not_depend_on_the_batch_it_is_solved_in(cells, L):
    """Whole solves, whose products gather their right-hand sides through maps: one column (the streaming
    kernel), 17 (32- and 16-row tiles of 32 columns) and 33 (two of them), bit for bit."""
    from helpers import gpu_rhs, gpu_tree
    from robinsolver_b200 import workloads as W
    wl = W.make_workload(1, N=cells, L=L, nrhs=33)
    T, op, opts = gpu_tree(wl)
    T.factor(wl.L, op, opts)
    out = {}
    for n in (33, 17, 1):
        T.solve(gpu_rhs(wl.rhs[:n]))
        out[n] = np.stack([T.solution_array(r) for r in range(n)])
    T.close()
    assert np.array_equal(out[33][:17], out[17])
    assert np.array_equal(out[33][:1], out[1])
