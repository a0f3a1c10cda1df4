"""The residue engine of the FP64 factor's large products (run on a GPU): against products summed in
extended precision, at shapes around its tiles (128 x 80, 64 of k), with rows and columns of very
different scales, zero rows, and infinities and NaNs.

Tolerance, per element relative to (largest |re|, |im| of A's row) (of B's column) k: both operands
are rounded to 2^-57 of their row's or column's largest entry (two parts each), 4 2^-57 k in all, and
the result is rounded once in FP64 (2 k 2^-53 at most, alpha and beta a few more): 2e-15 covers it,
fifty times below the FP64 engines' bar (test_gpu_tc5)."""
import numpy as np
import pytest

from test_gpu_tc5 import _run

pytestmark = pytest.mark.gpu

ALPHA, BETA = 0.7 - 0.2j, -0.5 + 0.25j


def _exact(A, B, C0):
    A, B, C0 = (x.astype(np.clongdouble) for x in (A, B, C0))
    return np.stack([ALPHA * (a @ b) + BETA * c for a, b, c in zip(A, B, C0)])


def _scale(A, B):
    ra = np.maximum(np.abs(A.real), np.abs(A.imag)).max(axis=2)
    cb = np.maximum(np.abs(B.real), np.abs(B.imag)).max(axis=1)
    return ra[:, :, None] * cb[:, None, :] * A.shape[2]


@pytest.mark.parametrize("m,n,k,cnt", [(128, 80, 64, 1), (1, 1, 1, 3), (129, 81, 65, 2), (300, 70, 123, 2), (256, 512, 256, 4),
                                       (200, 300, 512, 1), (64, 161, 1024, 1), (40, 1300, 31, 40)])
def test_crt_gemm_matches_extended_product(m, n, k, cnt):
    rng = np.random.default_rng(m + 5 * n + 7 * k)
    cx = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    A, B, C0 = cx(cnt, m, k), cx(cnt, k, n), cx(cnt, m, n)
    got = _run(4, A, B, C0, ALPHA, BETA)
    err = np.abs(got - _exact(A, B, C0).astype(np.complex128)) / (_scale(A, B) + np.abs(C0))
    assert err.max() < 2e-15, err.max()


def test_crt_gemm_scales_zero_rows_and_nonfinite():
    rng = np.random.default_rng(3)
    m, n, k = 150, 90, 100
    cx = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    A = cx(1, m, k) * 2.0 ** rng.integers(-300, 300, (1, m, 1))
    B = cx(1, k, n) * 2.0 ** rng.integers(-300, 300, (1, 1, n))
    A[0, 7] = 0.0
    C0 = np.zeros((1, m, n), dtype=np.complex128)
    got = _run(4, A, B, C0, ALPHA, 0j)
    s = _scale(A, B)
    ref = np.stack([ALPHA * (a @ b) for a, b in zip(A.astype(np.clongdouble), B.astype(np.clongdouble))])
    assert np.all(got[0, 7] == 0.0)
    rows = np.arange(m) != 7
    err = np.abs(got - ref.astype(np.complex128))[:, rows] / s[:, rows]
    assert err.max() < 2e-15, err.max()
    # an infinity or a NaN reaches its whole row or column and nothing else
    A2, B2 = A.copy(), B.copy()
    A2[0, 20, 5] = np.inf
    B2[0, 9, 30] = np.nan
    bad = _run(4, A2, B2, C0, ALPHA, 0j)
    mask = np.ones((m, n), dtype=bool)
    mask[20, :] = mask[:, 30] = False
    assert np.isnan(bad[0, 20]).all() and np.isnan(bad[0, :, 30]).all()
    assert np.array_equal(bad[0][mask], got[0][mask])


@pytest.mark.parametrize("m,n,k", [(130, 85, 70), (257, 80, 1024)])
def test_crt_gemm_problems_that_share_an_operand(m, n, k):
    """Neighbours with one A use one set of its planes: the same bits as with an A each."""
    import torch

    from robinsolver_b200 import _lib
    rng = np.random.default_rng(m)
    cx = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    A, B, C0 = np.repeat(cx(1, m, k), 3, axis=0), cx(3, k, n), cx(3, m, n)
    ref = _run(4, A, B, C0, ALPHA, BETA)
    dA, dB, dC = (torch.from_numpy(np.ascontiguousarray(x.transpose(0, 2, 1))).cuda() for x in (A[:1], B, C0))
    rc = _lib.lib.rb_test_zgemm(4, m, n, k, dA.data_ptr(), m, 0, dB.data_ptr(), k, k * n, dC.data_ptr(), m, m * n, ALPHA.real,
                                ALPHA.imag, BETA.real, BETA.imag, 3)
    assert rc == 0, _lib.last_error(None)
    assert np.array_equal(dC.cpu().numpy().transpose(0, 2, 1), ref)


def test_factor_without_room_for_the_residue_workspaces():
    """A budget that the workspaces do not fit leaves the products to the FP64 tiles, and one that
    they fit only until the solve's buffers come gives them back; nothing is refused.  Tolerance: both
    engines are FP64-accurate, and this system loses about 4 digits of 16 (1e-10 with room to spare)."""
    from helpers import gpu_rhs, gpu_tree
    from robinsolver_b200 import _lib
    from robinsolver_b200 import workloads as W
    wl = W.make_workload(2, nrhs=2)

    def run(budget):
        T, op, opts = gpu_tree(wl, device_budget=budget)
        T.plan(wl.L, op, opts)
        k = op.k(T.sample_points(_lib.RB_POINTS_POTENTIAL))
        T.factor_samples(k)
        held = T.info().device_bytes
        T.solve(gpu_rhs(wl.rhs))
        out = np.stack([T.solution_array(r) for r in range(2)])
        after = T.info().device_bytes
        T.factor_samples(k)                          # and again in the state that the solve left
        T.solve(gpu_rhs(wl.rhs))
        again = np.stack([T.solution_array(r) for r in range(2)])
        T.close()
        return held, after, out, again

    free = run(0)
    tight = run(free[0] - 1)
    assert tight[0] < free[0]
    late = run(free[0])
    assert late[0] == free[0] and late[1] == tight[1] < free[1]
    assert np.array_equal(late[2], free[2]) and np.array_equal(late[3], tight[3])
    for u in (tight[2], tight[3], late[3]):
        assert np.abs(u - free[2]).max() < 1e-10 * np.abs(free[2]).max()
