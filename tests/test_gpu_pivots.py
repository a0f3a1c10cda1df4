"""Pivot selection of the batched inversions (run on a GPU): the row of largest |re| + |im| in all 53 bits.

The kernels move no rows: an element's operations depend on its row's entries and the order of the pivots,
not on where the row stands.  So with the rows of a matrix permuted, and no two magnitudes equal, the
inverse is the same one with its columns permuted, bit for bit -- unless near-equal magnitudes are told
apart by position."""
import numpy as np
import pytest

from test_gpu_gj import _invert

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [2, 7, 16, 17, 32, 33, 50, 64, 100, 300])
def test_near_equal_pivots_do_not_fall_by_position(m):
    rng = np.random.default_rng(m)
    A = (rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m))) / np.sqrt(m)
    # every entry of the first columns within 2^-25 of magnitude 2, in random directions
    c = min(m, 4)
    t = rng.uniform(0.0, 2.0 * np.pi, (m, c))
    u = np.exp(1j * t)
    A[:, :c] = u / (np.abs(u.real) + np.abs(u.imag)) * (2.0 + rng.permuted(np.tile(np.arange(m), (c, 1)), axis=1).T * 2.0 ** -33)
    perms = [np.arange(m)] + [rng.permutation(m) for _ in range(3)]
    X, _ = _invert(np.stack([A[p] for p in perms]))
    assert np.abs(X[0] @ A - np.eye(m)).max() < 1e-9
    for x, p in zip(X[1:], perms[1:]):
        assert np.array_equal(x, X[0][:, p])


@pytest.mark.parametrize("m", [3, 20, 40])
def test_subnormal_column_keeps_its_largest_entry(m):
    """A column of zeros but for one subnormal entry: that row is the pivot (its reciprocal overflows, as
    it does on the host), not a zero that shares its leading bits."""
    A = np.eye(m, dtype=np.complex128)[None].copy()
    A[0, 0, 0] = 0.0
    A[0, m - 1, 0] = 2.0 ** -1060
    A[0, 0, m - 1], A[0, m - 1, m - 1] = 1.0, 0.0
    _invert(A)                            # no zero pivot reported
