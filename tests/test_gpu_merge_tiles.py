"""The FP64 tensor-core tiles of the larger merge products (run on a GPU): 32x32 tiles where 64x64 ones would
leave a wave mostly empty, 64x64 otherwise -- the same sums, so a problem's result may not depend on how
many share its batch.

Tolerance: three real products of k terms each and their combination, every sum and product rounded at
2^-53: within 8 2^-53 (k + 4) of (largest modulus of A) (largest of B), below 2e-15 k for k >= 4."""
import numpy as np
import pytest

from test_gpu_tc5 import _run

pytestmark = pytest.mark.gpu


# one problem, and as many as fill the 64x64 tiles' waves; rows, columns and k around the tiles
@pytest.mark.parametrize("m,n,k,many", [(256, 256, 256, 18), (200, 65, 128, 74), (193, 257, 131, 15), (512, 96, 129, 37)])
def test_merge_product_does_not_depend_on_the_batch(m, n, k, many):
    rng = np.random.default_rng(m + n + k)
    cx = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    A, B, C0 = cx(many, m, k), cx(many, k, n), cx(many, m, n)
    alpha, beta = 0.7 - 0.2j, -0.5 + 0.25j
    full = _run(0, A, B, C0, alpha, beta)
    one = _run(0, A[:1], B[:1], C0[:1], alpha, beta)
    assert np.array_equal(full[0], one[0])
    scale = np.abs(A).max() * np.abs(B).max() * k
    assert np.abs(full - (alpha * (A @ B) + beta * C0)).max() < 2e-15 * scale
