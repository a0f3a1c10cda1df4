"""The tensor-core GEMMs' copy rings at their ends (run on a GPU): every CTA waits for its last copies before
it leaves, so a wait on the wrong phase would run into its bound of a second.  Block counts of k below,
at and above the rings' stages, and several row tiles behind one column tile.

The values are exact: small whole numbers, whose products and sums the first two engines hold without
rounding (split TF32: 11 bits an operand, 24 bits a sum), the third up to its weights' cut."""
import numpy as np
import pytest

from test_gpu_tc5 import _run

pytestmark = pytest.mark.gpu


# blocks of 16 (split TF32), 32 (digit slices) and 128 k (residues; resident B up to four blocks)
@pytest.mark.parametrize("engine,block", [(1, 16), (2, 32), (4, 128)])
@pytest.mark.parametrize("blocks", [1, 2, 3, 4, 5, 8])
def test_ring_ends_after_any_number_of_blocks(engine, block, blocks):
    import torch

    from robinsolver_b200 import _lib
    k = blocks * block - (blocks % 2)                 # a partial last block among them
    m, n, cnt = 700, 90, 2
    rng = np.random.default_rng(k)
    whole = lambda *s: (rng.integers(-3, 4, s) + 1j * rng.integers(-3, 4, s)).astype(np.complex128)  # noqa: E731
    A, B, C0 = whole(cnt, m, k), whole(cnt, k, n), whole(cnt, m, n)
    got = _run(engine, A, B, C0, 1.0 + 0.0j, 1.0 + 0.0j)
    ref = A @ B + C0
    if engine == 4:
        # entries of up to 3 are scaled to 2^54 each; the cut weights are off by at most 2^53.4 on their 2^108:
        # under half a unit in the last place of any whole number but zero
        assert np.abs(got - ref).max() < 2.0 ** -54
        assert np.array_equal(got.real[ref.real != 0], ref.real[ref.real != 0])
        assert np.array_equal(got.imag[ref.imag != 0], ref.imag[ref.imag != 0])
    else:
        assert np.array_equal(got, ref)
    # a warm launch, well below the bound of a wait
    dA, dB = (torch.from_numpy(np.ascontiguousarray(x.transpose(0, 2, 1))).cuda() for x in (A, B))
    dC = torch.zeros(cnt, n, m, dtype=torch.complex128, device="cuda")
    ms = _lib.C.c_double()
    rc = _lib.lib.rb_test_zgemm_timed(engine, m, n, k, dA.data_ptr(), m, m * k, dB.data_ptr(), k, k * n, dC.data_ptr(), m,
                                      m * n, 1.0, 0.0, 0.0, 0.0, cnt, 3, _lib.C.byref(ms))
    assert rc == 0 and ms.value < 100.0, (rc, ms.value)
