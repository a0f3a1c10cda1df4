"""Where the residue engine's workspaces come from (run on a GPU): the plan, the precision and the handle's
budget decide whether a factor's maps use it; only a device with no room to speak of does besides, and then
the next factorization tries again.  rb_info.residue_maps says which engine the last one used."""
import numpy as np
import pytest

from robinsolver_b200 import workloads as W
from helpers import gpu_tree
from test_gpu_tc5 import _run

pytestmark = pytest.mark.gpu


def _hog(leave):
    """Device memory taken until `leave` bytes are free."""
    import torch
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    assert free > leave
    return torch.empty(free - leave, dtype=torch.uint8, device="cuda")


def _root_map(T, k):
    T.factor_samples(k)
    return np.array(T.get_rtr(0, 0)), T.info().residue_maps, T.info().device_bytes


def test_engine_does_not_depend_on_what_else_is_on_the_device():
    import torch
    wl = W.make_workload(2, nrhs=1)

    def tree():
        T, op, opts = gpu_tree(wl)
        T.plan(wl.L, op, opts)
        return T, wl.potential(T.sample_points(0))

    T, k = tree()
    ref, on, held = _root_map(T, k)
    assert on == 1
    T.close()
    # 4 GB beside the factor's storage: eight times the workspaces, less than sixteen times
    hog = _hog(held + (4 << 30))
    T, k = tree()
    got, on, _ = _root_map(T, k)
    assert on == 1 and np.array_equal(got, ref)
    T.close()
    del hog
    # no room beside the storage: FP64 tiles, and the engine again once there is some
    hog = _hog(held + (64 << 20))
    T, k = tree()
    tiles, on, bytes_without = _root_map(T, k)
    assert on == 0 and bytes_without < held
    assert not np.array_equal(tiles, ref) and np.abs(tiles - ref).max() < 1e-10 * np.abs(ref).max()
    del hog
    torch.cuda.empty_cache()
    for _ in range(3):                               # direct, captured, replayed
        got, on, again = _root_map(T, k)
        assert on == 1 and again == held and np.array_equal(got, ref)
    T.close()


def test_mixed_factor_without_fp64_maps_holds_no_workspaces():
    """Mixed precision with the top levels on the digit-slice engine as well: no map is left for the residues,
    and their workspaces come with the first FP64 factorization."""
    wl = W.make_workload(2, nrhs=1)
    T, op, opts = gpu_tree(wl, mixed_int8_top=True)
    T.plan(wl.L, op, opts)
    k = wl.potential(T.sample_points(0))
    T.factor_samples(k, "mixed")
    assert T.info().residue_maps == 0
    held = T.info().device_bytes
    T.factor_samples(k, "fp64")
    assert T.info().residue_maps == 1 and T.info().device_bytes > held
    T.factor_samples(k, "mixed")
    assert T.info().residue_maps == 0
    T.close()


@pytest.mark.parametrize("m,n,k,cnt", [(130, 85, 70, 5), (257, 80, 600, 4), (64, 300, 129, 3), (40, 40, 40, 1)])
def test_batch_in_parts_gives_the_same_bits(m, n, k, cnt):
    rng = np.random.default_rng(m + cnt)
    cx = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    A, B, C0 = cx(cnt, m, k), cx(cnt, k, n), cx(cnt, m, n)
    args = (A, B, C0, 0.7 - 0.2j, -0.5 + 0.25j)
    assert np.array_equal(_run(5, *args), _run(4, *args))
