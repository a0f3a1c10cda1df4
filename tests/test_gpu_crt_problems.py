"""The residue engine on the forms its callers give it (run on a GPU): problems of different sizes in one
batch, row maps, column maps and skipped bands, operands that neighbours share.

Values are small whole numbers: the engine returns every whole number but zero exactly, and zero within
2^-53 (entries of up to 3 are scaled to 2^54 each, the weights' cut is off by at most 2^53.4 on their
2^108)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INT_MAX = 2 ** 31 - 1


class View(C.Structure):            # ZView and ZOut (rb_common.cuh)
    _fields_ = [("p", C.c_void_p), ("rmap", C.c_void_p), ("cmap", C.c_void_p), ("ld", C.c_longlong), ("rs", C.c_int),
                ("rl", C.c_int), ("cs", C.c_int), ("cl", C.c_int)]


class Desc(C.Structure):            # GemmDesc
    _fields_ = [("A", View), ("B", View), ("C", View), ("D", View), ("alpha", C.c_double * 2), ("beta", C.c_double * 2),
                ("m", C.c_int), ("n", C.c_int), ("k", C.c_int), ("nobeta_r0", C.c_int), ("nobeta_r1", C.c_int),
                ("pad", C.c_int), ("tail", C.c_int * 2)]


class Operand:
    """A matrix in device memory (column-major) and the rows and columns of it that a problem takes."""

    def __init__(self, M, rows=None, cols=None, rband=None, cband=None):
        import torch
        self.M = M
        self.d = torch.from_numpy(np.ascontiguousarray(M.T)).cuda()
        self.maps = [None if x is None else torch.from_numpy(np.ascontiguousarray(x, dtype=np.int32)).cuda() for x in (rows, cols)]
        self.bands = [rband or (INT_MAX, 0), cband or (INT_MAX, 0)]
        ix = []
        for want, band, size in ((rows, self.bands[0], M.shape[0]), (cols, self.bands[1], M.shape[1])):
            i = np.arange(size)
            ix.append(np.asarray(want) if want is not None else i[(i < band[0]) | (i >= band[0] + band[1])])
        self.ix = ix

    def view(self):
        ptr = [0 if m is None else m.data_ptr() for m in self.maps]
        return View(self.d.data_ptr(), ptr[0] or None, ptr[1] or None, self.M.shape[0], *self.bands[0], *self.bands[1])

    def host(self, m, n):
        return self.M[np.ix_(self.ix[0][:m], self.ix[1][:n])]


NONE = View(None, None, None, 1, INT_MAX, 0, INT_MAX, 0)


def run(engine, problems):
    """problems: (A, B, C or None, D, alpha, beta, m, n, k); D's matrices afterwards."""
    from robinsolver_b200 import _lib
    h = (Desc * len(problems))()
    for g, (A, B, Cm, D, alpha, beta, m, n, k) in zip(h, problems):
        g.A, g.B, g.C, g.D = A.view(), B.view(), NONE if Cm is None else Cm.view(), D.view()
        g.alpha[:], g.beta[:] = (alpha.real, alpha.imag), (beta.real, beta.imag)
        g.m, g.n, g.k = m, n, k
    assert C.sizeof(Desc) == 256
    rc = _lib.lib.rb_test_zgemm_descs(engine, len(problems), C.cast(h, C.c_void_p))
    assert rc == 0, (rc, _lib.last_error(None))
    return [p[3].d.cpu().numpy().T for p in problems]


def whole(rng, *s):
    return (rng.integers(-3, 4, s) + 1j * rng.integers(-3, 4, s)).astype(np.complex128)


def same(got, ref):
    z = ref == 0
    return np.array_equal(got[~z].real[ref[~z].real != 0], ref[~z].real[ref[~z].real != 0]) and \
        np.array_equal(got[~z].imag[ref[~z].imag != 0], ref[~z].imag[ref[~z].imag != 0]) and \
        np.abs(got - ref).max(initial=0.0) < 2.0 ** -53


def test_a_problem_without_terms_beside_others():
    """k = 0: the product is empty, the result beta C; its neighbours are what they are alone."""
    rng = np.random.default_rng(1)
    sizes = [(130, 85, 200), (90, 40, 0), (300, 81, 129)]
    probs, refs = [], []
    for m, n, k in sizes:
        A, B, D = Operand(whole(rng, m, max(k, 1))), Operand(whole(rng, max(k, 1), n)), Operand(whole(rng, m, n))
        refs.append(A.M[:, :k] @ B.M[:k] + 2.0 * D.M)
        probs.append((A, B, D, D, 1.0 + 0j, 2.0 + 0j, m, n, k))
    for got, ref in zip(run(4, probs), refs):
        assert same(got, ref)
