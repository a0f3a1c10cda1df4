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


@pytest.mark.parametrize("engine", [0, 4, 5])
def test_maps_bands_and_uneven_problems(engine):
    """What the parent maps are made of: rows by a map or around a skipped band, columns around a band, D
    through row and column maps, C from a band of the same matrix, problems of different rows beside each
    other, neighbours with one A -- all on one engine, on the FP64 tiles (0) and in parts (5) alike."""
    rng = np.random.default_rng(7)
    T = whole(rng, 420, 420)                                  # a child's map: interface rows and columns 100 .. 229
    m, o = 130, 100
    N = np.setdiff1d(np.arange(420), np.arange(o, o + m))
    Y = whole(rng, m, 2 * len(N))
    face, rest = N[::3], np.setdiff1d(N, N[::3])
    probs, refs, n = [], [], len(N)
    for rows in (face, rest):
        for half in range(2):
            A = Operand(T[:, o:o + m], rows=rows)
            B = Operand(Y[:, half * n:(half + 1) * n])
            D = Operand(np.zeros((900, 900), dtype=np.complex128), rows=rng.permutation(900)[:len(rows)], cols=rng.permutation(900)[:n])
            Cm = Operand(T, rows=rows, cband=(o, m)) if half == 0 else None
            ref = T[np.ix_(rows, np.arange(o, o + m))] @ B.M + (Cm.host(len(rows), n) if Cm else 0.0)
            out = np.zeros((900, 900), dtype=np.complex128)
            out[np.ix_(D.ix[0], D.ix[1])] = ref
            refs.append(out)
            probs.append((A, B, Cm, D, 1.0 + 0j, 1.0 + 0j, len(rows), n, m))
    # and the whole map of the serial schedule: A and C around the band's rows
    A = Operand(T[:, o:o + m], rband=(o, m))
    D = Operand(np.zeros((n, n), dtype=np.complex128))
    Cm = Operand(T, rband=(o, m), cband=(o, m))
    refs.append(A.host(n, m) @ Y[:, :n] + Cm.host(n, n))
    probs.append((A, Operand(Y[:, :n]), Cm, D, 1.0 + 0j, 1.0 + 0j, n, n, m))
    for i, (got, ref) in enumerate(zip(run(engine, probs), refs)):
        assert same(got, ref), i


def test_a_map_in_row_sets_has_the_bits_of_the_whole():
    """An element depends on its row and column only: the face rows and the others, of other problem sizes,
    against the whole map, on operands of no special values."""
    rng = np.random.default_rng(8)
    cx = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    M, n, k = 700, 333, 576
    T, Y, C0 = cx(M, k), cx(k, n), cx(M, n)
    rows = [np.sort(rng.permutation(M)[:257])]
    rows.append(np.setdiff1d(np.arange(M), rows[0]))

    def problem(sel):
        out = Operand(np.zeros((M, n), dtype=np.complex128), rows=sel)
        return (Operand(T, rows=sel), Operand(Y), Operand(C0, rows=sel), out, 0.7 - 0.2j, -0.5 + 0.25j, len(sel), n, k)

    full, = run(4, [problem(np.arange(M))])
    a, b = run(4, [problem(r) for r in rows])
    assert np.array_equal(a[rows[0]], full[rows[0]]) and np.array_equal(b[rows[1]], full[rows[1]])


def _units(X, axis):
    """The spacing that X's entries are rounded to: 2^-57 times a power of two above twice their row's or
    column's largest part."""
    big = np.maximum(np.abs(X.real), np.abs(X.imag)).max(axis=axis)
    return 2.0 ** (np.frexp(big)[1] + 1 - 57)


# k around the blocks of 128, up to and past the four of a resident B (512), blocks that do not fill the four stages
@pytest.mark.parametrize("k", [1, 2, 31, 127, 128, 129, 513, 576, 640, 1000, 1024])
@pytest.mark.parametrize("graded", [False, True])
def test_error_is_the_rounding_of_the_operands(k, graded):
    """Against extended precision, with one rounding of every entry to its row's or column's units ua, ub:
    per part at most  sum_k ua/2 (|br| + |bi|) + ub/2 (|ar| + |ai|) + ua ub/2, the weights' cut, 2^53.4 ua ub, and a
    rounding of the result at 2^-53; and in the mean square twice what uniform roundings give,
    sum_k ua^2/12 |b|^2 + ub^2/12 |a|^2.  Neither has a factor of k for what does not grow with it.  Graded: entries
    spread over 2^-40 .. 1 inside every row and column."""
    from test_gpu_tc5 import _run
    rng = np.random.default_rng(1000 * graded + k)
    m, n = 173, 91
    cx = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    A, B = cx(m, k), cx(k, n)
    if graded:
        A *= 2.0 ** -rng.uniform(0.0, 40.0, (m, k))
        B *= 2.0 ** -rng.uniform(0.0, 40.0, (k, n))
    got = _run(4, A[None], B[None], np.zeros((1, m, n), dtype=np.complex128), 1.0 + 0j, 0j)[0]
    ref = A.astype(np.clongdouble) @ B.astype(np.clongdouble)
    ua, ub = _units(A, 1)[:, None], _units(B, 0)[None, :]
    sa, sb = (np.abs(A.real) + np.abs(A.imag)).sum(1)[:, None], (np.abs(B.real) + np.abs(B.imag)).sum(0)[None, :]
    cut = 2.0 ** 53.4 * ua * ub
    e = got - ref
    for part, r in ((e.real, ref.real), (e.imag, ref.imag)):
        bound = ua / 2 * sb + ub / 2 * sa + k * ua * ub / 2 + cut + 2.0 ** -53 * (np.abs(r) + cut)
        assert np.all(np.abs(part) <= bound.astype(float)), float(np.max(np.abs(part) / bound))
    sa2, sb2 = (np.abs(A) ** 2).sum(1)[:, None], (np.abs(B) ** 2).sum(0)[None, :]
    mean = ua ** 2 / 12 * sb2 + ub ** 2 / 12 * sa2 + cut ** 2 + (2.0 ** -53 * np.abs(ref)).astype(float) ** 2 / 3
    # relative to each element's own expectation, both parts together
    assert np.sqrt((np.abs(e).astype(float) ** 2 / (2 * mean)).mean()) < 2.0
