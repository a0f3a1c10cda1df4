"""The calls this library is used for, as timed cases: factorizations, solves and whole steps over
the sizes, leaf grids, right-hand-side counts, dimensions and precisions of its benchmark
configurations and tests.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) a planned (or, for solves, factored) tree and its seeded inputs
    run(state)          one pass through the public entry points; returns every solution
    work(case)          bytes and operations of one pass that no implementation can do without
    exact(case, seed)   the same solutions from a plain torch elimination in FP64

A case is a plain dict: ``kind`` is what one pass does,

    step    factor a new potential and solve its right-hand sides, device arrays in and out
    solve   solve right-hand sides on a resident factorization, device arrays in and out
    host    factor, solve and read every solution back through the Python API's host arrays
    forest  factor ``trees`` trees of uneven sizes together, then solve each of them

over a box of ``width`` x 1 (x 1) cut ``L`` times with ``leaf`` cells along x in every leaf.  The
equation is Helmholtz with a smooth bump potential and impedance data (u_n - i kb u = g in 2D); the
right-hand sides are Gaussian point sources, plane waves through the boundary, or both in turn.
"""
from __future__ import annotations

import math

import numpy as np
import torch

# ---------------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------------


def _case(name, kind, L, leaf, nrhs, kb, rhs, d=2, width=1.0, precision="fp64", overlap=False, trees=0):
    c = {"kind": kind, "d": d, "width": width, "L": L, "leaf": leaf, "nrhs": nrhs, "kb": kb, "rhs": rhs,
         "precision": precision, "overlap": overlap, "trees": trees}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the smallest configuration: 64^2, one point source; launches and latencies are all of it
        _case("step_64_1rhs", "step", 4, 16, 1, 20.0, "point"),
        # a host program through factor/solve/get_solution arrays: the serving set's smallest grid,
        # 256^2 with 32x32 leaves, a few right-hand sides
        _case("host_256_4rhs", "host", 6, 32, 4, 80.0, "both"),
        # the ordinary configuration: 512^2, 16 mixed right-hand sides, one factorization each
        _case("step_512_16rhs", "step", 10, 16, 16, 100.0, "both"),
        # the headline: 1024^2, 32 plane waves, the solve beside the factor (asynchronous factor)
        _case("step_1024_32rhs", "step", 12, 16, 32, 200.0, "plane", overlap=True),
        # the headline in mixed precision: tensor-core merges, refined solves
        _case("mixed_1024_32rhs", "step", 12, 16, 32, 200.0, "plane", precision="mixed", overlap=True),
        # a box that is no square and divides badly: 3:2, 19-cell leaves, an odd count
        _case("step_ragged_7rhs", "step", 7, 19, 7, 60.0, "both", width=1.5),
        # an interactive user of a resident factorization: one right-hand side at a time
        _case("solve_512_1rhs", "solve", 10, 16, 1, 100.0, "point"),
        # a saturated server's batch: 768^2 with 24x24 leaves, 64 right-hand sides
        _case("solve_768_64rhs", "solve", 10, 24, 64, 150.0, "both"),
        # the headline's resident solve
        _case("solve_1024_32rhs", "solve", 12, 16, 32, 200.0, "plane"),
        # many media at once: trees of 128^2 to 512^2 (24^2 and 32^2 leaves) factored as one forest
        _case("forest_10", "forest", 4, 32, 1, 60.0, "point", trees=10),
        # 3D: the small cube and the largest one the interface limit admits, dense 4^3 leaves
        _case("cube_16_8rhs", "step", 6, 4, 8, 1.0, "both", d=3),
        _case("cube_32_8rhs", "step", 9, 4, 8, 1.0, "both", d=3),
    ]


# a forest's trees by turns: (L, leaf) of 128^2, 192^2, 256^2, 384^2 and 512^2
_FOREST = [(4, 32), (6, 24), (6, 32), (8, 24), (8, 32)]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ones' ranges, its cost bounded by the headline step's."""
    limit = work(_case(None, "step", 12, 16, 32, 200.0, "plane"))
    while True:
        kind = rng.choice(["step", "step", "step", "solve", "solve", "host", "mixed", "forest", "cube"])
        nrhs = _log_int(rng, 1, 64)
        rhs = rng.choice(["point", "plane", "both"])
        if kind == "cube":
            # leaves of 3 to 5 cells a side, 4 to 9 cuts
            c = _case(None, "step", rng.randint(4, 9), rng.randint(3, 5), min(nrhs, 32), round(rng.uniform(1.0, 4.0), 3),
                      rhs, d=3)
        elif kind == "forest":
            c = _case(None, "forest", 4, rng.randint(24, 32), rng.randint(1, 4), round(rng.uniform(20.0, 120.0), 2),
                      rhs, trees=rng.randint(4, 16))
        else:
            leaf = 16 if rng.random() < 0.4 else _log_int(rng, 8, 32)
            L = rng.randint(4, 12)
            c = _case(None, "step" if kind == "mixed" else kind, L, leaf, nrhs if kind != "host" else min(nrhs, 8), 0.0,
                      rhs, width=rng.choice([1.0, 1.0, 1.5]), precision="mixed" if kind == "mixed" else "fp64",
                      overlap=kind == "mixed" or rng.random() < 0.3)
            if kind in ("host", "solve"):
                c["overlap"] = False
        try:
            g = Geometry(c)
        except ValueError:
            continue
        if c["kb"] == 0.0:
            # 3 to 6 cells along a radian of the wave at kb, as the configurations have
            c["kb"] = round(rng.uniform(0.15, 0.3) * g.cells[0] / g.width, 2)
        if g.d == 2 and (max(g.leaf) > 40 or max(g.cells) > 1024 or min(g.cells) < 64):
            continue
        if g.d == 3 and (max(l["m"] for l in g.levels) > 1024 or g.nleaf_cells * g.nl < 512):
            continue
        w = work(c)
        # a host pass moves its arrays over PCIe at a hundredth of the memory rate
        if w["flops"] <= limit["flops"] and w["bytes"] * (40 if kind == "host" else 1) <= limit["bytes"]:
            return c


# ---------------------------------------------------------------------------------------------------
# geometry: leaves in depth-first order, the longest side cut first, faces x1 x2 y1 y2 (z1 z2)
# ---------------------------------------------------------------------------------------------------


class Geometry:
    def __init__(self, case):
        d, L = case["d"], case["L"]
        self.d, self.L, self.width = d, L, case["width"]
        size = [case["width"], 1.0, 1.0][:d]
        self.size = list(size)
        cuts, w = [], list(size)
        for _ in range(L):
            e = max(range(d), key=lambda j: (w[j], -j))
            cuts.append(e)
            w[e] *= 0.5
        self.cuts = cuts                       # cut axis of every level, the root's first
        # leaf cells: `leaf` along x, the others at the same spacing
        self.h_tgt = w[0] / (case["leaf"] - 0.4)
        self.leaf = [max(3, math.ceil(w[j] / self.h_tgt)) for j in range(d)]
        self.nleaf_cells = math.prod(self.leaf)
        self.parts = [2 ** sum(1 for e in cuts if e == j) for j in range(d)]
        self.cells = [self.parts[j] * self.leaf[j] for j in range(d)]
        if max(self.cells) > 4096:
            raise ValueError("grid too large")
        self.h = [w[j] / self.leaf[j] for j in range(d)]
        self.nl = 2 ** L
        pf = [self.nleaf_cells // self.leaf[j] for j in range(d)]
        self.face = [pf[f // 2] for f in range(2 * d)]
        self.off = [0] * (2 * d)
        for f in range(1, 2 * d):
            self.off[f] = self.off[f - 1] + self.face[f - 1]
        self.nb = sum(self.face)
        self.n = self.nb + self.nleaf_cells
        # merges: interface points m and the nodes' boundary points, per level
        self.levels = []
        for l in range(L):
            grid = [self.cells[j] // 2 ** sum(1 for e in cuts[:l + 1] if e == j) for j in range(d)]   # a child's
            nbc = 2 * sum(math.prod(grid) // grid[j] for j in range(d))
            m = math.prod(grid) // grid[cuts[l]]
            self.levels.append({"nodes": 2 ** l, "m": m, "nbc": nbc, "nb": 2 * (nbc - m)})
        self.root_nb = self.levels[0]["nb"]
        # integer position of every leaf
        pos = np.zeros((self.nl, d), dtype=np.int64)
        for l, e in enumerate(cuts):
            bit = (np.arange(self.nl) >> (L - 1 - l)) & 1
            pos[:, e] = 2 * pos[:, e] + bit
        self.pos = pos

    def interior(self, dev):
        """Cell centres (leaves in order, x fastest): a list of d tensors of nl * cells values."""
        pos = torch.from_numpy(self.pos).to(dev)
        grids = [torch.arange(m, device=dev, dtype=torch.float64) + 0.5 for m in self.leaf]
        out = []
        for j in range(self.d):
            shape = [1] * self.d
            shape[self.d - 1 - j] = self.leaf[j]
            g = grids[j].reshape(shape).expand(*reversed(self.leaf)).reshape(-1)
            out.append(((pos[:, j:j + 1] * self.leaf[j]).double() + g).reshape(-1) * self.h[j])
        return out

    def face_points(self, f):
        """Integer cell coordinates (tangential) of face f's points in the face's own order."""
        ax = f // 2
        tang = [j for j in range(self.d) if j != ax]
        idx = np.arange(self.face[f])
        c = np.zeros((self.face[f], self.d), dtype=np.int64)
        c[:, tang[0]] = idx % self.leaf[tang[0]]
        if self.d == 3:
            c[:, tang[1]] = idx // self.leaf[tang[0]]
        c[:, ax] = 0 if f % 2 == 0 else self.leaf[ax] - 1
        return c

    def boundary(self):
        """Root boundary: (coordinates (root_nb, d), outward normals (root_nb, d), leaf rows)."""
        X, N, rows = [], [], []
        for f in range(2 * self.d):
            ax, side = f // 2, f % 2
            c = self.face_points(f)
            for i in np.nonzero(self.pos[:, ax] == (self.parts[ax] - 1 if side else 0))[0]:
                x = (self.pos[i] * np.array(self.leaf) + c + 0.5) * np.array(self.h)
                x[:, ax] = self.size[ax] if side else 0.0
                nrm = np.zeros_like(x)
                nrm[:, ax] = 1.0 if side else -1.0
                X.append(x)
                N.append(nrm)
                rows.append(i * self.nb + self.off[f] + np.arange(self.face[f]))
        return np.concatenate(X), np.concatenate(N), np.concatenate(rows)

    def mates(self):
        """mate[leaf * nb + r]: the neighbour's row of the same interface point, -1 on the domain boundary."""
        where = {tuple(p): i for i, p in enumerate(self.pos.tolist())}
        mate = np.full(self.nl * self.nb, -1, dtype=np.int64)
        for i, p in enumerate(self.pos.tolist()):
            for f in range(2 * self.d):
                q = list(p)
                q[f // 2] += 1 if f % 2 else -1
                j = where.get(tuple(q))
                if j is None:
                    continue
                fo = f ^ 1
                r = np.arange(self.face[f])
                mate[i * self.nb + self.off[f] + r] = j * self.nb + self.off[fo] + r
        return mate


# ---------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------


def _inputs(case, g, seed, dev):
    """(potential (nl*cells), sources (nrhs, nl*cells), boundary data (nrhs, root_nb)), complex128."""
    rng = np.random.default_rng(seed)
    d, kb, nrhs = g.d, case["kb"], case["nrhs"]
    X = g.interior(dev)
    nb = 5 if d == 3 else max(5, int(g.cells[0] // 10))
    size = np.array(g.size)
    s = torch.zeros_like(X[0])
    for _ in range(nb):
        c = rng.uniform(0.2, 0.8, d) * size
        a = rng.uniform(-1.0, 1.0)
        r2 = sum((X[j] - c[j]) ** 2 for j in range(d))
        s += a * torch.exp(-r2 / (2 * 0.08 ** 2))
    damp = 0.01 if d == 3 else 0.005
    k = torch.complex(kb * (1.0 + 0.3 * s), torch.full_like(s, damp * kb))
    F = torch.zeros(nrhs, X[0].numel(), dtype=torch.complex128, device=dev)
    G = torch.zeros(nrhs, g.root_nb, dtype=torch.complex128, device=dev)
    bx, bn, _ = g.boundary()
    bx, bn = torch.from_numpy(bx).to(dev), torch.from_numpy(bn).to(dev)
    for r in range(nrhs):
        point = case["rhs"] == "point" or (case["rhs"] == "both" and r % 2 == 0)
        if point:
            c = rng.uniform(0.1, 0.9, d) * size
            r2 = sum((X[j] - c[j]) ** 2 for j in range(d))
            F[r] = torch.exp(-r2 / (2 * 0.05 ** 2))
        else:
            t = rng.normal(size=d)
            t = torch.from_numpy(t / np.linalg.norm(t)).to(dev)
            G[r] = 1j * kb * (bn @ t - 1.0) * torch.exp(1j * kb * (bx @ t))
    return k, F, G


def _subcases(case):
    """A forest's single trees (or the case itself)."""
    if case["kind"] != "forest":
        return [case]
    out = []
    for i in range(case["trees"]):
        L, leaf = _FOREST[i % len(_FOREST)]
        leaf = min(leaf, case["leaf"])
        out.append(dict(case, kind="step", L=L, leaf=leaf, trees=0))
    return out


def prepare(case, seed):
    import robinsolver_b200 as rb
    from robinsolver_b200 import _lib

    dev = torch.device("cuda", 0)
    parts = []
    for i, sub in enumerate(_subcases(case)):
        g = Geometry(sub)
        k, F, G = _inputs(sub, g, seed + 1000 * i, dev)
        # the impedance condition u_n - i kb u = g: opts.kb = -kb and the matching Robin pair
        okb = -sub["kb"] if g.d == 2 else sub["kb"]
        T = rb.robin_tree(async_factor=sub["overlap"])
        T.bndry_params = np.array([[1j * okb, 1.0], [-1j * okb, 1.0]], dtype=np.complex128)
        dom = np.zeros((2, 3))
        dom[1, :g.d] = g.size
        inf = T.plan(g.L, rb.elliptic_operator(d=g.d, domain=dom), rb.solve_opts(h_tgt=g.h_tgt, kb=okb))
        grid = [inf.leaf_a, inf.leaf_b, inf.leaf_c][:g.d]
        if grid != g.leaf or inf.root_nb != g.root_nb or inf.nleaves != g.nl:
            raise ValueError("the planned grid is not the case's")
        p = {"T": T, "k": k, "F": F, "G": G, "nrhs": sub["nrhs"], "prec": sub["precision"]}
        if case["kind"] == "host":
            p.update(k=k.cpu().numpy(), F=F.cpu().numpy(), G=G.cpu().numpy())
        else:
            p["u"] = torch.empty(sub["nrhs"], g.nl, g.n, dtype=torch.complex128, device=dev)
        parts.append(p)
    torch.cuda.synchronize()
    state = {"kind": case["kind"], "parts": parts, "lib": _lib.lib}
    if case["kind"] == "forest":
        state["forest"] = rb.robin_forest([p["T"] for p in parts])
        state["ptrs"] = [p["k"].data_ptr() for p in parts]
    if case["kind"] == "solve":
        p = parts[0]
        _ok(state, p, _lib.lib.rb_tree_factor_device(p["T"].handle, p["k"].data_ptr(), 0, 1))
    return state


def _ok(state, p, rc):
    if rc:
        raise RuntimeError(state["lib"].rb_last_error(p["T"].handle))


def _solve(state, p):
    lib, h = state["lib"], p["T"].handle
    _ok(state, p, lib.rb_tree_solve_device(h, p["nrhs"], p["F"].data_ptr(), p["G"].data_ptr(), 0))
    _ok(state, p, lib.rb_get_solution_device(h, p["u"].data_ptr(), 1))
    return p["u"]


def run(state):
    kind, parts, lib = state["kind"], state["parts"], state["lib"]
    p = parts[0]
    if kind == "host":
        p["T"].factor_samples(p["k"], p["prec"])
        p["T"].solve_samples(p["F"], p["G"])
        return [p["T"].solution_array(r) for r in range(p["nrhs"])]
    if kind == "forest":
        state["forest"].factor(state["ptrs"])
        return [_solve(state, q) for q in parts]
    if kind == "step":
        _ok(state, p, lib.rb_tree_factor_device(p["T"].handle, p["k"].data_ptr(), 1 if p["prec"] == "mixed" else 0, 0))
    return [_solve(state, p)]


# ---------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------


def work(case):
    flops = nbytes = 0.0
    for sub in _subcases(case):
        g = Geometry(sub)
        r, cells, nb = sub["nrhs"], g.nleaf_cells, g.nb
        a, rest = g.leaf[0], cells // g.leaf[0]
        # the kept factorization: leaf blocks (2D) or inverses (3D) with the outgoing rows, every
        # node's map, interface matrices and interface response
        if g.d == 2:
            leaf_store, leaf_flops = rest * a * a, 8.0 * a ** 3 * rest + 16.0 * a * a * nb * rest
            leaf_solve = 8.0 * (2 * rest * a * a + nb * cells)
        else:
            leaf_store, leaf_flops = g.n ** 2, 8.0 * g.n ** 3
            leaf_solve = 8.0 * (g.n ** 2 + nb * cells)
        store = g.nl * (leaf_store + nb * g.n)
        read = g.nl * (leaf_store + nb * cells)          # what a solve reads of it
        fac, sol = g.nl * leaf_flops, g.nl * leaf_solve
        for i, l in enumerate(g.levels):
            m, n = l["m"], l["nb"]
            fac += l["nodes"] * 8.0 * (2 * m ** 3 + 2.5 * m * m * n + m * n * n)
            sol += l["nodes"] * 8.0 * (3 * m * m + m * n + (2 * m * n if i else 0))
            store += l["nodes"] * (n * n + 3 * m * m + 2 * m * n)
            read += l["nodes"] * (3 * m * m + m * n + (2 * m * n if i else 0))
        io = r * (g.nl * cells + g.root_nb + g.nl * g.n)
        if case["kind"] == "solve":
            flops += r * sol
            nbytes += 16.0 * (read + io)
        else:
            flops += fac + r * sol
            nbytes += 16.0 * (g.nl * cells + store + io)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------------------------------
# the same solutions in plain torch: dense leaf solves, then the interface systems level by level
# ---------------------------------------------------------------------------------------------------


def _weights(i, m):
    if i == 0:
        return 8.0 / 3.0, -4.0, 4.0 / 3.0
    if i == m - 1:
        return 4.0 / 3.0, -4.0, 8.0 / 3.0
    return 1.0, -2.0, 1.0


def _leaf_matrix(g, kb):
    """The FD matrix of one leaf without its potential: boundary rows first, then the cells."""
    A = np.zeros((g.n, g.n), dtype=np.complex128)
    out = np.zeros((g.nb, g.n), dtype=np.complex128)       # outgoing Robin data of a leaf vector
    stride = [1, g.leaf[0], g.leaf[0] * g.leaf[1]][:g.d]
    cell = lambda c: g.nb + int(sum(c[j] * stride[j] for j in range(g.d)))  # noqa: E731
    face = {}                                               # (face, cell) -> boundary row
    for f in range(2 * g.d):
        ax = f // 2
        for t, c in enumerate(g.face_points(f)):
            r = g.off[f] + t
            face[f, cell(c)] = r
            inner = c.copy()
            inner[ax] += 1 if f % 2 == 0 else -1
            h = g.h[ax]
            for M, s in ((A, 1j * kb), (out, -1j * kb)):
                M[r, r] = s + 8.0 / 3.0 / h
                M[r, cell(c)] = -3.0 / h
                M[r, cell(inner)] = 1.0 / 3.0 / h
    for q in range(g.nleaf_cells):
        c = [q // stride[j] % g.leaf[j] for j in range(g.d)]
        e = g.nb + q
        for j in range(g.d):
            lo, mid, hi = (w / g.h[j] ** 2 for w in _weights(c[j], g.leaf[j]))
            A[e, e] += mid
            A[e, e - stride[j] if c[j] > 0 else face[2 * j, e]] += lo
            A[e, e + stride[j] if c[j] < g.leaf[j] - 1 else face[2 * j + 1, e]] += hi
    return A, out


def _exact_tree(case, seed, dev):
    g = Geometry(case)
    k, F, G = _inputs(case, g, seed, dev)
    okb = -case["kb"] if g.d == 2 else case["kb"]
    R, nl, nb, n = case["nrhs"], g.nl, g.nb, g.n
    A0, out = (torch.from_numpy(m).to(dev) for m in _leaf_matrix(g, okb))
    A = A0.repeat(nl, 1, 1)
    diag = torch.arange(nb, n, device=dev)
    A[:, diag, diag] += k.reshape(nl, -1)
    B = torch.zeros(nl, n, nb + R, dtype=torch.complex128, device=dev)
    B[:, torch.arange(nb), torch.arange(nb)] = 1.0
    B[:, nb:, nb:] = F.reshape(R, nl, -1).permute(1, 2, 0)
    X = torch.cat([torch.linalg.solve(a, b) for a, b in zip(A.split(256), B.split(256))])
    del A, B
    T = out @ X
    T, h = T[:, :, :nb].contiguous(), T[:, :, nb:].contiguous()
    # merges from the leaves up; zeta = 0, nu = -1: T1_ii g1 + h1 = -g2 and T2_ii g2 + h2 = -g1
    mate = g.mates()
    ids = np.arange(nb)                                    # node 0's boundary rows
    steps = []
    for l in range(g.L - 1, -1, -1):
        size = g.nl // 2 ** (l + 1) * nb                   # leaf rows of one child
        i1 = np.nonzero((mate[ids] >= size) & (mate[ids] < 2 * size))[0]
        at = {v: q for q, v in enumerate((ids + size).tolist())}
        i2 = np.array([at[v] for v in mate[ids[i1]].tolist()])
        r1, r2 = np.setdiff1d(np.arange(len(ids)), i1), np.setdiff1d(np.arange(len(ids)), i2)
        t = [torch.from_numpy(v).to(dev) for v in (i1, i2, r1, r2)]
        m, n1, n2 = len(i1), len(r1), len(r2)
        T1, T2, h1, h2 = T[0::2], T[1::2], h[0::2], h[1::2]
        pick = lambda M, a, b: M[:, a][:, :, b]            # noqa: E731
        nn = T1.shape[0]
        M = torch.zeros(nn, 2 * m, 2 * m, dtype=torch.complex128, device=dev)
        M[:, :m, :m] = -pick(T1, t[0], t[0])
        M[:, m:, m:] = -pick(T2, t[1], t[1])
        e = torch.arange(m, device=dev)
        M[:, e, m + e] = -1.0
        M[:, m + e, e] = -1.0
        B = torch.zeros(nn, 2 * m, n1 + n2 + R, dtype=torch.complex128, device=dev)
        B[:, :m, :n1] = pick(T1, t[0], t[2])
        B[:, m:, n1:n1 + n2] = pick(T2, t[1], t[3])
        B[:, :m, n1 + n2:] = h1[:, t[0]]
        B[:, m:, n1 + n2:] = h2[:, t[1]]
        Y = torch.cat([torch.linalg.solve(a, b) for a, b in zip(M.split(256), B.split(256))])
        del M, B
        steps.append((t, Y))
        if l:
            P = torch.cat([pick(T1, t[2], t[0]) @ Y[:, :m], pick(T2, t[3], t[1]) @ Y[:, m:]], 1)
            P[:, :n1, :n1] += pick(T1, t[2], t[2])
            P[:, n1:, n1:n1 + n2] += pick(T2, t[3], t[3])
            P[:, :n1, n1 + n2:] += h1[:, t[2]]
            P[:, n1:, n1 + n2:] += h2[:, t[3]]
            T, h = P[:, :, :n1 + n2].contiguous(), P[:, :, n1 + n2:].contiguous()
        ids = np.concatenate([ids[r1], ids[r2] + size])
    # the root's incoming data in its own order of points
    where = np.full(nl * nb, -1, dtype=np.int64)
    rows = g.boundary()[2]
    where[rows] = np.arange(len(rows))
    inc = G[:, torch.from_numpy(where[ids]).to(dev)].T[None]
    for t, Y in reversed(steps):
        i1, i2, r1, r2 = t
        m, n1, n2 = len(i1), len(r1), len(r2)
        gi = Y[:, :, :n1 + n2] @ inc + Y[:, :, n1 + n2:]
        nxt = torch.empty(2 * inc.shape[0], m + n1, R, dtype=torch.complex128, device=dev)
        nxt[0::2, i1], nxt[1::2, i2] = gi[:, :m], gi[:, m:]
        nxt[0::2, r1], nxt[1::2, r2] = inc[:, :n1], inc[:, n1:]
        inc = nxt
    u = X[:, :, :nb] @ inc + X[:, :, nb:]
    return u.permute(2, 0, 1).contiguous()


def exact(case, seed):
    dev = torch.device("cuda", 0)
    u = [_exact_tree(sub, seed + 1000 * i, dev) for i, sub in enumerate(_subcases(case))]
    if case["kind"] == "host":
        return [v.cpu().numpy() for v in u[0]]
    return u
