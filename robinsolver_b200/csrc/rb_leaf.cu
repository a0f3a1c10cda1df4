// rb_leaf.cu -- structured leaf factor and leaf solve for sm_100a.
//
// Leaf algebra.  The reference's leaf matrix A (FD_matrix_row, fd_module.f90:104-224) has its rows/
// columns in lin2fgrid order: the nb = 2(a+b) cornerless boundary points first (faces
// x1 x2 y1 y2), then the a*b interior points x-fastest.  Every boundary row r reads only
// itself and two interior points along the inward normal:
//     A(r,r) = i*kb + (8/3)/h,  A(r,p1) = -3/h,  A(r,p2) = (1/3)/h        (fd_module.f90:207-215)
// so A_bb is diagonal and the boundary unknowns condense exactly.  With
// d_r = A(r,r), c1 = -3/h, c2 = 1/(3h) and w_c = (8/3)/h^2 (the interior row next to boundary
// point c couples to it with that weight, fd_module.f90:150-153):
//     S      = A_ii - A_ib A_bb^-1 A_bi                       (a*b x a*b)
//     A^-1   = [[ (I - A_bi A^-1_ib) / d ,  -A_bi S^-1 / d ],
//               [ -S^-1 A_ib / d          ,   S^-1          ]]
// The reference's leaf Robin-to-Robin map is R X with X = A^-1 [I; 0] and R the outgoing rows
// sigma*u + tau*(8/3 u - 3 u_p1 + 1/3 u_p2)/h, sigma = -i*kb, tau = 1
// (RTR_update, robin_tree_module.f90:683-713).  Row r of Y = R A^-1 is
//     Y(r,:) = (sigma'_r / d_r) e_r + (2 i kb / d_r) (c1 A^-1(p1,:) + c2 A^-1(p2,:)),
// sigma'_r = sigma + (8/3)/h, because sigma'_r - d_r = -2 i kb.  Y(:, 0:nb) is the leaf RtR,
// Y(:, nb:n) maps an interior source to the outgoing data of the particular solution
// (fd_leaf_solve + fd_outgoing_bc, fd_module.f90:390-513).
//
// The condensed interior operator S inherits the 5-point stencil of FD_matrix_row
// (fd_module.f90:140-181): with the interior points ordered x-fastest (igrid2lin, fd_module.f90:835-841) it is block tridiagonal,
// b blocks of a x a,
//     S = tridiag(Lo_j, D_j, Up_j),  D_j tridiagonal,  Lo_j = diag(lam_j),  Up_j = diag(mu_j).
// Block elimination without exchanges between blocks (the blocks are diagonally dominant
// Laplacian blocks shifted by the potential; each block inverse pivots by |re|+|im|):
//     Sig_1 = D_1,  Sig_j = D_j - Lo_j Sig_{j-1}^-1 Up_{j-1},       S = L U,
//     L = [I; Lo_j Sig_{j-1}^-1 below],  U = [Sig_j; Up_j above].
// The leaf factor keeps Sig_j^-1 (b a^2 values instead of the reference's (ab+nb)^2 LU) and
// forms the Robin-to-Robin data Y = R A^-1 from Q = C S^-1, where row r of C is
// c1 e_p1(r) + c2 e_p2(r) (the interior part of the outgoing row of RTR_update,
// robin_tree_module.f90:699-713): Q^T = S^-T C^T by one block forward and one block backward
// sweep with nb right-hand sides.  Then, by the row formula above,
//     Y(r, nb+s) = f_r Q(r,s),   Y(r,c) = (sigma'_r/d_r) delta_rc - f_r (w_c/d_c) Q(r, p1(c)),
//     f_r = 2 i kb / d_r.
// The leaf solve applies A^-1 [g; f] (fd_leaf_solve + fd_leaf_update, fd_module.f90:390-566)
// through the same block factors: t = f - A_ib A_bb^-1 g, S u_i = t, u_b = (g - A_bi u_i)/d.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include "rb_gemm_dmma.cuh"   // dmma884
#include "rb_kernels.h"
#include "rb_pivot.cuh"

namespace rb {

__device__ __forceinline__ void leaf_bpoint2(int a, int b, int r, int& axis, int& p1, int& p2) {
    if (r < b) { axis = 0; p1 = r * a; p2 = r * a + 1; }
    else if (r < 2 * b) { const int j = r - b; axis = 0; p1 = j * a + (a - 1); p2 = j * a + (a - 2); }
    else if (r < 2 * b + a) { const int i = r - 2 * b; axis = 1; p1 = i; p2 = a + i; }
    else { const int i = r - 2 * b - a; axis = 1; p1 = (b - 1) * a + i; p2 = (b - 2) * a + i; }
}

__device__ __forceinline__ void stencil1(int i, int a, double& wm, double& w0, double& wp) {
    if (i == 1) { wm = 8.0 / 3.0; w0 = -4.0; wp = 4.0 / 3.0; }
    else if (i == a) { wm = 4.0 / 3.0; w0 = -4.0; wp = 8.0 / 3.0; }
    else { wm = 1.0; w0 = -2.0; wp = 1.0; }
}

// constants of one leaf's condensed stencil
struct LeafConst {
    double hx, hy, hx2, hy2;
    z rdx, rdy;                 // 1 / d for x-face and y-face boundary points
    double c1x, c2x, c1y, c2y;  // -3/h, 1/(3h)
    double wbx, wby;            // (8/3)/h^2
};

__device__ __forceinline__ LeafConst leaf_const(const double* hh, int leaf, double kb) {
    LeafConst c;
    c.hx = hh[2 * leaf];
    c.hy = hh[2 * leaf + 1];
    c.hx2 = c.hx * c.hx;
    c.hy2 = c.hy * c.hy;
    c.rdx = zrcp(zmk((8.0 / 3.0) / c.hx, kb));
    c.rdy = zrcp(zmk((8.0 / 3.0) / c.hy, kb));
    c.c1x = -3.0 / c.hx; c.c2x = (1.0 / 3.0) / c.hx;
    c.c1y = -3.0 / c.hy; c.c2y = (1.0 / 3.0) / c.hy;
    c.wbx = (8.0 / 3.0) / c.hx2;
    c.wby = (8.0 / 3.0) / c.hy2;
    return c;
}

// entry (r, c) of the diagonal block D_j (grid row jj = j+1) of S
__device__ __forceinline__ z block_d(const LeafConst& L, int a, int b, int jj, int r, int c, z k) {
    const int i = r + 1;
    double wxm, wx0, wxp, wym, wy0, wyp;
    stencil1(i, a, wxm, wx0, wxp);
    stencil1(jj, b, wym, wy0, wyp);
    z v = zmk(0.0, 0.0);
    if (c == r) {
        v = zmk((k.x + wx0 / L.hx2) + wy0 / L.hy2, k.y);
        if (i == 1 || i == a) v = zsub(v, zscale(L.wbx * L.c1x, L.rdx));
        if (jj == 1 || jj == b) v = zsub(v, zscale(L.wby * L.c1y, L.rdy));
    } else if (c == r + 1 && i < a) {
        v = zmk(wxp / L.hx2, 0.0);
        if (i == 1) v = zsub(v, zscale(L.wbx * L.c2x, L.rdx));
    } else if (c == r - 1 && i > 1) {
        v = zmk(wxm / L.hx2, 0.0);
        if (i == a) v = zsub(v, zscale(L.wbx * L.c2x, L.rdx));
    }
    return v;
}
// Lo_j(i,i) = S(e, e-a) for grid row jj >= 2 and Up_j(i,i) = S(e, e+a) for jj <= b-1
__device__ __forceinline__ z block_lo(const LeafConst& L, int b, int jj) {
    double wm, w0, wp;
    stencil1(jj, b, wm, w0, wp);
    z v = zmk(wm / L.hy2, 0.0);
    if (jj == b) v = zsub(v, zscale(L.wby * L.c2y, L.rdy));
    return v;
}
__device__ __forceinline__ z block_up(const LeafConst& L, int b, int jj) {
    double wm, w0, wp;
    stencil1(jj, b, wm, w0, wp);
    z v = zmk(wp / L.hy2, 0.0);
    if (jj == 1) v = zsub(v, zscale(L.wby * L.c2y, L.rdy));
    return v;
}

// Lo_j and Up_j of every block, formed once (block_lo and block_up divide)
struct BlockCoupling {
    z lo_in, lo_last, up_first, up_in;
    int b;
    __device__ __forceinline__ BlockCoupling(const LeafConst& L, int b_) : b(b_) {
        lo_in = up_in = zmk(1.0 / L.hy2, 0.0);       // stencil1 inside
        lo_last = block_lo(L, b, b);
        up_first = block_up(L, b, 1);
    }
    __device__ __forceinline__ z lo(int jj) const { return jj == b ? lo_last : lo_in; }
    __device__ __forceinline__ z up(int jj) const { return jj == 1 ? up_first : up_in; }
};

// In-place Gauss-Jordan inverse of an m x m column-major matrix in shared memory by the whole
// CTA (partial pivoting by |re|+|im|, first maximum).  Returns false on an exactly zero pivot.
__device__ bool cta_gj_invert(z* S, int m, z* fcol, int* ipiv, int* sp) {
    const int tid = threadIdx.x, nt = blockDim.x;
    bool ok = true;
    for (int k = 0; k < m; ++k) {
        if (tid < 32) {
            double best = -1.0;
            int bi = m;
            for (int r = k + tid; r < m; r += 32) {
                const double v = zabs1(S[r + k * m]);
                if (v > best) { best = v; bi = r; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double ov = __shfl_down_sync(0xffffffffu, best, o);
                const int oi = __shfl_down_sync(0xffffffffu, bi, o);
                if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
            }
            if (tid == 0) { *sp = bi; ipiv[k] = bi; }
        }
        __syncthreads();
        const int p = *sp;
        if (p != k)
            for (int c = tid; c < m; c += nt) {
                const z t = S[k + c * m];
                S[k + c * m] = S[p + c * m];
                S[p + c * m] = t;
            }
        __syncthreads();
        const z piv = S[k + k * m];
        if (piv.x == 0.0 && piv.y == 0.0) ok = false;
        const z pinv = zrcp(piv);
        for (int i = tid; i < m; i += nt) fcol[i] = S[i + k * m];
        __syncthreads();
        for (int c = tid; c < m; c += nt) S[k + c * m] = (c == k) ? pinv : zmul(S[k + c * m], pinv);
        __syncthreads();
        for (int e = tid; e < m * m; e += nt) {
            const int i = e % m, c = e / m;
            if (i == k) continue;
            const z f = fcol[i];
            if (c == k) S[e] = zneg(zmul(f, pinv));
            else zfms(S[e], f, S[k + c * m]);
        }
        __syncthreads();
    }
    for (int r = tid; r < m; r += nt)
        for (int k = m - 1; k >= 0; --k) {
            const int p = ipiv[k];
            if (p != k) {
                const z t = S[r + k * m];
                S[r + k * m] = S[r + p * m];
                S[r + p * m] = t;
            }
        }
    __syncthreads();
    return ok;
}

// ---------------------------------------------------------------------------------------------------
// Leaf factor: Sig_j^-1 for every block and Y = R A^-1 (nb x n, ld nb).  Shared memory:
// sig (a^2), sigp (a^2), v0, v1 (a x nb each), fcol (a), ipiv (a), sp.
__global__ void __launch_bounds__(256) leaf_block_factor_kernel(LeafGeom g, const double* __restrict__ hh,
                                                                const z* __restrict__ kv, z* __restrict__ sinv,
                                                                z* __restrict__ Y, int* status) {
    extern __shared__ z sm[];
    const int leaf = blockIdx.x;
    const int a = g.a, b = g.b, nb = g.nb, n = g.n, ab = a * b, aa = a * a;
    const int tid = threadIdx.x, nt = blockDim.x;
    z* sig = sm;
    z* sigp = sig + aa;
    z* v0 = sigp + aa;
    z* v1 = v0 + (size_t)a * nb;
    z* fcol = v1 + (size_t)a * nb;
    int* ipiv = reinterpret_cast<int*>(fcol + a);
    int* sp = ipiv + a;
    const LeafConst L = leaf_const(hh, leaf, g.kb);
    const z* kl = kv + (size_t)leaf * ab;
    z* Sl = sinv + (size_t)leaf * b * aa;
    z* Yl = Y + (size_t)leaf * nb * n;
    bool ok = true;

    // ---- block LU: Sig_j^-1, j = 0..b-1 ------------------------------------------------------
    for (int j = 0; j < b; ++j) {
        const int jj = j + 1;
        const z lam = jj > 1 ? block_lo(L, b, jj) : zmk(0.0, 0.0);
        const z mup = jj > 1 ? block_up(L, b, jj - 1) : zmk(0.0, 0.0);
        for (int e = tid; e < aa; e += nt) {
            const int r = e % a, c = e / a;
            z v = block_d(L, a, b, jj, r, c, kl[j * a + r]);
            if (jj > 1) zfms(v, zmul(lam, mup), sigp[e]);
            sig[e] = v;
        }
        __syncthreads();
        ok &= cta_gj_invert(sig, a, fcol, ipiv, sp);
        for (int e = tid; e < aa; e += nt) {
            Sl[(size_t)j * aa + e] = sig[e];
            sigp[e] = sig[e];
        }
        __syncthreads();
    }

    // ---- forward sweep of S^T Z = C^T: v_j = Sig_j^-T (c_j - Up_{j-1} v_{j-1}) ---------------------
    // v_j (a x nb, ld a) is kept in shared memory and stored transposed into Y(:, nb + j*a + i).
    z* vp = v0;
    z* vc = v1;
    for (int j = 0; j < b; ++j) {
        const int jj = j + 1;
        for (int e = tid; e < aa; e += nt) sig[e] = Sl[(size_t)j * aa + e];
        const z mup = jj > 1 ? block_up(L, b, jj - 1) : zmk(0.0, 0.0);
        __syncthreads();
        for (int e = tid; e < a * nb; e += nt) {
            const int i = e % a, r = e / a;
            int ax, p1, p2;
            leaf_bpoint2(a, b, r, ax, p1, p2);
            const double hr = ax == 0 ? L.hx : L.hy;
            const double c1 = -3.0 / hr, c2 = (1.0 / 3.0) / hr;
            z acc = zmk(0.0, 0.0);
            for (int q = 0; q < a; ++q) {
                const int eq = j * a + q;
                z rhs = zmk((eq == p1 ? c1 : 0.0) + (eq == p2 ? c2 : 0.0), 0.0);
                if (jj > 1) zfms(rhs, mup, vp[q + r * a]);
                zfma(acc, sig[q + i * a], rhs);       // (Sig^-T)(i,q) = Sig^-1(q,i)
            }
            vc[e] = acc;
            Yl[r + (size_t)(nb + j * a + i) * nb] = acc;
        }
        __syncthreads();
        z* t = vp; vp = vc; vc = t;
    }
    // ---- backward sweep: z_{j-1} = v_{j-1} - Sig_{j-1}^-T Lo_j z_j; z_{b-1} = v_{b-1} (in vp) -------
    for (int j = b - 1; j >= 1; --j) {
        const int jj = j + 1;              // grid row of block j
        const z lam = block_lo(L, b, jj);
        for (int e = tid; e < aa; e += nt) sig[e] = Sl[(size_t)(j - 1) * aa + e];
        __syncthreads();
        for (int e = tid; e < a * nb; e += nt) {
            const int i = e % a, r = e / a;
            z acc = Yl[r + (size_t)(nb + (j - 1) * a + i) * nb];
            for (int q = 0; q < a; ++q) zfms(acc, sig[q + i * a], zmul(lam, vp[q + r * a]));
            vc[e] = acc;
            Yl[r + (size_t)(nb + (j - 1) * a + i) * nb] = acc;
        }
        __syncthreads();
        z* t = vp; vp = vc; vc = t;
    }
    __syncthreads();
    // ---- Y = R A^-1 from Q(r, s) = Z(s, r) = Y(r, nb+s) -------------------------------------------
    for (int e = tid; e < nb * nb; e += nt) {
        const int r = e % nb, c = e / nb;
        int ax, p1, p2, axc, p1c, p2c;
        leaf_bpoint2(a, b, r, ax, p1, p2);
        leaf_bpoint2(a, b, c, axc, p1c, p2c);
        const z rd = ax == 0 ? L.rdx : L.rdy;
        const z f = zmul(zmk(0.0, 2.0 * g.kb), rd);
        const z wd = axc == 0 ? zscale(L.wbx, L.rdx) : zscale(L.wby, L.rdy);
        z v = zneg(zmul(zmul(f, wd), Yl[r + (size_t)(nb + p1c) * nb]));
        if (c == r) {
            const double hr = ax == 0 ? L.hx : L.hy;
            v = zadd(v, zmul(zmk((8.0 / 3.0) / hr, -g.kb), rd));
        }
        Yl[e] = v;
    }
    __syncthreads();
    for (int e = tid; e < nb * ab; e += nt) {
        const int r = e % nb;
        int ax, p1, p2;
        leaf_bpoint2(a, b, r, ax, p1, p2);
        const z f = zmul(zmk(0.0, 2.0 * g.kb), ax == 0 ? L.rdx : L.rdy);
        Yl[(size_t)nb * nb + e] = zmul(f, Yl[(size_t)nb * nb + e]);
    }
    if (!ok && tid == 0) atomicOr(status, 1);
}

size_t leaf_block_factor_smem(const LeafGeom& g) {
    return (2 * (size_t)g.a * g.a + 2 * (size_t)g.a * g.nb + g.a) * sizeof(z) + (g.a + 1) * sizeof(int) + 16;
}

// ---------------------------------------------------------------------------------------------------
// Leaf factor for blocks of up to 32 x 32 in two kernels: the chain of block inverses, then the
// sweeps of S^T Z = C^T, whose right-hand sides are independent of one another.
//
// leaf_chain: Sig_j^-1 for j = 0..b-1.  Each Sig_j needs Sig_{j-1}^-1, so a leaf is a chain of a*b
// pivot steps (rb_pivot.cuh), and the time of a step is what counts.  The row and column orders are
// restored once per block, on the way through shared memory.
// Latency-bound: 4.3 us a block of 16 rows (69 us a 16x16 leaf, 345 us for 4096 leaves), 13.9 us a
// block of 32 (445 us a 32x32 leaf).  One warp or CTA forming Sig_j^-1 and both sweeps of a leaf took
// 406 us for 16 leaves of 16x16 (now 105 with leaf_sweep), 2.25 ms for 4096 (now 1.28), and 6.6 ms
// for 64 leaves of 32x32 (now 0.71).

// what one row of the diagonal blocks D_j is made of, formed once per leaf: the chain pays for
// every division of a block
struct ChainRow {
    double wx0, wy_in, wy_end;   // diagonal stencil weights over h^2: x; y of an inner and of an end block
    z dx, dy;                    // what the condensed x (end rows) and y (end blocks) faces take off
    z up, lo;                    // right and left neighbour
    z lm_first, lm_in, lm_last;  // Lo_j Up_{j-1} of block 1, an inner block and block b-1
};
__device__ __forceinline__ ChainRow chain_row(const LeafConst& L, int a, int b, int r) {
    ChainRow c;
    double wm, w0, wp;
    stencil1(r + 1, a, wm, w0, wp);
    c.wx0 = w0 / L.hx2;
    c.up = zmk(wp / L.hx2, 0.0);
    c.lo = zmk(wm / L.hx2, 0.0);
    c.dx = zmk(0.0, 0.0);
    if (r == 0 || r == a - 1) {
        c.dx = zscale(L.wbx * L.c1x, L.rdx);
        const z n = zscale(L.wbx * L.c2x, L.rdx);
        if (r == 0) c.up = zsub(c.up, n);
        if (r == a - 1) c.lo = zsub(c.lo, n);
    }
    stencil1(2, b, wm, w0, wp);
    c.wy_in = w0 / L.hy2;
    stencil1(1, b, wm, w0, wp);
    c.wy_end = w0 / L.hy2;
    c.dy = zscale(L.wby * L.c1y, L.rdy);
    c.lm_first = zmul(block_lo(L, b, 2), block_up(L, b, 1));
    c.lm_in = b > 3 ? zmul(block_lo(L, b, 3), block_up(L, b, 2)) : zmk(0.0, 0.0);
    c.lm_last = zmul(block_lo(L, b, b), block_up(L, b, b - 1));
    return c;
}

// the entries of row r at columns c0..c0+7 of D_j, minus Lo_j Up_{j-1} prev
__device__ __forceinline__ void chain_form(const ChainRow& cr, int a, int b, int j, int r, int c0, z k,
                                           const z (&prev)[PV_CG], z (&v)[PV_CG]) {
    const bool end = j == 0 || j == b - 1;
    z d = zsub(zmk((k.x + cr.wx0) + (end ? cr.wy_end : cr.wy_in), k.y), cr.dx);
    if (end) d = zsub(d, cr.dy);
    const z lm = j == 0 ? zmk(0.0, 0.0) : j == b - 1 ? cr.lm_last : j == 1 ? cr.lm_first : cr.lm_in;
#pragma unroll
    for (int e = 0; e < PV_CG; ++e) {
        const int c = c0 + e;
        z x = c == r ? d : c == r + 1 ? cr.up : c == r - 1 ? cr.lo : zmk(0.0, 0.0);
        zfms(x, lm, prev[e]);                        // prev is zero before block 1
        v[e] = r < a && c < a ? x : zmk(0.0, 0.0);
    }
}

// Blocks of up to 16 rows: one warp per leaf, lane = row + 16 * column group, no block barriers.
__global__ void __launch_bounds__(128) leaf_chain16_kernel(LeafGeom g, int nleaves, const double* __restrict__ hh,
                                                           const z* __restrict__ kv, z* __restrict__ sinv, int* status) {
    __shared__ z blk[4][256];
    __shared__ z prow[4][32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int leaf = blockIdx.x * (blockDim.x >> 5) + wib;
    if (leaf >= nleaves) return;
    const int a = g.a, b = g.b, aa = a * a;
    z* sm = blk[wib];
    const LeafConst L = leaf_const(hh, leaf, g.kb);
    const z* kl = kv + (size_t)leaf * a * b;
    z* Sl = sinv + (size_t)leaf * b * aa;
    const int r = lane & 15, hf = lane >> 4;
    const ChainRow cr = chain_row(L, a, b, r);
    z v[PV_CG], prev[PV_CG];
#pragma unroll
    for (int e = 0; e < PV_CG; ++e) prev[e] = zmk(0.0, 0.0);
    bool ok = true;
    z kn = r < a ? kl[r] : zmk(0.0, 0.0);
    for (int j = 0; j < b; ++j) {
        chain_form(cr, a, b, j, r, PV_CG * hf, kn, prev, v);
        if (j + 1 < b && r < a) kn = kl[(j + 1) * a + r];          // the next block's potential
        int myk, pk;
        if (!warp_invert16(v, a, prow[wib], myk, pk)) ok = false;
#pragma unroll
        for (int e = 0; e < PV_CG; ++e) {
            const int q = hf * PV_CG + e;
            const int pq = __shfl_sync(0xffffffffu, pk, q);
            if (r < a && q < a) sm[myk + pq * a] = v[e];
        }
        __syncwarp();
#pragma unroll
        for (int e = 0; e < PV_CG; ++e) {
            const int q = hf * PV_CG + e;
            if (r < a && q < a) {
                prev[e] = sm[r + q * a];
                Sl[(size_t)j * aa + r + q * a] = prev[e];
            }
        }
        __syncwarp();
    }
    if (!ok) atomicOr(status, RB_STATUS_ZERO_PIVOT);
}

// Blocks of 17 to 32 rows: one CTA of NG warps per leaf, lane = row, warp = column group.
template <int NG>
__global__ void __launch_bounds__(32 * NG) leaf_chain32_kernel(LeafGeom g, const double* __restrict__ hh,
                                                               const z* __restrict__ kv, z* __restrict__ sinv,
                                                               int* status) {
    __shared__ z sm[32 * 32];
    __shared__ PivotShared<1, NG> sh;
    const int leaf = blockIdx.x;
    const int r = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int a = g.a, b = g.b, aa = a * a;
    const LeafConst L = leaf_const(hh, leaf, g.kb);
    const z* kl = kv + (size_t)leaf * a * b;
    z* Sl = sinv + (size_t)leaf * b * aa;
    const ChainRow cr = chain_row(L, a, b, r);
    z v[1][PV_CG], prev[PV_CG];
#pragma unroll
    for (int e = 0; e < PV_CG; ++e) prev[e] = zmk(0.0, 0.0);
    bool ok = true;
    z kn = r < a ? kl[r] : zmk(0.0, 0.0);
    for (int j = 0; j < b; ++j) {
        chain_form(cr, a, b, j, r, PV_CG * w, kn, prev, v[0]);
        if (j + 1 < b && r < a) kn = kl[(j + 1) * a + r];
        int myk[1];
        if (!cta_invert<1, NG>(v, a, sh, myk)) ok = false;
#pragma unroll
        for (int e = 0; e < PV_CG; ++e) {
            const int q = w * PV_CG + e;
            if (r < a && q < a) sm[myk[0] + sh.pk[q] * a] = v[0][e];
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < PV_CG; ++e) {
            const int q = w * PV_CG + e;
            if (r < a && q < a) {
                prev[e] = sm[r + q * a];
                Sl[(size_t)j * aa + r + q * a] = prev[e];
            }
        }
        // sm is written again only after the next block's barriers
    }
    if (!ok) atomicOr(status, RB_STATUS_ZERO_PIVOT);
}

// leaf_sweep: Y = R A^-1 from the block inverses.  The sweeps of S^T Z = C^T treat every
// right-hand side (a boundary point, a row of Y) alone, so a warp takes 8 of them through all
// 2b - 1 block steps with the running block vector in registers:
//   forward:  R_0 = C_0;  V_j = Sig_j^-T R_j;  R_{j+1} = C_{j+1} - Up_j V_j
//   backward: Z_{b-1} = V_{b-1};  Z_{j-1} = V_{j-1} - Sig_{j-1}^-T (Lo_j Z_j)
// A step is V^T (8 x a) = R^T (8 x a) Sig_j^-1 (a x a) on the FP64 tensor cores (m8n8k4, four real
// products per complex one).  The k order of the MMAs is chosen so that the accumulator layout
// (row lane/4, columns 2 (lane%4) + {0,1}) is the next step's A fragment as it stands: k-step
// (t, h) sums the rows q = 8t + 2 (lane%4) + h of the block, so nothing moves between steps.  The
// blocks stream through shared memory in a ring of cp.async stages, padded with zeros to multiples of
// 8 and with an odd leading dimension (conflict-free 16-byte fragment loads).
// Measured: 16 leaves of 16x16 36 us, 4096 of them 0.93 ms (17.2 GFLOP, 18 TFLOP/s; two CTAs of 8 warps
// per SM, three spill: 1.02); 64 leaves of 32x32 260 us.
// C_j holds, per right-hand side, c1 and c2 at the interior points next to its boundary point.
template <int NT>
struct SweepCfg {
    static constexpr int AP = 8 * NT;            // padded block size
    static constexpr int LD = AP + 1;
    static constexpr int STAGES = NT <= 2 ? 4 : 3;
    static constexpr size_t SMEM = STAGES * (size_t)AP * LD * sizeof(z);
};

// The ring of a leaf's blocks in the order of a forward and a backward sweep: 0..b-1, b-2..0.
template <int NT>
struct BlockRing {
    using Cfg = SweepCfg<NT>;
    z* sm;
    const z* Sl;
    int a, aa, b, nsteps;
    __device__ __forceinline__ void issue(int st) {
        if (st < nsteps) {
            const int j = st < b ? st : 2 * b - 2 - st;
            const z* src = Sl + (size_t)j * aa;
            z* dst = sm + (st % Cfg::STAGES) * Cfg::AP * Cfg::LD;
            // a warp copies CPW columns at a time (no division by a: one warp may copy it all)
            constexpr int CPW = NT == 1 ? 4 : NT == 2 ? 2 : 1;
            const int i = threadIdx.x & (32 / CPW - 1);
            if (i < a)
                for (int c = threadIdx.x / (32 / CPW); c < a; c += blockDim.x / (32 / CPW))
                    cp_async16(dst + i + c * Cfg::LD, src + i + c * a, 16);
        }
        cp_async_commit();
    }
    __device__ __forceinline__ void start() {
        for (int e = threadIdx.x; e < Cfg::STAGES * Cfg::AP * Cfg::LD; e += blockDim.x) sm[e] = zmk(0.0, 0.0);
        __syncthreads();
        for (int st = 0; st < Cfg::STAGES - 1; ++st) issue(st);
    }
    // the block of step st, and the fetch of the block STAGES - 1 steps on
    __device__ __forceinline__ const z* next(int st) {
        cp_async_wait<Cfg::STAGES - 2>();
        __syncthreads();               // block st landed; every warp is past step st-1's reads
        issue(st + Cfg::STAGES - 1);
        return sm + (st % Cfg::STAGES) * Cfg::AP * Cfg::LD;
    }
};

template <int NT>
__global__ void __launch_bounds__(256, NT <= 3 ? 2 : 1) leaf_sweep_kernel(LeafGeom g, int nchunk, const double* __restrict__ hh,
                                                         const z* __restrict__ sinv, z* __restrict__ Y) {
    using Cfg = SweepCfg<NT>;
    constexpr int LD = Cfg::LD;
    extern __shared__ z sm[];
    const int nthr = blockDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lr = lane >> 2, lc = lane & 3;
    const int leaf = blockIdx.x / nchunk, chunk = blockIdx.x % nchunk;
    const int a = g.a, b = g.b, nb = g.nb, n = g.n, aa = a * a;
    const LeafConst L = leaf_const(hh, leaf, g.kb);
    const z* Sl = sinv + (size_t)leaf * b * aa;
    z* Yl = Y + (size_t)leaf * nb * n;
    const int nsteps = 2 * b - 1;
    BlockRing<NT> ring{sm, Sl, a, aa, b, nsteps};
    ring.start();
    const BlockCoupling cpl(L, b);
    // this lane's right-hand side and its two interior points
    const int row = (chunk * (nthr >> 5) + warp) * 8 + lr;
    const bool live = row < nb;
    int ax, q1, q2;
    leaf_bpoint2(a, b, live ? row : 0, ax, q1, q2);
    const double h = ax == 0 ? L.hx : L.hy;
    const double c1 = live ? -3.0 / h : 0.0, c2 = live ? (1.0 / 3.0) / h : 0.0;
    const z rd = ax == 0 ? L.rdx : L.rdy;
    const z fc = zmul(zmk(0.0, 2.0 * g.kb), rd);                      // Y(r, nb+s) = f_r Q(r, s)
    const z dg = zmul(zmk((8.0 / 3.0) / h, -g.kb), rd);               // (sigma'_r / d_r)
    const z wdx = zscale(L.wbx, L.rdx), wdy = zscale(L.wby, L.rdy);
    z* Yr = Yl + (live ? row : 0);
    // the final value s = Y(row, nb + j a + i): it, and its multiples in the boundary columns
    auto store = [&](int j, int i, z s) {
        Yr[(size_t)(nb + j * a + i) * nb] = s;
        auto bcol = [&](int c, z wd) {
            z v = zneg(zmul(wd, s));
            if (c == row) v = zadd(v, dg);
            Yr[(size_t)c * nb] = v;
        };
        if (i == 0) bcol(j, wdx);
        if (i == a - 1) bcol(b + j, wdx);
        if (j == 0) bcol(2 * b + i, wdy);
        if (j == b - 1) bcol(2 * b + a + i, wdy);
    };
    double rre[2 * NT], rim[2 * NT];                 // R^T, [2t + h]: column 8t + 2lc + h
    z vn[2 * NT];                                    // the backward step's V, fetched a step ahead
#pragma unroll
    for (int e = 0; e < 2 * NT; ++e) {
        const int q = 8 * (e >> 1) + 2 * lc + (e & 1);
        rre[e] = q < a ? (q == q1 ? c1 : 0.0) + (q == q2 ? c2 : 0.0) : 0.0;
        rim[e] = 0.0;
        vn[e] = zmk(0.0, 0.0);
    }
    for (int st = 0; st < nsteps; ++st) {
        const bool fwd = st < b;
        const int j = fwd ? st : 2 * b - 2 - st;
        const z* S = ring.next(st) + 2 * lc + lr * LD;
        double cre[NT][2], cim[NT][2];
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                cre[t][q] = fwd ? 0.0 : vn[2 * t + q].x;
                cim[t][q] = fwd ? 0.0 : vn[2 * t + q].y;
            }
        // the V of the next backward step: block b-2 first (written two steps before)
        if (st + 1 >= b && st + 1 < nsteps) {
            const int jn = 2 * b - 3 - st;
#pragma unroll
            for (int e = 0; e < 2 * NT; ++e) {
                const int i = 8 * (e >> 1) + 2 * lc + (e & 1);
                vn[e] = (live && i < a) ? Yr[(size_t)(nb + jn * a + i) * nb] : zmk(0.0, 0.0);
            }
        }
#pragma unroll
        for (int e = 0; e < 2 * NT; ++e) {           // k-step (t, h): rows 8t + 2lc + h of the block
            z bf[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) bf[t] = S[8 * (e >> 1) + (e & 1) + 8 * t * LD];
#pragma unroll
            for (int t = 0; t < NT; ++t) dmma884(cre[t][0], cre[t][1], rre[e], bf[t].x);
#pragma unroll
            for (int t = 0; t < NT; ++t) dmma884(cim[t][0], cim[t][1], rre[e], bf[t].y);
#pragma unroll
            for (int t = 0; t < NT; ++t) dmma884(cre[t][0], cre[t][1], -rim[e], bf[t].y);
#pragma unroll
            for (int t = 0; t < NT; ++t) dmma884(cim[t][0], cim[t][1], rim[e], bf[t].x);
        }
        // next R: C_{j+1} - Up_j V_j forward, -Lo_j Z_j backward (Lo_j couples block j to j-1)
        const bool up = fwd && j + 1 < b;
        const z co = up ? cpl.up(j + 1) : cpl.lo(j + 1);
        const bool fin = !up;
        const int qn = (j + 1) * a;
#pragma unroll
        for (int e = 0; e < 2 * NT; ++e) {
            const int i = 8 * (e >> 1) + 2 * lc + (e & 1);
            z s = zmk(cre[e >> 1][e & 1], cim[e >> 1][e & 1]);
            z nx = zneg(zmul(co, s));
            if (up && i < a) nx.x += (qn + i == q1 ? c1 : 0.0) + (qn + i == q2 ? c2 : 0.0);
            rre[e] = nx.x;
            rim[e] = nx.y;
            if (live && i < a) {
                if (fin) store(j, i, zmul(fc, s));
                else Yr[(size_t)(nb + j * a + i) * nb] = s;
            }
        }
    }
}

template <int NT>
static cudaError_t launch_sweep(const LeafGeom& g, int nleaves, const double* h, const z* sinv, z* Y, cudaStream_t s) {
    const int units = (g.nb + 7) / 8;                // warps a leaf needs
    // few leaves: two warps per CTA, to spread a leaf over several SMs; many: up to eight, which
    // share each staged block
    const int wpc = std::min(units, (long long)nleaves * units <= 8 * 148 ? 2 : 8);
    const int nchunk = (units + wpc - 1) / wpc;
    static DeviceAttrCache attr;
    cudaError_t e = ensure_smem_attr(leaf_sweep_kernel<NT>, SweepCfg<NT>::SMEM, attr);
    if (e != cudaSuccess) return e;
    leaf_sweep_kernel<NT><<<(unsigned)nleaves * nchunk, 32 * wpc, SweepCfg<NT>::SMEM, s>>>(g, nchunk, h, sinv, Y);
    note_launch();
    return cudaGetLastError();
}

cudaError_t leaf_block_factor(const LeafGeom& g, int nleaves, const double* h, const z* k, z* sinv, z* Y,
                              int* status, cudaStream_t s) {
    const size_t sh = leaf_block_factor_smem(g);
    if (g.a <= 32) {
        // The leaf grids this library accepts stay those that fit the one-CTA form below, and all that are 16
        // wide, although these kernels need less.
        if (g.a != 16 && sh > (size_t)227 * 1024) return cudaErrorInvalidValue;
        if (g.a <= 16) {
            const int wpc = nleaves >= 4 * 148 ? 4 : 1;
            leaf_chain16_kernel<<<(nleaves + wpc - 1) / wpc, 32 * wpc, 0, s>>>(g, nleaves, h, k, sinv, status);
        } else if (g.a <= 24) {
            leaf_chain32_kernel<3><<<nleaves, 96, 0, s>>>(g, h, k, sinv, status);
        } else {
            leaf_chain32_kernel<4><<<nleaves, 128, 0, s>>>(g, h, k, sinv, status);
        }
        note_launch();
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        if (g.a <= 8) return launch_sweep<1>(g, nleaves, h, sinv, Y, s);
        if (g.a <= 16) return launch_sweep<2>(g, nleaves, h, sinv, Y, s);
        if (g.a <= 24) return launch_sweep<3>(g, nleaves, h, sinv, Y, s);
        return launch_sweep<4>(g, nleaves, h, sinv, Y, s);
    }
    if (sh > 48 * 1024) {
        static DeviceAttrCache attr;
        cudaError_t e = ensure_smem_attr(leaf_block_factor_kernel, sh, attr);
        if (e != cudaSuccess) return e;
    }
    leaf_block_factor_kernel<<<nleaves, 256, sh, s>>>(g, h, k, sinv, Y, status);
    note_launch();
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------------
// Leaf solve: u = A^-1 [g; f] for every leaf and right-hand side into sol [rhs][leaf][n].
// RHS are processed in chunks of KC columns; shared memory: sig (a^2), w0, w1 (a x KC each).
constexpr int LEAF_KC = 32;

__global__ void __launch_bounds__(256) leaf_block_solve_kernel(LeafGeom g, int nleaves, int nrhs,
                                                               const double* __restrict__ hh,
                                                               const z* __restrict__ f, const z* __restrict__ gb,
                                                               const z* __restrict__ sinv, z* __restrict__ sol) {
    extern __shared__ z sm[];
    const int leaf = blockIdx.x;
    const int a = g.a, b = g.b, nb = g.nb, n = g.n, ab = a * b, aa = a * a;
    const int tid = threadIdx.x, nt = blockDim.x;
    z* sig = sm;
    z* w0 = sig + aa;
    z* w1 = w0 + (size_t)a * LEAF_KC;
    const LeafConst L = leaf_const(hh, leaf, g.kb);
    const z* Sl = sinv + (size_t)leaf * b * aa;
    const z wdx = zscale(L.wbx, L.rdx), wdy = zscale(L.wby, L.rdy);
    for (int r0 = 0; r0 < nrhs; r0 += LEAF_KC) {
        const int kc = min(LEAF_KC, nrhs - r0);
        z* wp = w0;
        z* wc = w1;
        // forward: w_j = Sig_j^-1 (t_j - Lo_j w_{j-1}),  t = f - A_ib A_bb^-1 g
        for (int j = 0; j < b; ++j) {
            const int jj = j + 1;
            for (int e = tid; e < aa; e += nt) sig[e] = Sl[(size_t)j * aa + e];
            const z lam = jj > 1 ? block_lo(L, b, jj) : zmk(0.0, 0.0);
            __syncthreads();
            // right-hand side of block j into wc (t_j - Lo_j w_{j-1})
            for (int e = tid; e < a * kc; e += nt) {
                const int q = e % a, rc = e / a, rh = r0 + rc;
                const int i = q + 1;
                const z* gl = gb + ((size_t)leaf * nrhs + rh) * nb;
                z t = f ? f[((size_t)rh * nleaves + leaf) * ab + j * a + q] : zmk(0.0, 0.0);
                if (i == 1) zfms(t, wdx, gl[j]);
                if (i == a) zfms(t, wdx, gl[b + j]);
                if (jj == 1) zfms(t, wdy, gl[2 * b + q]);
                if (jj == b) zfms(t, wdy, gl[2 * b + a + q]);
                if (jj > 1) zfms(t, lam, wp[q + rc * a]);
                wc[e] = t;
            }
            __syncthreads();
            for (int e = tid; e < a * kc; e += nt) {
                const int i = e % a, rc = e / a;
                z acc = zmk(0.0, 0.0);
                for (int q = 0; q < a; ++q) zfma(acc, sig[i + q * a], wc[q + rc * a]);
                sol[((size_t)(r0 + rc) * nleaves + leaf) * n + nb + j * a + i] = acc;
                wp[e] = acc;    // w_j becomes the previous block for j+1
            }
            __syncthreads();
        }
        // backward: x_{b-1} = w_{b-1} (in wp); x_j = w_j - Sig_j^-1 Up_j x_{j+1}
        for (int j = b - 2; j >= 0; --j) {
            const int jj = j + 1;
            const z mu = block_up(L, b, jj);
            for (int e = tid; e < aa; e += nt) sig[e] = Sl[(size_t)j * aa + e];
            __syncthreads();
            for (int e = tid; e < a * kc; e += nt) {
                const int i = e % a, rc = e / a;
                z* up = sol + ((size_t)(r0 + rc) * nleaves + leaf) * n + nb + j * a;
                z acc = up[i];
                for (int q = 0; q < a; ++q) zfms(acc, sig[i + q * a], zmul(mu, wp[q + rc * a]));
                wc[e] = acc;
                up[i] = acc;
            }
            __syncthreads();
            z* t = wp; wp = wc; wc = t;
        }
        __syncthreads();
        // boundary values u_b = (g - c1 u(p1) - c2 u(p2)) / d
        for (int e = tid; e < nb * kc; e += nt) {
            const int r = e % nb, rc = e / nb, rh = r0 + rc;
            int ax, p1, p2;
            leaf_bpoint2(a, b, r, ax, p1, p2);
            const double h = ax == 0 ? L.hx : L.hy;
            z* u = sol + ((size_t)rh * nleaves + leaf) * n;
            z v = gb[((size_t)leaf * nrhs + rh) * nb + r];
            v = zsub(v, zadd(zscale(-3.0 / h, u[nb + p1]), zscale((1.0 / 3.0) / h, u[nb + p2])));
            u[r] = zmul(v, ax == 0 ? L.rdx : L.rdy);
        }
        __syncthreads();
    }
}

// The same solve for blocks of up to 32 x 32 on the FP64 tensor cores, with leaf_sweep's layout: a warp
// takes 8 right-hand sides of a leaf through all block steps with the running block vector in
// registers,
//   forward:  w_j = Sig_j^-1 (t_j - Lo_j w_{j-1}),  t = f - A_ib A_bb^-1 g
//   backward: x_{b-1} = w_{b-1};  x_j = w_j - Sig_j^-1 Up_j x_{j+1},
// each step W^T (8 x a) = T^T (8 x a) Sig_j^-T (four real products per complex one).  The warps of a
// CTA share a leaf's staged blocks.  The right-hand side (f forward, the stored w backward) is read
// two steps ahead.  A right-hand side's operations do not depend on the others of its warp.
// Measured: 4096 leaves of 16x16, 32 right-hand sides 0.69 ms (3 GB of loads and stores; half-warp
// DFMA columns 0.76), 1024 leaves, 16: 102 us (205); 1024 leaves of 24x24, 64: 1.14 ms (one CTA per
// leaf with scalar products 1.85); 64 leaves of 32x32, one: 205 us.  Two CTAs of 8 warps per SM: at
// three (80 registers) the spills cost more (0.85 ms).
template <int NT>
__global__ void __launch_bounds__(256, NT <= 3 ? 2 : 1) leaf_solve_kernel(LeafGeom g, int nleaves, int nrhs, int nchunk,
                                                         const double* __restrict__ hh, const z* __restrict__ f,
                                                         const z* __restrict__ gb, const z* __restrict__ sinv,
                                                         z* __restrict__ sol) {
    using Cfg = SweepCfg<NT>;
    constexpr int LD = Cfg::LD;
    extern __shared__ z sm[];
    const int nthr = blockDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lr = lane >> 2, lc = lane & 3;
    const int leaf = blockIdx.x / nchunk, chunk = blockIdx.x % nchunk;
    const int a = g.a, b = g.b, nb = g.nb, n = g.n, ab = a * b, aa = a * a;
    const LeafConst L = leaf_const(hh, leaf, g.kb);
    const int nsteps = 2 * b - 1;
    BlockRing<NT> ring{sm, sinv + (size_t)leaf * b * aa, a, aa, b, nsteps};
    pdl_launch();
    ring.start();
    const BlockCoupling cpl(L, b);
    pdl_wait();                            // the factor's blocks are complete; f, g and sol are the chain's
    const int rh0 = (chunk * (nthr >> 5) + warp) * 8, rh = rh0 + lr;
    const bool live = rh < nrhs;
    const int rs = live ? rh : 0;
    const z* fl = f ? f + ((size_t)rs * nleaves + leaf) * ab : nullptr;
    const z* gl = gb + ((size_t)leaf * nrhs + rs) * nb;
    z* ul = sol + ((size_t)rs * nleaves + leaf) * n;
    const z wdx = zscale(L.wbx, L.rdx), wdy = zscale(L.wby, L.rdy);
    // this lane's part of step st's right-hand side
    auto fetch = [&](int st, z (&v)[2 * NT]) {
        const bool fwd = st < b;
        const int j = fwd ? st : 2 * b - 2 - st;
#pragma unroll
        for (int e = 0; e < 2 * NT; ++e) {
            const int i = 8 * (e >> 1) + 2 * lc + (e & 1);
            v[e] = zmk(0.0, 0.0);
            if (live && i < a && st < nsteps) {
                if (!fwd) v[e] = ul[nb + j * a + i];
                else if (fl) v[e] = fl[j * a + i];
            }
        }
    };
    // and what the boundary data adds to it in a forward step
    auto gfetch = [&](int j, z (&v)[2 * NT]) {
#pragma unroll
        for (int e = 0; e < 2 * NT; ++e) {
            const int i = 8 * (e >> 1) + 2 * lc + (e & 1);
            if (!live || i >= a || j >= b) continue;
            if (i == 0) zfms(v[e], wdx, gl[j]);
            if (i == a - 1) zfms(v[e], wdx, gl[b + j]);
            if (j == 0) zfms(v[e], wdy, gl[2 * b + i]);
            if (j == b - 1) zfms(v[e], wdy, gl[2 * b + a + i]);
        }
    };
    z t0[2 * NT], t1[2 * NT];              // right-hand sides of the current and the next step
    fetch(0, t0);
    gfetch(0, t0);
    fetch(1, t1);
    gfetch(1, t1);
    double wre[2 * NT], wim[2 * NT];       // the running block vector
#pragma unroll
    for (int e = 0; e < 2 * NT; ++e) wre[e] = wim[e] = 0.0;
    for (int st = 0; st < nsteps; ++st) {
        const bool fwd = st < b;
        const int j = fwd ? st : 2 * b - 2 - st;
        const z* S = ring.next(st) + lr + 2 * lc * LD;
        // forward: R = t - Lo_j w; backward: R = -Up_j x_{j+1}, added to w_j
        const z co = fwd ? cpl.lo(j + 1) : cpl.up(j + 1);
        double rre[2 * NT], rim[2 * NT], cre[NT][2], cim[NT][2];
#pragma unroll
        for (int e = 0; e < 2 * NT; ++e) {
            z v = fwd ? t0[e] : zmk(0.0, 0.0);
            if (st > 0) zfms(v, co, zmk(wre[e], wim[e]));
            rre[e] = v.x;
            rim[e] = v.y;
            cre[e >> 1][e & 1] = fwd ? 0.0 : t0[e].x;
            cim[e >> 1][e & 1] = fwd ? 0.0 : t0[e].y;
            t0[e] = t1[e];
        }
        // two steps on: a forward block's f, or a w of this thread, stored at least two steps ago
        if (st + 2 < b) {
            fetch(st + 2, t1);
            gfetch(st + 2, t1);
        } else if (st + 2 > b) {
            fetch(st + 2, t1);
        }
#pragma unroll
        for (int e = 0; e < 2 * NT; ++e) {           // k-step: columns q = 8 (e/2) + 2 lc + e%2 of the block
            z bf[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) bf[t] = S[8 * t + (8 * (e >> 1) + (e & 1)) * LD];
#pragma unroll
            for (int t = 0; t < NT; ++t) dmma884(cre[t][0], cre[t][1], rre[e], bf[t].x);
#pragma unroll
            for (int t = 0; t < NT; ++t) dmma884(cim[t][0], cim[t][1], rre[e], bf[t].y);
#pragma unroll
            for (int t = 0; t < NT; ++t) dmma884(cre[t][0], cre[t][1], -rim[e], bf[t].y);
#pragma unroll
            for (int t = 0; t < NT; ++t) dmma884(cim[t][0], cim[t][1], rim[e], bf[t].x);
        }
#pragma unroll
        for (int e = 0; e < 2 * NT; ++e) {
            const int i = 8 * (e >> 1) + 2 * lc + (e & 1);
            wre[e] = cre[e >> 1][e & 1];
            wim[e] = cim[e >> 1][e & 1];
            if (live && i < a) ul[nb + j * a + i] = zmk(wre[e], wim[e]);
            if (st + 2 == b) t1[e] = zmk(wre[e], wim[e]);          // w_{b-2}, the first backward step's
        }
    }
    __syncwarp();
    // boundary values u_b = (g - c1 u(p1) - c2 u(p2)) / d of the warp's right-hand sides
    const int live_rhs = min(8, nrhs - rh0);
    for (int e = lane; e < nb * live_rhs; e += 32) {
        const int r = e % nb, rr = rh0 + e / nb;
        int ax, p1, p2;
        leaf_bpoint2(a, b, r, ax, p1, p2);
        const double h = ax == 0 ? L.hx : L.hy;
        z* u = sol + ((size_t)rr * nleaves + leaf) * n;
        z v = gb[((size_t)leaf * nrhs + rr) * nb + r];
        v = zsub(v, zadd(zscale(-3.0 / h, u[nb + p1]), zscale((1.0 / 3.0) / h, u[nb + p2])));
        u[r] = zmul(v, ax == 0 ? L.rdx : L.rdy);
    }
}

template <int NT>
static cudaError_t launch_solve(const LeafGeom& g, int nleaves, int nrhs, const double* h, const z* f, const z* gb,
                                const z* sinv, z* sol, cudaStream_t s, bool pdl) {
    const int units = (nrhs + 7) / 8, wpc = std::min(units, 8), nchunk = (units + wpc - 1) / wpc;
    static DeviceAttrCache attr;
    cudaError_t e = ensure_smem_attr(leaf_solve_kernel<NT>, SweepCfg<NT>::SMEM, attr);
    if (e != cudaSuccess) return e;
    note_launch();
    return launch_kernel(leaf_solve_kernel<NT>, dim3((unsigned)nleaves * nchunk), 32 * wpc, SweepCfg<NT>::SMEM, s, pdl, g,
                         nleaves, nrhs, nchunk, h, f, gb, sinv, sol);
}

cudaError_t leaf_block_solve(const LeafGeom& g, int nleaves, int nrhs, const double* h, const z* f, const z* gb,
                             const z* sinv, z* sol, cudaStream_t s, bool pdl) {
    if (g.a <= 8) return launch_solve<1>(g, nleaves, nrhs, h, f, gb, sinv, sol, s, pdl);
    if (g.a <= 16) return launch_solve<2>(g, nleaves, nrhs, h, f, gb, sinv, sol, s, pdl);
    if (g.a <= 24) return launch_solve<3>(g, nleaves, nrhs, h, f, gb, sinv, sol, s, pdl);
    if (g.a <= 32) return launch_solve<4>(g, nleaves, nrhs, h, f, gb, sinv, sol, s, pdl);
    const size_t sh = ((size_t)g.a * g.a + 2 * (size_t)g.a * LEAF_KC) * sizeof(z);
    if (sh > 48 * 1024) {
        static DeviceAttrCache attr;
        cudaError_t e = ensure_smem_attr(leaf_block_solve_kernel, sh, attr);
        if (e != cudaSuccess) return e;
    }
    leaf_block_solve_kernel<<<nleaves, 256, sh, s>>>(g, nleaves, nrhs, h, f, gb, sinv, sol);
    note_launch();
    return cudaGetLastError();
}

}  // namespace rb
