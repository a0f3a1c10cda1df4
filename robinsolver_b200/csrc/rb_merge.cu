// rb_merge.cu -- K-form merge of the levels whose interface has up to 32 points, for sm_100a.
//
// [Y1; Y2] = M^-1 blockdiag(T1_iN, T2_iN) and the parent map (compute_RTR,
// robin_tree_module.f90:375-650).  These levels' products are small and short, so as separate
// launches they are bound by the launches themselves and by the passes over what lies between them.
//   merge_interface (m <= 32): one CTA per node forms A1, A2, K = nu^2 I - A2 A1 and inverts K in
//     registers, in place of three copies, a GEMM and an inversion.
//   merge_columns (m <= 16): the rest is independent from column to column of [T1_iN, T2_iN].  A warp
//     takes 8 columns through  B1 = -A2 X,  Y1 = K^-1 B1,  Y2 = (X - A1 Y1) / nu  and the parent
//     map's columns  T_NN + [T1_Ni Y1; T2_Ni Y2]  with all vectors in registers: the products are
//     V^T (8 x rows) = X^T (8 x m) W^T on the FP64 tensor cores (m8n8k4, three real products per
//     complex one), the k order chosen so that one product's accumulators are the next one's A
//     fragments as they stand.  The matrices W come straight from memory; the warps of a CTA work
//     on the same node and share them in L1.
// Measured: the interface of 2048 nodes, m = 16, 37 us (was 128), of 1024, m = 32, 78 us (was 105 after
// the register inversion); at m = 64 the product K costs one CTA more than a GEMM launch (78 us for
// one to four nodes against 75).  The columns of 2048 nodes, m = 16, 347 us (four GEMM launches: 429).  Longer vectors leave a
// warp too few chains of MMAs to hide their latency: at m = 32 the columns took 910 us against the
// GEMMs' 356, at m = 64 1405 against 524, so above 16 they stay GEMMs.
#include "rb_gemm_dmma.cuh"
#include "rb_kernels.h"
#include "rb_pivot.cuh"

namespace rb {

__global__ void __launch_bounds__(128) merge_interface_kernel(MergeSmall g, int* status) {
    extern __shared__ z sm[];
    __shared__ PivotShared<1, 4> sh;
    const int m = g.m, mm = m * m, node = blockIdx.x;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, w = tid >> 5;
    z* s1 = sm;
    z* s2 = sm + mm;
    const z* t1 = g.child.rtr + (2LL * node) * g.child.stride + g.o1 + (long long)g.o1 * g.child.ld;
    const z* t2 = g.child.rtr + (2LL * node + 1) * g.child.stride + g.o2 + (long long)g.o2 * g.child.ld;
    z* a1 = g.a1 + (long long)node * mm;
    z* a2 = g.a2 + (long long)node * mm;
    for (int e = tid; e < mm; e += nt) {
        const int r = e % m, q = e / m;
        z v1 = zneg(t1[r + (long long)q * g.child.ld]), v2 = zneg(t2[r + (long long)q * g.child.ld]);
        if (r == q) {
            v1 = zadd(v1, g.zeta);
            v2 = zadd(v2, g.zeta);
        }
        s1[e] = v1;
        s2[e] = v2;
        a1[e] = v1;
        a2[e] = v2;
    }
    __syncthreads();
    const z nu2 = zmul(g.nu, g.nu);
    z v[1][PV_CG];
#pragma unroll
    for (int e = 0; e < PV_CG; ++e) v[0][e] = lane == w * PV_CG + e && lane < m ? nu2 : zmk(0.0, 0.0);
    for (int q = 0; q < m; ++q) {
        const z x = lane < m ? s2[lane + q * m] : zmk(0.0, 0.0);
#pragma unroll
        for (int e = 0; e < PV_CG; ++e) {
            const int c = w * PV_CG + e;
            zfms(v[0][e], x, c < m ? s1[q + c * m] : zmk(0.0, 0.0));
        }
    }
    int myk[1];
    const bool ok = cta_invert<1, 4>(v, m, sh, myk);
    z* kv = g.kinv + (long long)node * mm;
#pragma unroll
    for (int e = 0; e < PV_CG; ++e) {
        const int q = w * PV_CG + e;
        if (lane < m && q < m) kv[myk[0] + sh.pk[q] * m] = v[0][e];
    }
    if (!ok) atomicOr(status, RB_STATUS_ZERO_PIVOT);
}

// A warp's 8 columns of a vector with up to 8 NT rows: lane (column lane/4) holds rows
// 8t + 2 (lane%4) + h at [2t + h].
template <int NT>
struct ColVec {
    double re[2 * NT], im[2 * NT];
};

// one 8-row tile of W X: acc[h] = sum_q W(row, q) X(q), row = 8t + 2 (lane%4) + h of the output; wrow:
// this lane's fragment row W(8t + lane/4, .), ok its validity
template <int NT>
__device__ __forceinline__ void col_tile(const z* wrow, long long ld, bool ok, int m, const ColVec<NT>& x, int lc,
                                         z (&acc)[2]) {
    z f[2 * NT];
#pragma unroll
    for (int e = 0; e < 2 * NT; ++e) {
        const int q = 8 * (e >> 1) + 2 * lc + (e & 1);
        f[e] = ok && q < m ? wrow[(long long)q * ld] : zmk(0.0, 0.0);
    }
    double p1[2] = {0.0, 0.0}, p2[2] = {0.0, 0.0}, p3[2] = {0.0, 0.0};
#pragma unroll
    for (int e = 0; e < 2 * NT; ++e) {
        dmma884(p1[0], p1[1], x.re[e], f[e].x);
        dmma884(p2[0], p2[1], x.im[e], f[e].y);
        dmma884(p3[0], p3[1], x.re[e] + x.im[e], f[e].x + f[e].y);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) acc[h] = zmk(p1[h] - p2[h], p3[h] - p1[h] - p2[h]);
}

// y = alpha W x + beta x0, W m x m with leading dimension m; x0 this lane's column in memory, read
// again here rather than held (null: none)
template <int NT>
__device__ __forceinline__ void col_apply(const z* W, int m, const ColVec<NT>& x, z alpha, const z* x0, z beta, int lr,
                                          int lc, ColVec<NT>& y) {
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        z acc[2];
        const int i = 8 * t + lr;
        col_tile<NT>(W + (i < m ? i : 0), m, i < m, m, x, lc, acc);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            z v = zmul(alpha, acc[h]);
            const int q = 8 * t + 2 * lc + h;
            if (x0 && q < m) zfma(v, beta, x0[q]);
            y.re[2 * t + h] = v.x;
            y.im[2 * t + h] = v.y;
        }
    }
}

constexpr int MC_WARPS = 4;

template <int NT>
__global__ void __launch_bounds__(32 * MC_WARPS) merge_columns_kernel(MergeSmall g, int u1, int nunits, int nchunk) {
    const int node = blockIdx.x / nchunk;
    const int unit = (blockIdx.x % nchunk) * MC_WARPS + (threadIdx.x >> 5);
    if (unit >= nunits) return;
    const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
    const int m = g.m, mm = m * m;
    const int ch = unit < u1 ? 0 : 1;                // the child whose columns these are
    const int nc = ch ? g.n2 : g.n1, oc = ch ? g.o2 : g.o1;
    const int j = (ch ? unit - u1 : unit) * 8 + lr;  // this lane's column among the child's outer points
    const bool live = j < nc;
    const long long ld = g.child.ld;
    const z* r1 = g.child.rtr + (2LL * node) * g.child.stride;
    const z* r2 = r1 + g.child.stride;
    const z* tc = ch ? r2 : r1;
    const long long pc = live ? (long long)(j + (j >= oc ? m : 0)) * ld : 0;     // its physical column
    const int col = (ch ? g.n1 : 0) + j;             // its column of Y1, Y2
    const z rnu = zrcp(g.nu), mrnu = zneg(rnu);
    ColVec<NT> x, y;
#pragma unroll
    for (int e = 0; e < 2 * NT; ++e) {
        const int q = 8 * (e >> 1) + 2 * lc + (e & 1);
        const z v = live && q < m ? tc[oc + q + pc] : zmk(0.0, 0.0);
        x.re[e] = v.x;
        x.im[e] = v.y;
    }
    const z* kv = g.kinv + (long long)node * mm;
    if (ch == 0) {
        // Y1 = K^-1 (-A2 X); Y2 = (X - A1 Y1) / nu
        ColVec<NT> b;
        col_apply<NT>(g.a2 + (long long)node * mm, m, x, zmk(-1.0, 0.0), nullptr, rnu, lr, lc, b);
        col_apply<NT>(kv, m, b, zmk(1.0, 0.0), nullptr, rnu, lr, lc, y);
        ColVec<NT> t;
        col_apply<NT>(g.a1 + (long long)node * mm, m, y, mrnu, live ? tc + oc + pc : nullptr, rnu, lr, lc, t);
        x = t;
    } else {
        // Y1 = nu K^-1 X; Y2 = -A1 Y1 / nu
        col_apply<NT>(kv, m, x, g.nu, nullptr, rnu, lr, lc, y);
        col_apply<NT>(g.a1 + (long long)node * mm, m, y, mrnu, nullptr, rnu, lr, lc, x);
    }
    // y = Y1, x = Y2
    const long long yo = (long long)node * m * (g.n1 + g.n2) + (long long)col * m;
#pragma unroll
    for (int e = 0; e < 2 * NT; ++e) {
        const int q = 8 * (e >> 1) + 2 * lc + (e & 1);
        if (live && q < m) {
            g.y1[yo + q] = zmk(y.re[e], y.im[e]);
            g.y2[yo + q] = zmk(x.re[e], x.im[e]);
        }
    }
    if (!g.par) return;
    z* par = g.par + (long long)node * g.nbp * g.nbp + (live ? (long long)(ch ? g.pmap2 : g.pmap1)[j] * g.nbp : 0);
    for (int a = 0; a < 2; ++a) {
        // rows of child a + 1: T_Ni times its interface values, plus T_NN where the column is the child's own
        const z* ra = a ? r2 : r1;
        const int na = a ? g.n2 : g.n1, oa = a ? g.o2 : g.o1;
        const int* pm = a ? g.pmap2 : g.pmap1;
        const z* tni = ra + (long long)oa * ld;
        const ColVec<NT> s = a ? x : y;
#pragma unroll 4
        for (int i0 = 0; i0 < na; i0 += 8) {
            const int i = i0 + lr;
            z acc[2];
            col_tile<NT>(tni + (i < na ? i + (i >= oa ? m : 0) : 0), ld, i < na, m, s, lc, acc);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = i0 + 2 * lc + h;
                if (!live || r >= na) continue;
                z v = acc[h];
                if (a == ch) v = zadd(v, ra[r + (r >= oa ? m : 0) + pc]);
                par[pm[r]] = v;
            }
        }
    }
}

cudaError_t merge_small_interface(const MergeSmall& g, int* status, cudaStream_t s) {
    const size_t sh = 2 * (size_t)g.m * g.m * sizeof(z);
    const int threads = (g.m + 7) / 8 * 32;
    if (g.m > MERGE_SMALL_MAX) return cudaErrorInvalidValue;
    merge_interface_kernel<<<g.nnodes, threads, sh, s>>>(g, status);
    note_launch();
    return cudaGetLastError();
}

cudaError_t merge_small_columns(const MergeSmall& g, cudaStream_t s) {
    if (g.m > MERGE_COLUMNS_MAX) return cudaErrorInvalidValue;
    const int u1 = (g.n1 + 7) / 8, nunits = u1 + (g.n2 + 7) / 8, nchunk = (nunits + MC_WARPS - 1) / MC_WARPS;
    merge_columns_kernel<2><<<(unsigned)g.nnodes * nchunk, 32 * MC_WARPS, 0, s>>>(g, u1, nunits, nchunk);
    note_launch();
    return cudaGetLastError();
}

}  // namespace rb
