// rb_gj.cu -- batched in-place Gauss-Jordan inversion of complex128 matrices for sm_100a.
//
// The reference forms inv(D) explicitly (zgetri after zgetrf, robin_tree_module.f90:449-455)
// and applies D and S through their LU factors.  Here every dense inverse the factor/solve
// needs (the leaf's interior Schur complement, D and S of each merge) is formed explicitly by
// Gauss-Jordan elimination with partial pivoting, so that later applications are GEMMs.
// Pivots are ranked as LAPACK's izamax does, by |re|+|im| in all its bits.  Exactly equal ones go to the row
// that stands first: in the matrix as given where rows stay in place, after the exchanges so far in the
// blocked path.
//
// m <= 64: the whole matrix in the registers of a warp (m <= 16) or a CTA (rb_pivot.cuh).
// m  > 64: blocked Gauss-Jordan by panels of nb = 8 columns.  Per panel:
//   1. elimination of the panel: the pivot search below the diagonal, row exchange, scaling and
//      elimination of every other row, leaving the accumulated transform W in the panel columns;
//   2. update of every other column: the panel's row exchanges, then
//      A[i, rest] += W[i,:] Z for rows outside the panel and A[P, rest] = W_P Z for the panel
//      rows, Z = A[P, rest] after the exchanges.  (Writing the panel rows as Z + (W_P - I) Z
//      instead cancels catastrophically: W_P's diagonal holds the reciprocal pivots, ~h^2 for
//      the FD matrices here.)
//   The resident kernel (gj_resident) runs the whole batch in one cooperative launch with the
//   columns held in shared memory (in several, when they do not fit at once); gj_panel + gj_apply, two
//   launches per panel, are the same arithmetic in the same order, used when a device cannot hold one
//   matrix and to compare.
// After the last panel the column exchanges are undone in reverse order (by the resident kernel as it
// writes, by gj_unscramble after the blocked path).
#include <algorithm>
#include <cstdlib>
#include "rb_gemm_tile.cuh"
#include "rb_kernels.h"
#include "rb_pivot.cuh"

namespace rb {

// the resident path's two words per panel of 8 columns and its counter, in complex elements per matrix
long long gj_workspace_elems(int m) { return m <= GJ_SMALL_MAX ? 0 : (m + 7) / 8 + 1; }

// warp argmax: larger value wins, equal values go to the smaller index
__device__ __forceinline__ void argmax_warp(double& v, int& i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ov = __shfl_down_sync(0xffffffffu, v, o);
        const int oi = __shfl_down_sync(0xffffffffu, i, o);
        if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
    }
}

// a b and 1/a with the roundings spelled out: the two paths above m = 64 agree bit for bit whichever
// product of a sum the compiler would have fused
__device__ __forceinline__ z gj_mul(z a, z b) {
    return zmk(__fma_rn(-a.y, b.y, __dmul_rn(a.x, b.x)), __fma_rn(a.y, b.x, __dmul_rn(a.x, b.y)));
}
__device__ __forceinline__ z gj_rcp(z a) {
    const double r = 1.0 / __fma_rn(a.y, a.y, __dmul_rn(a.x, a.x));
    return zmk(__dmul_rn(a.x, r), __dmul_rn(-a.y, r));
}

__device__ __forceinline__ bool zis0(z a) { return a.x == 0.0 && a.y == 0.0; }

// ---------------------------------------------------------------------------------------------------
// m <= 64: the whole matrix in registers (rb_pivot.cuh).  The result goes back in place with its
// rows and columns in order; a column's permuted rows cover whole memory sectors between them.
__global__ void __launch_bounds__(128) gj_warp_kernel(const GJDesc* __restrict__ descs, int count, int m, int* status) {
    __shared__ z prow[4][32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int mat = blockIdx.x * (blockDim.x >> 5) + wib;
    if (mat >= count) return;
    const GJDesc g = descs[mat];
    const int r = lane & 15, hf = lane >> 4;
    z v[PV_CG];
#pragma unroll
    for (int e = 0; e < PV_CG; ++e) {
        const int q = hf * PV_CG + e;
        v[e] = r < m && q < m ? g.A[r + (long long)q * g.ld] : zmk(0.0, 0.0);
    }
    int myk, pk;
    const bool ok = warp_invert16(v, m, prow[wib], myk, pk);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < PV_CG; ++e) {
        const int q = hf * PV_CG + e;
        const int pq = __shfl_sync(0xffffffffu, pk, q);
        if (r < m && q < m) g.A[myk + (long long)pq * g.ld] = v[e];
    }
    if (!ok) atomicOr(status, RB_STATUS_ZERO_PIVOT);
}

template <int RPL, int NG>
__global__ void __launch_bounds__(32 * NG) gj_cta_kernel(const GJDesc* __restrict__ descs, int m, int* status) {
    __shared__ PivotShared<RPL, NG> sh;
    const GJDesc g = descs[blockIdx.x];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    z v[RPL][PV_CG];
#pragma unroll
    for (int i = 0; i < RPL; ++i)
#pragma unroll
        for (int e = 0; e < PV_CG; ++e) {
            const int r = lane + 32 * i, q = w * PV_CG + e;
            v[i][e] = r < m && q < m ? g.A[r + (long long)q * g.ld] : zmk(0.0, 0.0);
        }
    int myk[RPL];
    const bool ok = cta_invert<RPL, NG>(v, m, sh, myk);
    __syncthreads();                              // sh.pk is complete
#pragma unroll
    for (int i = 0; i < RPL; ++i)
#pragma unroll
        for (int e = 0; e < PV_CG; ++e) {
            const int r = lane + 32 * i, q = w * PV_CG + (RPL > 1 ? (e + m) % PV_CG : e);
            if (r < m && q < m) g.A[myk[i] + (long long)sh.pk[q] * g.ld] = v[i][e];
        }
    if (!ok) atomicOr(status, RB_STATUS_ZERO_PIVOT);
}

// ---------------------------------------------------------------------------------------------------
// MAXT: largest matrix (= threads per CTA) a panel instance serves; it bounds the registers
// available to row[NB]
template <int NB, int MAXT>
__global__ void __launch_bounds__(MAXT) gj_panel_kernel(const GJDesc* __restrict__ descs, int m,
                                                        int k0, int nbk, int* status) {
    // two block barriers per column: (1) per-warp pivot candidates, (2) the scaled pivot row and
    // the displaced row.  Every warp reduces the 32 candidates itself, so the pivot index needs no
    // extra barrier; the holder of the pivot row publishes it already scaled, the holder of row c
    // publishes its row, and after barrier (2) row c takes the pivot row while the pivot's old
    // row takes row c's values and is eliminated like any other row.
    __shared__ z xb[2][NB], prow[2][NB];
    __shared__ double wv[2][32];
    __shared__ int wi[2][32];
    const GJDesc g = descs[blockIdx.x];
    const int r = threadIdx.x;
    const bool own = r < m;
    const int lane = r & 31, warp = r >> 5, nwarps = (blockDim.x + 31) >> 5;
    z row[NB];
#pragma unroll
    for (int kk = 0; kk < NB; ++kk)
        row[kk] = (own && kk < nbk) ? g.A[r + (long long)(k0 + kk) * g.ld] : zmk(0.0, 0.0);
    bool bad = false;
#pragma unroll
    for (int kk = 0; kk < NB; ++kk) {
        if (kk >= nbk) break;
        const int c = k0 + kk;
        const int sb = kk & 1;           // alternate buffers so that barrier (1) of the next column
                                         // also orders this column's reads of prow/xb
        double v = (own && r >= c) ? zabs1(row[kk]) : -1.0;
        int idx = own ? r : 0x7fffffff;
        argmax_warp(v, idx);
        if (lane == 0) { wv[sb][warp] = v; wi[sb][warp] = idx; }
        __syncthreads();                                   // (1)
        v = lane < nwarps ? wv[sb][lane] : -1.0;
        idx = lane < nwarps ? wi[sb][lane] : 0x7fffffff;
        argmax_warp(v, idx);
        const int p = __shfl_sync(0xffffffffu, idx, 0);
        if (r == p) {
            if (zis0(row[kk])) bad = true;
            const z pinv = gj_rcp(row[kk]);
#pragma unroll
            for (int j = 0; j < NB; ++j) prow[sb][j] = (j == kk) ? pinv : gj_mul(row[j], pinv);
            g.ipiv[c] = p;
        }
        if (r == c && p != c) {
#pragma unroll
            for (int j = 0; j < NB; ++j) xb[sb][j] = row[j];
        }
        __syncthreads();                                   // (2)
        if (r == c) {
#pragma unroll
            for (int j = 0; j < NB; ++j) row[j] = prow[sb][j];
        } else if (own) {
            if (r == p) {
#pragma unroll
                for (int j = 0; j < NB; ++j) row[j] = xb[sb][j];
            }
            const z f = row[kk];
#pragma unroll
            for (int j = 0; j < NB; ++j)
                if (j != kk) zfms(row[j], f, prow[sb][j]);
            row[kk] = zneg(gj_mul(f, prow[sb][kk]));
        }
    }
    if (own) {
#pragma unroll
        for (int kk = 0; kk < NB; ++kk) {
            if (kk >= nbk) break;
            g.A[r + (long long)(k0 + kk) * g.ld] = row[kk];
        }
    }
    if (bad) atomicOr(status, 1);
}

// Applies one panel to the other columns: CW whole columns per CTA are staged in shared memory,
// the panel's row exchanges are applied there, and the CTA writes
//     A[i, j] + W[i,:] Z[:, j]   for rows i outside the panel,   W[i,:] Z[:, j]   for panel rows,
// with Z = the (exchanged) panel rows of its own columns and W = the panel columns of A.  A CTA
// owns whole columns, so no other CTA reads what it overwrites.
template <int CW, int NBMAX>
__global__ void __launch_bounds__(256) gj_apply_kernel(const GJDesc* __restrict__ descs, int m, int k0, int nbk) {
    extern __shared__ z cols[];                 // m x CW, column-major (ld m)
    const GJDesc g = descs[blockIdx.y];
    const int rest = m - nbk;
    const int j0 = blockIdx.x * CW;
    const int ncol = min(CW, rest - j0);
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int e = tid; e < m * ncol; e += nt) {
        const int r = e % m, q = e / m;
        const int jl = j0 + q;
        const int col = jl < k0 ? jl : jl + nbk;
        cols[r + q * m] = g.A[r + (long long)col * g.ld];
    }
    __syncthreads();
    // the panel's exchanges, in order (each thread owns columns)
    if (tid < ncol)
        for (int kk = 0; kk < nbk; ++kk) {
            const int c = k0 + kk, p = g.ipiv[c];
            if (p != c) {
                const z t = cols[c + tid * m];
                cols[c + tid * m] = cols[p + tid * m];
                cols[p + tid * m] = t;
            }
        }
    __syncthreads();
    for (int r = tid; r < m; r += nt) {
        z w[NBMAX];
#pragma unroll
        for (int kk = 0; kk < NBMAX; ++kk)
            w[kk] = kk < nbk ? g.A[r + (long long)(k0 + kk) * g.ld] : zmk(0.0, 0.0);
        const bool in_panel = r >= k0 && r < k0 + nbk;
        for (int q = 0; q < ncol; ++q) {
            z v = in_panel ? zmk(0.0, 0.0) : cols[r + q * m];
#pragma unroll
            for (int kk = 0; kk < NBMAX; ++kk)
                if (kk < nbk) zfma(v, w[kk], cols[k0 + kk + q * m]);
            const int jl = j0 + q;
            const int col = jl < k0 ? jl : jl + nbk;
            g.A[r + (long long)col * g.ld] = v;
        }
    }
}

// ---------------------------------------------------------------------------------------------------
// Resident Gauss-Jordan: the whole batch in one launch.  Matrix i is split over P CTAs by whole
// panels of NB columns; CTA j keeps its ppc panels (m x cw complex, cw <= ppc*NB) in shared
// memory for the whole inversion.  No row is exchanged: a pivot's row stays where it is and is passed
// over by later searches, and the permutation goes into the final write.  The owner of panel p
// eliminates it (one or two rows per thread in registers), writes the accumulated transform W_p to the
// matrix's own global storage at panel p's columns (unused while the columns live in shared memory), and
// publishes the panel's pivot rows in its two words.  Every CTA then applies step p (A += W_p Z outside
// the pivots' rows and W_p Z on them, Z the pivots' rows) to its resident columns.  The owner of panel
// p+1 applies step p to that panel first, eliminates and publishes it, and only then updates its other
// columns, so the dependent chain per step is one hand-off, one panel update and one panel elimination.
// After the last step a per-matrix counter holds every CTA until all have stopped reading W slots; then
// the columns go back.  The arithmetic is the blocked path's, in its order (rows of equal magnitude are
// ranked by where they stand, so exactly tied pivots may fall differently).
//
// The launch is cooperative (all CTAs co-resident), and every wait is bounded in time: a CTA
// that waits longer than GJ_WAIT_NS sets RB_STATUS_GJ_TIMEOUT in the status word and returns.
constexpr unsigned long long GJ_WAIT_NS = 1000000000ull;

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long ld_acquire_gpu(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(unsigned long long* p, unsigned long long v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Shared state of a CTA.  Everything is double-buffered by the parity of its column or step: it is
// written again two later, after a block barrier that follows its last read.
template <int NB>
struct ResShared {
    z prow[2][NB];                       // a column's scaled pivot row
    uint4 cand[2][32];                   // per warp: its candidate's key (high, low word) and row
    int spv[2][NB];                      // a step's pivot rows
    int ok[2], done_ok;
};

// A panel's two words: four pivot rows each, 12 bits a row, under the top bit
static_assert(8 == 2 * 4, "pivots of a panel in two words");
constexpr unsigned long long GJ_READY = 1ull << 63;

// The words of step p, awaited by two lanes (bounded); the pivots go to shared memory, the outcome to
// every thread of the CTA.
template <int NB>
__device__ __forceinline__ bool res_wait_step(const unsigned long long* words, int p, int* status, ResShared<NB>& sh) {
    if (threadIdx.x < 2) {
        unsigned long long w = ld_acquire_gpu(words + 2 * p + threadIdx.x);
        if (!(w & GJ_READY)) {
            const unsigned long long t0 = global_ns();
            int spins = 0;
            while (!((w = ld_acquire_gpu(words + 2 * p + threadIdx.x)) & GJ_READY)) {
                if (++spins > 32) __nanosleep(40);
                if (global_ns() - t0 > GJ_WAIT_NS) {
                    sh.ok[p & 1] = 0;
                    atomicOr(status, RB_STATUS_GJ_TIMEOUT);
                    break;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) sh.spv[p & 1][4 * threadIdx.x + i] = (int)((w >> (12 * i)) & 0xFFF);
    }
    __syncthreads();
    return sh.ok[p & 1] != 0;
}

// The largest key (hi, lo) -- the bit pattern of a non-negative double, which orders like the value -- of a
// warp, ties to the smaller row: true on the lane that holds it.  One reduction and a vote unless two
// high words tie.
__device__ __forceinline__ bool warp_key_best(unsigned hi, unsigned lo, int id, unsigned& best) {
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    best = __ballot_sync(0xffffffffu, hi == mh);
    if (best & (best - 1)) {
        const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
        const bool tie = hi == mh && lo == ml;
        const int mi = __reduce_min_sync(0xffffffffu, tie ? id : 0x7fffffff);
        best = __ballot_sync(0xffffffffu, tie && id == mi);
    }
    return (best >> (threadIdx.x & 31)) & 1u;
}

// this thread's candidate for column kk (its largest entry in rows no pivot has taken) reduced over the
// warp into the column's slots
template <int NB, int RPT>
__device__ __forceinline__ void res_candidate(const z (&row)[RPT][NB], int kk, int m, unsigned used, ResShared<NB>& sh) {
    const int tid = threadIdx.x, nt = blockDim.x;
    double v = 0.0;
    int vr = -1;
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = tid + i * nt;
        const double a = zabs1(row[i][kk]);
        if (r < m && !((used >> i) & 1u) && (vr < 0 || a > v)) { v = a; vr = r; }
    }
    const unsigned hi = vr >= 0 ? (unsigned)__double2hiint(v) : 0u, lo = vr >= 0 ? (unsigned)__double2loint(v) : 0u;
    const int id = vr >= 0 ? vr : 0x7fffffff;
    unsigned best;
    if (warp_key_best(hi, lo, id, best)) sh.cand[kk & 1][tid >> 5] = make_uint4(hi, lo, (unsigned)id, 0u);
}

// Eliminates a panel of nbk columns whose current values are in row[][]: RPT rows per thread (rows
// tid + i*blockDim.x), two block barriers per column (pivot candidates; scaled pivot row).  Rows stay where
// they are: a pivot's row is marked in `used` (bit i: row i of this thread).  On return row[][] holds the
// panel's transform W and pv its pivot rows.  The chain of a column is its latency: of a column's update
// only the next column is brought up to date before that one's pivot search; the rest runs beside the
// pivot's reciprocal.
template <int NB, int RPT>
__device__ __forceinline__ void res_eliminate_regs(z (&row)[RPT][NB], int m, int nbk, unsigned& used, int (&pv)[NB], int* status,
                                                   ResShared<NB>& sh) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, nwarps = (nt + 31) >> 5;
    bool bad = false;
    z f[RPT];                                     // the multipliers of the column before
    unsigned upd = 0;                             // rows it updates: all but its own
    res_candidate<NB, RPT>(row, 0, m, used, sh);
#pragma unroll
    for (int kk = 0; kk < NB; ++kk) pv[kk] = 0xFFF;
#pragma unroll
    for (int kk = 0; kk < NB; ++kk) {
        if (kk >= nbk) break;
        const int b = kk & 1;
        __syncthreads();
        const uint4 q = lane < nwarps ? sh.cand[b][lane] : make_uint4(0u, 0u, 0x7fffffffu, 0u);
        unsigned best;
        warp_key_best(q.x, q.y, (int)q.z, best);
        const int p = __shfl_sync(0xffffffffu, (int)q.z, __ffs(best) - 1);
        pv[kk] = p;
        z pinv[RPT];
#pragma unroll
        for (int i = 0; i < RPT; ++i)
            if (tid + i * nt == p) {
                if (zis0(row[i][kk])) bad = true;
                pinv[i] = gj_rcp(row[i][kk]);
            }
        if (kk > 0) {
#pragma unroll
            for (int i = 0; i < RPT; ++i)
                if ((upd >> i) & 1u) {
#pragma unroll
                    for (int j = 0; j < NB; ++j)
                        if (j != kk - 1 && j != kk) zfms(row[i][j], f[i], sh.prow[b ^ 1][j]);
                    row[i][kk - 1] = zneg(gj_mul(f[i], sh.prow[b ^ 1][kk - 1]));
                }
        }
        upd = (1u << RPT) - 1u;
#pragma unroll
        for (int i = 0; i < RPT; ++i)
            if (tid + i * nt == p) {
#pragma unroll
                for (int j = 0; j < NB; ++j) {
                    row[i][j] = (j == kk) ? pinv[i] : gj_mul(row[i][j], pinv[i]);
                    sh.prow[b][j] = row[i][j];
                }
                used |= 1u << i;
                upd &= ~(1u << i);
            }
        __syncthreads();
        const bool more = kk + 1 < NB && kk + 1 < nbk;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            f[i] = row[i][kk];
            if (((upd >> i) & 1u) && more) zfms(row[i][(kk + 1) % NB], f[i], sh.prow[b][(kk + 1) % NB]);
        }
        if (more) {
            res_candidate<NB, RPT>(row, (kk + 1) % NB, m, used, sh);
        } else {
#pragma unroll
            for (int i = 0; i < RPT; ++i)
                if ((upd >> i) & 1u) {
#pragma unroll
                    for (int j = 0; j < NB; ++j)
                        if (j != kk) zfms(row[i][j], f[i], sh.prow[b][j]);
                    row[i][kk] = zneg(gj_mul(f[i], sh.prow[b][kk]));
                }
        }
    }
    if (bad) atomicOr(status, RB_STATUS_ZERO_PIVOT);
}

// Stores an eliminated panel, W to the local columns at c and to Wg (ld wld), then publishes it with its
// pivots: the releases order the stores of the whole CTA, ahead of them by the block barrier.
template <int NB, int RPT>
__device__ __forceinline__ void res_publish(const z (&row)[RPT][NB], const int (&pv)[NB], z* c, int m, int nbk, z* Wg, long long wld,
                                            unsigned long long* words, int p, ResShared<NB>& sh) {
    const int tid = threadIdx.x, nt = blockDim.x;
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = tid + i * nt;
        if (r >= m) continue;
#pragma unroll
        for (int kk = 0; kk < NB; ++kk) {
            if (kk >= nbk) break;
            Wg[r + (long long)kk * wld] = row[i][kk];
            c[r + kk * m] = row[i][kk];
        }
    }
    if (tid == 0) {
#pragma unroll
        for (int kk = 0; kk < NB; ++kk) sh.spv[p & 1][kk] = pv[kk];
    }
    __syncthreads();
    if (tid < 2) {
        unsigned long long w = GJ_READY;
#pragma unroll
        for (int i = 0; i < 4; ++i) w |= (unsigned long long)(tid == 0 ? pv[i] : pv[4 + i]) << (12 * i);
        st_release_gpu(words + 2 * p + tid, w);
    }
}

// The values that a step (nbk pivots, W at W with ld wld, read through L2 when w_global) gives the rows
// of this thread in the nq <= NB columns at c: A + W Z outside the pivots' rows, W_P Z on them (bit i of
// `mine`), Z = the pivots' rows.  The columns in shared memory are read only; w holds W already when `held`.
template <int NB, int RPT>
__device__ __forceinline__ void res_updated(z (&row)[RPT][NB], const z (&w)[RPT][NB], bool held, unsigned mine, const z* c, int nq,
                                            int m, int nbk, const z* W, long long wld, bool w_global, const int* spv) {
    const int tid = threadIdx.x, nt = blockDim.x;
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = tid + i * nt;
        const bool keep = r < m && !((mine >> i) & 1u);
#pragma unroll
        for (int q = 0; q < NB; ++q) row[i][q] = keep && q < nq ? c[r + q * m] : zmk(0.0, 0.0);
    }
#pragma unroll
    for (int kk = 0; kk < NB; ++kk) {
        if (kk >= nbk) break;
        z wk[RPT];
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int r = tid + i * nt;
            if (held) wk[i] = w[i][kk];
            else wk[i] = r < m ? (w_global ? __ldcg(W + r + kk * wld) : W[r + kk * wld]) : zmk(0.0, 0.0);
        }
        const z* zk = c + spv[kk];
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            const z zv = q < nq ? zk[q * m] : zmk(0.0, 0.0);
#pragma unroll
            for (int i = 0; i < RPT; ++i) zfma(row[i][q], wk[i], zv);
        }
    }
}

// A step takes the CTA that owns the next panel through wait, W, update and elimination of that panel and
// the hand-over; that chain, latencies and one SM's FP64 rate, is the time.  A column waits for two
// barriers, two warp reductions and a reciprocal; the update goes from shared memory through registers
// into the elimination.
// Against exchanging rows in registers and shared memory and a gather, an update and an elimination in
// separate passes, with the columns' exchanges undone by a kernel of their own: one matrix of 128 135 to 112
// us, 256 297 to 248, 512 786 to 656, 1024 2490 to 2113.
template <int NB, int MAXT, int RPT>
__global__ void __launch_bounds__(MAXT, MAXT <= 256 ? 512 / MAXT : 1) gj_resident_kernel(
    const GJDesc* __restrict__ descs, int m, int npanels, int ppc, int P, int* status) {
    extern __shared__ z sm[];
    __shared__ ResShared<NB> sh;
    const int mat = blockIdx.x / P, j = blockIdx.x % P;
    const GJDesc g = descs[mat];
    const int pa = j * ppc, pb = min(npanels, pa + ppc);
    const int c0 = pa * NB, cw = min(m, pb * NB) - c0;
    z* cols = sm;                                   // m x cw, column-major (ld m)
    int* perm = reinterpret_cast<int*>(sm + (size_t)m * ppc * NB);    // the pivot row of every column
    unsigned long long* words = reinterpret_cast<unsigned long long*>(g.Zb);      // two per panel
    int* done = reinterpret_cast<int*>(words + 2 * npanels);          // CTAs past their last step
    const int tid = threadIdx.x, nt = blockDim.x;
    if (tid == 0) sh.ok[0] = sh.ok[1] = sh.done_ok = 1;
    for (int e = tid; e < m * cw; e += nt) {
        const int r = e % m, q = e / m;
        cols[r + q * m] = __ldcg(g.A + r + (long long)(c0 + q) * g.ld);
    }
    __syncthreads();
    z row[RPT][NB];
    int pv[NB];
    unsigned used = 0;                              // rows of this thread that a pivot has taken
    if (pa == 0) {
        const int nb0 = min(NB, m);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int r = tid + i * nt;
#pragma unroll
            for (int q = 0; q < NB; ++q) row[i][q] = r < m && q < nb0 ? cols[r + q * m] : zmk(0.0, 0.0);
        }
        res_eliminate_regs<NB, RPT>(row, m, nb0, used, pv, status, sh);
        res_publish<NB, RPT>(row, pv, cols, m, nb0, g.A, g.ld, words, 0, sh);
    }
    for (int p = 0; p < npanels; ++p) {
        const int k0 = p * NB, nbk = min(NB, m - k0);
        const bool own = p >= pa && p < pb;
        // the step's pivots are here, and every column that the step before wrote
        if (own) __syncthreads();
        else if (!res_wait_step<NB>(words, p, status, sh)) return;
        const int* spv = sh.spv[p & 1];
        const z* W = own ? cols + (size_t)(k0 - c0) * m : g.A + (long long)k0 * g.ld;
        const long long wld = own ? m : g.ld;
        constexpr bool HELD = RPT == 1;             // with one row a thread there are registers for W
        z w[RPT][NB];
        if (HELD) {
#pragma unroll
            for (int i = 0; i < RPT; ++i)
#pragma unroll
                for (int kk = 0; kk < NB; ++kk) {
                    const int r = tid + i * nt;
                    w[i][kk] = r < m && kk < nbk ? (own ? W[r + kk * wld] : __ldcg(W + r + kk * wld)) : zmk(0.0, 0.0);
                }
        }
        unsigned mine = 0;                          // this step's pivots among this thread's rows
#pragma unroll
        for (int i = 0; i < RPT; ++i)
#pragma unroll
            for (int kk = 0; kk < NB; ++kk)
                if (kk < nbk && spv[kk] == tid + i * nt) mine |= 1u << i;
        used |= mine;
        if (tid < nbk) perm[k0 + tid] = spv[tid];
        const int nx = p + 1;
        const bool next = nx < npanels && nx >= pa && nx < pb;
        if (next) {
            const int qn = nx * NB - c0, nbn = min(NB, m - nx * NB);
            res_updated<NB, RPT>(row, w, HELD, mine, cols + (size_t)qn * m, nbn, m, nbk, W, wld, !own, spv);
            // its barriers end every read of the panel's columns before they are stored
            res_eliminate_regs<NB, RPT>(row, m, nbn, used, pv, status, sh);
            res_publish<NB, RPT>(row, pv, cols + (size_t)qn * m, m, nbn, g.A + (long long)nx * NB * g.ld, g.ld, words, nx, sh);
        }
        for (int lp = pa; lp < pb; ++lp) {
            if (lp == p || (next && lp == nx)) continue;
            const int nq = min(NB, m - lp * NB);
            z* c = cols + (size_t)(lp - pa) * NB * m;
            res_updated<NB, RPT>(row, w, HELD, mine, c, nq, m, nbk, W, wld, !own, spv);
            __syncthreads();
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int r = tid + i * nt;
#pragma unroll
                for (int q = 0; q < NB; ++q)
                    if (r < m && q < nq) c[r + q * m] = row[i][q];
            }
        }
    }
    // no CTA of this matrix reads a W slot any more once all have arrived here
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        atomicAdd(done, 1);
        const unsigned long long t0 = global_ns();
        while (ld_acquire_gpu(done) < P) {
            __nanosleep(40);
            if (global_ns() - t0 > GJ_WAIT_NS) {
                sh.done_ok = 0;
                atomicOr(status, RB_STATUS_GJ_TIMEOUT);
                break;
            }
        }
    }
    __syncthreads();
    if (!sh.done_ok) return;
    // column q was eliminated by row perm[q]: the inverse has its rows in the columns' order and its
    // columns in the pivots'
    for (int e = tid; e < m * cw; e += nt) {
        const int r = e % m, q = e / m;
        g.A[r + (long long)perm[c0 + q] * g.ld] = cols[perm[r] + q * m];
    }
}

__global__ void gj_unscramble_kernel(const GJDesc* __restrict__ descs, int m) {
    const GJDesc g = descs[blockIdx.y];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= m) return;
    for (int k = m - 1; k >= 0; --k) {
        const int p = g.ipiv[k];
        if (p != k) {
            const z t = g.A[r + (long long)k * g.ld];
            g.A[r + (long long)k * g.ld] = g.A[r + (long long)p * g.ld];
            g.A[r + (long long)p * g.ld] = t;
        }
    }
}

template <int NB, int MAXT>
static cudaError_t gj_blocked(const GJDesc* d, int count, int m, int* st, cudaStream_t s) {
    const int threads = ((m + 31) / 32) * 32;
    if (threads > MAXT) return cudaErrorInvalidValue;
    constexpr int CW = 8;
    const size_t sh = (size_t)m * CW * sizeof(z);
    static DeviceAttrCache attr;
    {
        cudaError_t e = ensure_smem_attr(gj_apply_kernel<CW, NB>, 1024 * CW * sizeof(z), attr);
        if (e != cudaSuccess) return e;
    }
    for (int k0 = 0; k0 < m; k0 += NB) {
        const int nbk = (m - k0) < NB ? (m - k0) : NB;
        gj_panel_kernel<NB, MAXT><<<count, threads, 0, s>>>(d, m, k0, nbk, st);
        note_launch();
        const int rest = m - nbk;
        if (rest > 0) {
            gj_apply_kernel<CW, NB><<<dim3((rest + CW - 1) / CW, count), 256, sh, s>>>(d, m, k0, nbk);
            note_launch();
        }
    }
    gj_unscramble_kernel<<<dim3((m + 127) / 128, count), 128, 0, s>>>(d, m);
    note_launch();
    return cudaGetLastError();
}

// slots[i]: matrices that are co-resident with i + 1 panels per CTA.  The fewest launches that take `count`
// matrices, in equal parts of *chunk, and the fewest panels per CTA that hold one; 0 where not one does.
int gj_resident_split(int count, const int* slots, int n, int* chunk) {
    int most = 0;
    for (int i = 0; i < n; ++i) most = std::max(most, slots[i]);
    if (most == 0) return 0;
    const int parts = (count + most - 1) / most;
    *chunk = (count + parts - 1) / parts;
    int i = 0;
    while (slots[i] < *chunk) ++i;
    return i + 1;
}

// Resident path: the fewest launches, then the fewest panels per CTA, whose grids are co-resident; false
// when not even one matrix is (the caller then runs the blocked path).
template <int NB, int MAXT, int RPT>
static cudaError_t gj_resident(const GJDesc* d, int count, int m, void* flags, int* st, cudaStream_t s, bool* done) {
    *done = false;
    const int threads = ((m + RPT - 1) / RPT + 31) / 32 * 32;
    if (threads > MAXT) return cudaSuccess;
    const int npanels = (m + NB - 1) / NB;
    int dev = 0, nsm = 0, coop = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev)) != cudaSuccess) return e;
    if (!coop) return cudaSuccess;
    constexpr int SMEM_MAX = 227 * 1024;
    static DeviceAttrCache attr;
    e = ensure_smem_attr(gj_resident_kernel<NB, MAXT, RPT>, SMEM_MAX - sizeof(ResShared<NB>), attr);
    if (e != cudaSuccess) return e;
    // A batch that is not co-resident as a whole goes in as few equal launches as make it so: 512 matrices
    // of 160 2604 to 1923 us, 8 of 512 2086 to 1429 against the blocked path, whose two launches per panel pass over
    // every matrix in memory.  (65 to 512 points: faster at every count up to 4096, by 6 to 60%.  Above 512 a launch
    // holds one or two matrices, and four of 600 take 2438 against 2195 us: two launches for up to three only.)
    // Fewest panels per CTA: a CTA that owns more panels updates its others before it can
    // eliminate its next one, which lengthens the chain (1024^2, L=12: 25.5 ms factor with one
    // panel per CTA, 26.9 with at least two, 29.3 with at least six)
    auto smem = [&](int ppc) { return (size_t)m * ppc * NB * sizeof(z) + (size_t)m * sizeof(int); };
    int slots[GJ_MAX_PPC];                           // matrices co-resident with 1, 2, .. panels per CTA
    int n = 0;
    while (n < npanels && n < GJ_MAX_PPC && smem(n + 1) + sizeof(ResShared<NB>) <= (size_t)SMEM_MAX) {
        int per_sm = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gj_resident_kernel<NB, MAXT, RPT>, threads, smem(n + 1));
        if (e != cudaSuccess) return e;
        slots[n] = (int)((long long)per_sm * nsm / ((npanels + n) / (n + 1)));
        if (slots[n++] >= count) break;              // the whole batch: no need to look further
    }
    int chunk = 0;
    const int ppc = gj_resident_split(count, slots, n, &chunk);
    if (ppc == 0 || (chunk < count && m > 512 && count > 3)) return cudaSuccess;
    const int P = (npanels + ppc - 1) / ppc;
    if ((e = cudaMemsetAsync(flags, 0, (size_t)(count * gj_workspace_elems(m)) * sizeof(z), s)) != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem(ppc);
    cfg.stream = s;
    cudaLaunchAttribute la[1];
    la[0].id = cudaLaunchAttributeCooperative;
    la[0].val.cooperative = 1;
    cfg.attrs = la;
    cfg.numAttrs = 1;
    for (int off = 0; off < count; off += chunk) {
        cfg.gridDim = dim3((unsigned)(std::min(chunk, count - off) * P));
        e = cudaLaunchKernelEx(&cfg, gj_resident_kernel<NB, MAXT, RPT>, d + off, m, npanels, ppc, P, st);
        if (e != cudaSuccess) return e;
        note_launch();
    }
    *done = true;
    return cudaGetLastError();
}

// RB_GJ_RESIDENT=0 selects the blocked path (read at every launch, so that a process can compare)
static bool resident_enabled() {
    const char* v = std::getenv("RB_GJ_RESIDENT");
    return !(v && v[0] == '0');
}

cudaError_t gj_invert_batch(const GJDesc* d_desc, int count, int m, void* work, int* d_status, cudaStream_t s) {
    if (count <= 0 || m <= 0) return cudaSuccess;
    if (m <= GJ_SMALL_MAX) {
        if (m <= 16) {
            const int wpc = count >= 4 * 148 ? 4 : 1;
            gj_warp_kernel<<<(count + wpc - 1) / wpc, 32 * wpc, 0, s>>>(d_desc, count, m, d_status);
        } else if (m <= 32) {
            gj_cta_kernel<1, 4><<<count, (m + 7) / 8 * 32, 0, s>>>(d_desc, m, d_status);
        } else {
            gj_cta_kernel<2, 8><<<count, (m + 7) / 8 * 32, 0, s>>>(d_desc, m, d_status);
        }
        note_launch();
        return cudaGetLastError();
    }
    if (resident_enabled() && work) {
        bool done = false;
        cudaError_t e = cudaSuccess;
        if (m <= 128) e = gj_resident<8, 128, 1>(d_desc, count, m, work, d_status, s, &done);
        else if (m <= 256) e = gj_resident<8, 256, 1>(d_desc, count, m, work, d_status, s, &done);
        else if (m <= 512) e = gj_resident<8, 512, 1>(d_desc, count, m, work, d_status, s, &done);
        else if (m <= 1024) e = gj_resident<8, 512, 2>(d_desc, count, m, work, d_status, s, &done);
        if (e != cudaSuccess || done) return e;
    }
    if (m <= 256) return gj_blocked<8, 256>(d_desc, count, m, d_status, s);
    if (m <= 512) return gj_blocked<8, 512>(d_desc, count, m, d_status, s);
    if (m <= 1024) return gj_blocked<8, 1024>(d_desc, count, m, d_status, s);
    return cudaErrorInvalidValue;
}

}  // namespace rb
