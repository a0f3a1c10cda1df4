// rb_pivot.cuh -- Gauss-Jordan inversion of one small complex128 matrix held in registers, by a warp
// (m <= 16) or a CTA (m <= 64); shared by the leaf factor's block chain (rb_leaf.cu) and the batched
// interface inversions (rb_gj.cu).
//
// The inversion is a chain of m pivot steps, and the time of a step is what counts.  A thread holds
// whole 8-column pieces of its rows.  Rows are not exchanged: each remembers the step at which it
// was the pivot, and the caller restores the orders as it writes the result.  With row p the pivot
// of column k and x = 1/A(p,k), one step is
//     A(i,:) = A(i,:) - (A(i,k) x) A(p,:),  A(i,k) = -A(i,k) x     (i != p)
//     A(p,:) = x A(p,:),                    A(p,k) = x,
// and after the last step inv(A)(k, p_q) = A(p_k, q).
// The pivot is the row not yet used with the largest |re|+|im|; equal ones go to the smaller row.  The
// leading 15 (m <= 32) or 14 bits of the value and the row travel in one 32-bit warp reduction, and only
// where two rows share the largest such bits are their values compared whole (PivotPick; the factor
// of 16 leaves of 16 x 16 120 us without that, 123 with).
// Measured (launch included): m = 16: 6.8 us (21 with the matrix in shared memory and five block
// barriers a step), m = 32: 17 (53), m = 64: 58 (74 over several CTAs).
// With two rows per lane (m > 32) the columns rotate by one register with each step, so that the
// step is one loop body: eight of them in a row, one per register, do not stay in the instruction
// caches (m = 64: 87 us, 56 rotating; m = 32: 17, 21 rotating).
#pragma once
#include "rb_common.cuh"

namespace rb {

constexpr int PV_CG = 8;         // columns a thread holds

// The row of a warp's largest magnitude, ties to the smaller row, in two parts: what follows from the leading
// bits, and, where those tie, from the whole values.  BITS: width of the row index.  The bits of a
// non-negative double order like its value.
template <int BITS>
struct PivotPick {
    double mag;
    int r;
    unsigned key, best;
    // mag, r: this lane's candidate, if it has one (valid)
    __device__ __forceinline__ PivotPick(double mag_, bool valid, int r_) : mag(mag_), r(r_) {
        key = valid ? ((((unsigned)__double2hiint(mag) >> BITS) + 1u) << BITS) | (unsigned)((1 << BITS) - 1 - r) : 0u;
        best = __reduce_max_sync(0xffffffffu, key);
    }
    __device__ __forceinline__ int row() const { return (1 << BITS) - 1 - (int)(best & ((1u << BITS) - 1)); }
    __device__ __forceinline__ bool leads() const { return (key >> BITS) == (best >> BITS); }
    __device__ __forceinline__ bool tied() const {
        const unsigned t = __ballot_sync(0xffffffffu, leads());
        return (t & (t - 1)) != 0;
    }
    __device__ __forceinline__ int exact_row() const {
        bool in = leads();
        const unsigned hi = (unsigned)__double2hiint(mag), lo = (unsigned)__double2loint(mag);
        const unsigned mh = __reduce_max_sync(0xffffffffu, in ? hi : 0u);
        in = in && hi == mh;
        const unsigned ml = __reduce_max_sync(0xffffffffu, in ? lo : 0u);
        return (int)__reduce_min_sync(0xffffffffu, in && lo == ml ? (unsigned)r : 0xffffffffu);
    }
};

__device__ __forceinline__ z shfl_z(z v, int src) {
    return zmk(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// one element of a step: q the pivot row's value, mult = A(i,k) x (-x for the pivot row itself);
// is_k: in the pivot column
__device__ __forceinline__ void pivot_update(z& v, z q, z mult, bool is_p, bool is_k) {
    z base = v;
    if (is_p) base = zmk(0.0, 0.0);
    zfms(base, mult, q);
    v = is_k ? zneg(mult) : base;
}

// m <= 16, one warp: lane = row + 16 * column group; prow: 32 elements of the warp's shared
// memory.  myk: the step of this lane's row; pk: on lane k, the pivot row of step k.  False on an
// exactly zero pivot.
__device__ __forceinline__ bool warp_invert16(z (&v)[PV_CG], int m, z* prow, int& myk, int& pk) {
    const int lane = threadIdx.x & 31, r = lane & 15, hf = lane >> 4;
    bool ok = true, used = r >= m;
    myk = 0;
    pk = 0;
#pragma unroll
    for (int grp = 0; grp < 2; ++grp) {
#pragma unroll
        for (int e = 0; e < PV_CG; ++e) {
            const int k = grp * PV_CG + e;
            if (k >= m) break;
            const bool mine = hf == grp;
            const PivotPick<5> pick(zabs1(v[e]), mine && !used, r);
            const z f = shfl_z(v[e], r + 16 * grp);
            int p = pick.row();
            const bool tied = pick.tied();
            z pv, x;
            for (bool again = tied;; again = false) {  // looked at behind the reciprocal, where it is free
                pv = shfl_z(v[e], p + 16 * grp);
                x = zrcp(pv);
                if (!again) break;
                p = pick.exact_row();
            }
            const bool is_p = r == p;
            z* pr = prow + (k & 1) * 16 + hf * PV_CG;
            if (is_p) {
#pragma unroll
                for (int c = 0; c < PV_CG; ++c) pr[c] = v[c];
            }
            if (pv.x == 0.0 && pv.y == 0.0) ok = false;
            const z mult = is_p ? zneg(x) : zmul(f, x);
            if (is_p) { used = true; myk = k; }
            if (lane == k) pk = p;
            __syncwarp();
#pragma unroll
            for (int c = 0; c < PV_CG; ++c) pivot_update(v[c], pr[c], mult, is_p, mine && c == e);
        }
    }
    return ok;
}

// m <= 32 RPL, one CTA: lane + 32 i = row, warp = column group; as many warps as column groups.
// The warp that holds the next pivot column updates that column first, finds its pivot and publishes
// it (the column, the pivot row, the reciprocal) before it updates its other columns: one block
// barrier per step.  myk[i]: the step of row lane + 32 i; sh.pk[k]: the pivot row of step k.  With
// RPL > 1, v[i][c] is column 8 * warp + (c + m) % 8 on return.  False on an exactly zero pivot (on
// some thread).  The caller has a block barrier between two calls on the same sh.
template <int RPL, int NG>
struct PivotShared {
    z fcol[2][32 * RPL];
    z prow[NG][2][PV_CG];
    z pinv[2];
    int piv[2];
    int pk[32 * RPL];
};

template <int RPL, int NG>
__device__ __forceinline__ bool cta_invert(z (&v)[RPL][PV_CG], int m, PivotShared<RPL, NG>& sh, int (&myk)[RPL]) {
    constexpr int BITS = RPL == 1 ? 5 : 6;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    bool ok = true;
    bool used[RPL];
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
        used[i] = lane + 32 * i >= m;
        myk[i] = 0;
    }
    // finds and publishes the pivot of column k, this warp's register column c
    auto publish = [&](int c, int k) {
        const int s = k & 1;
        double mag = 0.0;
        int row = -1;
#pragma unroll
        for (int i = 0; i < RPL; ++i) {
            const double a = zabs1(v[i][c]);
            if (!used[i] && (row < 0 || a > mag)) {
                mag = a;
                row = lane + 32 * i;
            }
        }
        const PivotPick<BITS> pick(mag, row >= 0, row);
        const bool tied = pick.tied();
        bool zero = false;
        auto put = [&](int p) {
            zero = false;
#pragma unroll
            for (int i = 0; i < RPL; ++i)
                if (lane + 32 * i == p) {
                    sh.pinv[s] = zrcp(v[i][c]);
                    sh.piv[s] = p;
                    sh.pk[k] = p;
                    zero = v[i][c].x == 0.0 && v[i][c].y == 0.0;
                }
        };
#pragma unroll
        for (int i = 0; i < RPL; ++i) sh.fcol[s][lane + 32 * i] = v[i][c];
        put(pick.row());
        if (tied) {                                    // looked at behind the reciprocal, where it is free
            __syncwarp();
            put(pick.exact_row());
        }
        if (zero) ok = false;
    };
    if (w == 0) publish(0, 0);
    constexpr int STEPS = RPL == 1 ? PV_CG : 1;      // steps per loop body; with 1 the columns rotate
    for (int k0 = 0; k0 < m; k0 += STEPS) {
#pragma unroll
        for (int e = 0; e < STEPS; ++e) {
            const int k = k0 + e, s = k & 1;
            if (k >= m) break;
            const int en = (e + 1) % PV_CG;                        // the next pivot column's register
            __syncthreads();
            const int p = sh.piv[s];
            const z x = sh.pinv[s];
            const bool next = k + 1 < m && w == (k + 1) / PV_CG;
            const bool mine = w == k / PV_CG;
            z* pr = sh.prow[w][s];
            z mult[RPL];
            bool is_p[RPL];
            z vp = zmk(0.0, 0.0);
#pragma unroll
            for (int i = 0; i < RPL; ++i) {
                is_p[i] = lane + 32 * i == p;
                if (is_p[i]) {
#pragma unroll
                    for (int c = 0; c < PV_CG; ++c) pr[c] = v[i][c];
                    used[i] = true;
                    myk[i] = k;
                }
                if (RPL == 1 || (p >> 5) == i) vp = v[i][en];
                mult[i] = is_p[i] ? zneg(x) : zmul(sh.fcol[s][lane + 32 * i], x);
            }
            const z qn = shfl_z(vp, p & 31);                       // the pivot row at the next pivot column
#pragma unroll
            for (int i = 0; i < RPL; ++i) pivot_update(v[i][en], qn, mult[i], is_p[i], false);
            if (next) publish(en, k + 1);
            __syncwarp();
#pragma unroll
            for (int c = 0; c < PV_CG; ++c) {
                if (c == en) continue;
                const z q = pr[c];
#pragma unroll
                for (int i = 0; i < RPL; ++i) pivot_update(v[i][c], q, mult[i], is_p[i], mine && c == e);
            }
            if (STEPS == 1) {
#pragma unroll
                for (int i = 0; i < RPL; ++i) {
                    const z t = v[i][0];
#pragma unroll
                    for (int c = 1; c < PV_CG; ++c) v[i][c - 1] = v[i][c];
                    v[i][PV_CG - 1] = t;
                }
            }
        }
    }
    return ok;
}

}  // namespace rb
