// rb_gemm_stream.cuh -- the solve's complex128 GEMM for up to 8 right-hand sides:
// D (m x n) = alpha A B + beta C, n <= 8.
//
// What bounds it: every element of A (the factorization) is used once per right-hand side, so the
// lower levels of a sweep should run at the memory rate and the upper ones, few rows each, at the
// latency of one dependent launch.  The 32x32 tile (rb_gemm_dmma.cuh) spends 32 columns of MMAs on
// them and, where it splits k, a second launch.  Here:
//  * the MMAs (m8n8k4, three real products per complex one) take the right-hand sides as their 8
//    rows and 8 rows of A as their columns;
//  * operands go from global memory to registers, U k-steps ahead of the MMAs, with no shared
//    memory and no block barrier in the k loop;
//  * a warp owns 8 RT rows; the k ranges of a split batch are the warps of one CTA, and their sums
//    meet in shared memory, in range order: no workspace and no second kernel.
// Every element sums its k-steps of 4 in order within a range and the ranges in order, with the
// ranges of the 32x32 tile (planned from count, m and k alone) and the same three products and
// epilogue: a right-hand side's result does not depend on how many are solved together.
// Measured, one right-hand side on 512^2, L=10: the leaves' 64x1x256 x1024 130 -> 72 us, a level's
// interface products 11-17 us -> 8-13 us, its parent rows 17-22 -> 13-17, the backward products
// 25-46 -> 17-29; the solve 1065 -> 795 us.  Above 8 right-hand sides it loses to the 32x32 tile,
// whose operands are shared by four warps (32 of them on 1024^2: 7.5 ms against 4.2).
#pragma once
#include "rb_gemm_dmma.cuh"

namespace rb {

constexpr int STREAM_WARPS = 16;             // most warps of a CTA, and most k ranges of a batch

// one output element's epilogue
__device__ __forceinline__ void stream_store(const GemmDesc& g, int i, int j, z acc) {
    z v = gemm_alpha(g.alpha, acc);
    if (g.C.p && !(i >= g.nobeta_r0 && i < g.nobeta_r1))
        v = gemm_beta(v, g.beta, g.C.p[vrow(g.C, i) + (long long)vcol(g.C, j) * g.C.ld]);
    g.D.p[vrow(g.D, i) + (long long)vcol(g.D, j) * g.D.ld] = v;
}

// grid: x row blocks of (warps / ks) * 8 RT rows, y problem; ks k ranges of kc (ks = 1: all of k)
template <int RT>
__global__ void __launch_bounds__(32 * STREAM_WARPS) zgemm_stream_kernel(const GemmDesc* __restrict__ descs, int ks,
                                                                         int kc) {
    constexpr int U = RT == 1 ? 4 : 3;               // k-steps fetched ahead (128 registers at 16 warps)
    constexpr int E = 2 * RT;                        // output elements per lane
    __shared__ z red[STREAM_WARPS * E * 32];
    __shared__ GemmDesc g;
    {
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(descs + blockIdx.y);
        unsigned long long* dst = reinterpret_cast<unsigned long long*>(&g);
        for (int w = threadIdx.x; w < (int)(sizeof(GemmDesc) / 8); w += blockDim.x) dst[w] = src[w];
    }
    __syncthreads();
    pdl_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lr = lane >> 2, lc = lane & 3;
    const int ngrp = (blockDim.x >> 5) / ks;
    const int slice = warp % ks, rg = warp / ks;
    if (blockIdx.x * ngrp * 8 * RT >= g.m) {         // the whole CTA
        pdl_wait();
        return;
    }
    const int r0 = (blockIdx.x * ngrp + rg) * 8 * RT;
    const bool work = r0 < g.m;
    const int kb = ks > 1 ? slice * kc : 0;
    const int ke = work ? (ks > 1 ? min(g.k, kb + kc) : g.k) : kb;

    const z* ap[RT];
    bool aok[RT];
#pragma unroll
    for (int t = 0; t < RT; ++t) {
        const int i = r0 + 8 * t + lr;
        aok[t] = i < g.m;
        ap[t] = g.A.p + (aok[t] ? vrow(g.A, i) : 0);
    }
    const bool xok = lr < g.n;
    const z* xp = g.B.p + (xok ? (long long)vcol(g.B, lr) * g.B.ld : 0);
    const int* acm = g.A.cmap;
    const int* brm = g.B.rmap;
    const int acs = g.A.cs, acl = g.A.cl, brs = g.B.rs, brl = g.B.rl;
    const long long ald = g.A.ld;

    z a[2][U][RT], x[2][U];
    auto fetch_a = [&](int k0, z (&fa)[U][RT]) {
#pragma unroll
        for (int s = 0; s < U; ++s) {
            const int k = k0 + 4 * s + lc;
            const bool ok = k < ke;
            const int kk = ok ? k : 0;
            const long long ac = (long long)(acm ? __ldg(acm + kk) : kk + (kk >= acs ? acl : 0)) * ald;
#pragma unroll
            for (int t = 0; t < RT; ++t) fa[s][t] = (ok && aok[t]) ? ap[t][ac] : zmk(0.0, 0.0);
        }
    };
    auto fetch_x = [&](int k0, z (&fx)[U]) {
#pragma unroll
        for (int s = 0; s < U; ++s) {
            const int k = k0 + 4 * s + lc;
            const bool ok = k < ke;
            const int kk = ok ? k : 0;
            const int br = brm ? __ldg(brm + kk) : kk + (kk >= brs ? brl : 0);
            fx[s] = (ok && xok) ? xp[br] : zmk(0.0, 0.0);
        }
    };
    auto fetch = [&](int k0, z (&fa)[U][RT], z (&fx)[U]) {
        fetch_a(k0, fa);
        fetch_x(k0, fx);
    };
    double p1[RT][2], p2[RT][2], p3[RT][2];
#pragma unroll
    for (int t = 0; t < RT; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) p1[t][h] = p2[t][h] = p3[t][h] = 0.0;
    auto mac = [&](const z (&fa)[U][RT], const z (&fx)[U]) {
#pragma unroll
        for (int s = 0; s < U; ++s) {
            const double xs = fx[s].x + fx[s].y;
#pragma unroll
            for (int t = 0; t < RT; ++t) dmma884(p1[t][0], p1[t][1], fx[s].x, fa[s][t].x);
#pragma unroll
            for (int t = 0; t < RT; ++t) dmma884(p2[t][0], p2[t][1], fx[s].y, fa[s][t].y);
#pragma unroll
            for (int t = 0; t < RT; ++t) dmma884(p3[t][0], p3[t][1], xs, fa[s][t].x + fa[s][t].y);
        }
    };
    if (kb < ke) fetch_a(kb, a[0]);                  // the factorization: complete before this chain
    pdl_wait();
    if (kb < ke) {
        fetch_x(kb, x[0]);
        for (int k0 = kb; k0 < ke; k0 += 8 * U) {
            fetch(k0 + 4 * U, a[1], x[1]);           // beyond ke: zeros, no loads
            mac(a[0], x[0]);
            if (k0 + 4 * U >= ke) break;
            fetch(k0 + 8 * U, a[0], x[0]);
            mac(a[1], x[1]);
        }
    }
    if (ks == 1) {
        if (!work) return;
#pragma unroll
        for (int t = 0; t < RT; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = r0 + 8 * t + 2 * lc + h;
                if (i < g.m && lr < g.n) stream_store(g, i, lr, zmk(p1[t][h] - p2[t][h], p3[t][h] - p1[t][h] - p2[t][h]));
            }
        return;
    }
#pragma unroll
    for (int t = 0; t < RT; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            red[(warp * E + 2 * t + h) * 32 + lane] = zmk(p1[t][h] - p2[t][h], p3[t][h] - p1[t][h] - p2[t][h]);
    __syncthreads();
    if (!work) return;
    // the group's ks warps share its elements; each sums the ranges in order
    for (int e = slice; e < E; e += ks) {
        z acc = red[(rg * ks * E + e) * 32 + lane];
        for (int s = 1; s < ks; ++s) acc = zadd(acc, red[((rg * ks + s) * E + e) * 32 + lane]);
        const int i = r0 + 8 * (e >> 1) + 2 * lc + (e & 1);
        if (i < g.m && lr < g.n) stream_store(g, i, lr, acc);
    }
}

}  // namespace rb
