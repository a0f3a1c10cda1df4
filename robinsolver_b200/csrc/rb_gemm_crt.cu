// rb_gemm_crt.cu -- batched complex GEMM to FP64 accuracy on the int8 tensor cores: products modulo 16
// coprime numbers, put together by the Chinese remainder theorem (the "Ozaki scheme II" of Ozaki,
// Uchino and Imamura, arXiv:2504.08009, here for complex operands).
//
// FP64 tensor cores give 37 TFLOP/s of real products, the int8 ones about 45 times that.  Every row of
// A and column of B is scaled by a power of two and rounded to integers of CRT_P = 57 bits (their largest
// entry below 2^56): anything within 2^-4 of its row's largest entry exactly, every entry to 2^-57 of
// it, where FP64 products and sums round at 2^-53.  The integers are reduced modulo 16 numbers up to
// 256; the integer product, below 2^123, is known from its 16 residues, each an int8 product with
// exact int32 accumulation.  So the whole sum over k is exact, and the result is rounded once.  Five
// passes:
//  1. launch_operand_scales: the row and column exponents;
//  2. crt_split_kernel: 16 residues of the real and imaginary parts, one byte each, laid out block by
//     block as the product kernel's shared-memory stages hold them (K-major, no swizzle);
//  3. zgemm_crt_kernel: one CTA per 128 x 80 output tile and group of moduli.  Per modulus it streams
//     the residues of A (Ar, Ai) and B ([Br | Bi], 160 rows) through a ring of bulk-copied stages;
//     two MMAs of 128 x 160 x 32 per k-step accumulate Ar Br, the sum Ar Bi + Ai Br and Ai Bi in 240
//     tensor-memory columns (the second MMA's columns overlap the first's by half, so the sum forms by
//     itself).  The next modulus' MMAs run on the other half of tensor memory while eight warps read
//     the accumulators, reduce them and write one byte per real output;
//  4. crt_combine_kernel: the 16 residues of an output to its value, sum_s r_s w_s mod M with the
//     weights in two parts of 41 bits (every sum exact in FP64), the scales, and the usual epilogue.
// Why N = 160: an MMA reads its operands from shared memory, and below N of about 128 that, not the
// tensor pipe, is its time; two accumulator sets of 3 x 80 columns fill tensor memory.
// A row or column that holds an infinity or a NaN gives NaN.
// @@FIG@@
#include <algorithm>
#include <climits>
#include <cstdint>

#include "rb_gemm_dmma.cuh"      // gemm_alpha, gemm_beta
#include "rb_kernels.h"
#include "rb_tc5.cuh"

namespace rb {

namespace {

constexpr int CRT_S = 16;                    // moduli
constexpr int CRT_P = 57;                    // bits of the scaled integers, sign included
constexpr int CRT_BM = 128, CRT_BN = 80;     // output tile
constexpr int CRT_KB = 32;                   // k of one MMA and of one plane block
constexpr int CRT_A_BLOCK = 2 * CRT_BM * CRT_KB;           // bytes per block: Ar, Ai
constexpr int CRT_B_ROWS = 2 * CRT_BN;                     // Br, Bi
constexpr int CRT_B_BLOCK = CRT_B_ROWS * CRT_KB;
constexpr int CRT_STAGE = 2 * (CRT_A_BLOCK + CRT_B_BLOCK); // two blocks (64 k)
constexpr int CRT_STAGES = 8;
constexpr int CRT_SMEM = CRT_STAGES * CRT_STAGE + 1024;
constexpr int CRT_THREADS = 384;             // producer, issuer, two idle, eight epilogue warps
constexpr int CRT_EPI = 8;
constexpr int CRT_OUT = CRT_BM * CRT_BN;     // residues of one part of a tile
constexpr int CRT_NONFINITE = 1 << 20;       // exponent mark of a row or column with an inf or NaN

// the moduli, pairwise coprime
__host__ __device__ constexpr int crt_mod(int i) {
    constexpr int t[CRT_S] = {256, 251, 249, 247, 245, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193, 191};
    return t[i];
}
__constant__ int c_mod[CRT_S] = {256, 251, 249, 247, 245, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193, 191};
// ceil(2^38 / m): x - m (mulhi(x, c) >> 6) is x's residue in [0, m] for |x| < 2^26 (m itself only for a
// negative multiple of an odd m: the error of c, below 2^-12, takes the quotient under it)
__constant__ int c_magic[CRT_S] = {1073741824, 1095131104, 1103927338, 1112866021, 1121950641, 1140572228, 1150116766, 1179733507, 1200340205, 1210915890, 1232636355, 1302738896, 1381296015, 1395319325, 1424237860, 1439151346};
// the weights w_s = (M / m_s) ((M / m_s)^-1 mod m_s) and M itself, in units of 2^CRT_LO: bits from
// 2^(125-40) up, and the 41 below
__constant__ double c_whi[CRT_S] = {
    0x1.6cfbafb7c8000p+80, 0x1.45ff525348000p+78, 0x1.f8068d00d6000p+80, 0x1.f9de50413e000p+80,
    0x1.54c0373bd2000p+80, 0x1.f41c28110c000p+79, 0x1.ca07876d08000p+80, 0x1.263bba502a000p+80,
    0x1.4f96530c30000p+80, 0x1.d3a106ee80000p+75, 0x1.b459512edc000p+80, 0x1.8ba8977d46000p+80,
    0x1.6ebafc8308000p+78, 0x1.dd196b1eb8000p+79, 0x1.bee1ecad30000p+80, 0x1.b231b3cc40000p+79};
__constant__ double c_wlo[CRT_S] = {
    0x1.d2d330a470000p+36, 0x1.95f577a67e000p+39, 0x1.b5d54881e0000p+35, 0x1.2468b62802000p+39,
    0x1.44bea91835000p+40, 0x1.e09f6f8de0000p+37, 0x1.cefcd580ca000p+40, 0x1.45af82c5c4000p+39,
    0x1.5c3119ce78000p+38, 0x1.41ee3b193a000p+40, 0x1.457c4a49ac000p+38, 0x1.33a9c7c62a000p+39,
    0x1.6d735e7a50000p+39, 0x1.c0def54f7e000p+39, 0x1.93547f5268000p+37, 0x1.a3a51c6698000p+38};
constexpr double CRT_MHI = 0x1.146fdb6e6a000p+81, CRT_MLO = 0x1.f2fddf2940000p+37;
constexpr int CRT_LO = 44;

struct CrtGeom {
    int MT, NT, KB2;                         // row tiles, column tiles, 64-deep k-steps
    long long a_bytes, b_bytes, c_off, ea_off, fb_off, total;
};
CrtGeom crt_geom(const GemmBatch& b) {
    CrtGeom g;
    g.MT = (b.max_m + CRT_BM - 1) / CRT_BM;
    g.NT = (b.max_n + CRT_BN - 1) / CRT_BN;
    g.KB2 = (b.max_k + 2 * CRT_KB - 1) / (2 * CRT_KB);
    g.a_bytes = (long long)b.count * g.MT * CRT_S * g.KB2 * 2 * CRT_A_BLOCK;
    g.b_bytes = (long long)b.count * g.NT * CRT_S * g.KB2 * 2 * CRT_B_BLOCK;
    g.c_off = g.a_bytes + g.b_bytes;
    g.ea_off = g.c_off + (long long)b.count * g.MT * g.NT * CRT_S * 2 * CRT_OUT;
    g.fb_off = g.ea_off + 4LL * b.count * g.MT * CRT_BM;
    g.total = (g.fb_off + 4LL * b.count * g.NT * CRT_BN + 255) / 256 * 256;
    return g;
}

__host__ __device__ constexpr uint32_t crt_idesc(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(CRT_BM >> 4) << 24);
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// residues of x (an integer below 2^56 in magnitude) as signed bytes, byte kk & 3 of word[s]
__device__ __forceinline__ void crt_residues(double x, int sh, uint32_t (&word)[CRT_S]) {
    constexpr double magic = 6755399441055744.0;         // 1.5 * 2^52: rounds to an integer in the low word
    constexpr float fmagic = 12582912.0f;                // 1.5 * 2^23
#pragma unroll
    for (int p = 0; p < CRT_S / 2; ++p) {
        // modulo the product of two moduli first: |y| <= (1/2 + 2^-12) 2^16
        const double mp = (double)(crt_mod(2 * p) * crt_mod(2 * p + 1)), ip = 1.0 / mp;
        const double q = rint(x * ip);
        const double y = __fma_rn(-q, mp, x);
        const float f = __int_as_float(0x4B400000 + __double2loint(__dadd_rn(y, magic))) - fmagic;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float m = (float)crt_mod(2 * p + h);
            const float t = __fadd_rn(__fmaf_rn(f, 1.0f / m, fmagic), -fmagic);
            const float r = __fmaf_rn(-t, m, f);         // |r| <= m / 2
            word[2 * p + h] |= ((uint32_t)__float_as_int(__fadd_rn(r, fmagic)) & 0xFFu) << sh;
        }
    }
}

// v 2^(CRT_P - e) rounded to an integer; the power in two factors, since neither end of the exponent
// range has it as one double.  Zero for a marked row.
__device__ __forceinline__ double crt_round(double v, int e) {
    if (e >= CRT_NONFINITE) return 0.0;
    const int p = CRT_P - e, p1 = p / 2, p2 = p - p1;
    return rint(v * oz_pow2(p1) * oz_pow2(p2));
}

// exponents of rows or columns with an infinity or a NaN (frexp exponent 1025) become the mark
__device__ __forceinline__ int crt_exp(int e) { return e > 1025 ? CRT_NONFINITE : e; }

}  // namespace

// Residue planes of one slab: s < nA an A block (problem, mt, kb: 128 rows x 32 k), else a B block
// (problem, nt, kb: 80 columns x 32 k).  Block (tile, modulus, kb) holds 16-byte chunk c (16 k) of
// row r of part p at ((p * 2 + c) * 128 + r) * 16 (A) or of row p * 80 + r at (c * 160 + row) * 16 (B).
__global__ void __launch_bounds__(256, 2) crt_split_kernel(const GemmDesc* __restrict__ descs, int MT, int NT, int KBN,
                                                           long long nA, unsigned char* __restrict__ planes,
                                                           long long a_bytes, const int* __restrict__ ea,
                                                           const int* __restrict__ fb) {
    __shared__ z S[CRT_BM * 17];             // also 80 x 17: half a block at a time
    const int tid = threadIdx.x;
    long long s = blockIdx.x;
    const bool isA = s < nA;
    if (!isA) s -= nA;
    const int kb = (int)(s % KBN);
    s /= KBN;
    const int tiles = isA ? MT : NT;
    const int tile = (int)(s % tiles);
    const int prob = (int)(s / tiles);
    const GemmDesc& g = descs[prob];
    const int rows = isA ? CRT_BM : CRT_BN;
    const long long mstride = (long long)KBN * (isA ? CRT_A_BLOCK : CRT_B_BLOCK);      // between moduli
    unsigned char* blk = planes + (isA ? 0 : a_bytes) +
                         ((long long)prob * tiles + tile) * CRT_S * mstride + (long long)kb * (isA ? CRT_A_BLOCK : CRT_B_BLOCK);
    const int* ex = (isA ? ea : fb) + ((long long)prob * tiles + tile) * rows;
    for (int half = 0; half < 2; ++half) {
        const int k0 = kb * CRT_KB + half * 16;
        for (int e = tid; e < rows * 16; e += 256) {
            // rows of A run contiguously, k runs contiguously down a column of B
            const int r = isA ? e % CRT_BM : e / 16, kk = isA ? e / CRT_BM : e % 16;
            const int i = tile * rows + r, k = k0 + kk;
            z val = zmk(0.0, 0.0);
            if (k < g.k) {
                if (isA && i < g.m) val = g.A.p[vrow(g.A, i) + (long long)vcol(g.A, k) * g.A.ld];
                if (!isA && i < g.n) val = g.B.p[vrow(g.B, k) + (long long)vcol(g.B, i) * g.B.ld];
            }
            S[r * 17 + kk] = val;
        }
        __syncthreads();
        for (int u = tid; u < 2 * rows; u += 256) {
            // unit: row r, part (0 re, 1 im): 16 values -> one 16-byte chunk per modulus
            const int r = u % rows, part = u / rows;
            const int e = crt_exp(ex[r]);
            unsigned char* dst = blk + (isA ? ((part * 2 + half) * CRT_BM + r) * 16
                                            : (half * CRT_B_ROWS + part * CRT_BN + r) * 16);
#pragma unroll 1
            for (int w = 0; w < 4; ++w) {
                uint32_t word[CRT_S];
#pragma unroll
                for (int j = 0; j < CRT_S; ++j) word[j] = 0u;
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    const z x = S[r * 17 + 4 * w + kk];
                    crt_residues(crt_round(part ? x.y : x.x, e), 8 * kk, word);
                }
#pragma unroll
                for (int j = 0; j < CRT_S; ++j) *reinterpret_cast<uint32_t*>(dst + j * mstride + 4 * w) = word[j];
            }
        }
        __syncthreads();
    }
}

// One CTA per output tile (blockIdx.x), problem (y) and group of moduli (z).  Every mbarrier wait is
// bounded; a CTA that gives up sets RB_TC5_TIMEOUT, waits (bounded) for the copies and MMAs it
// issued, frees its tensor memory and returns.
__global__ void __launch_bounds__(CRT_THREADS, 1) zgemm_crt_kernel(const GemmDesc* __restrict__ descs, int prob0, int* status,
                                                                  const unsigned char* __restrict__ planes, int MT, int NT,
                                                                  int KB2, long long a_bytes, unsigned char* __restrict__ out,
                                                                  int per_group) {
    extern __shared__ __align__(1024) unsigned char crt_smem[];
    __shared__ __align__(8) unsigned long long bars[2 * CRT_STAGES + 5];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const GemmDesc& g = descs[blockIdx.y];
    const int tiles_m = (g.m + CRT_BM - 1) / CRT_BM, tiles_n = (g.n + CRT_BN - 1) / CRT_BN;
    if ((int)blockIdx.x >= tiles_m * tiles_n) return;            // the whole CTA
    const int tm = blockIdx.x % tiles_m, tn = blockIdx.x / tiles_m;
    const long long prob = prob0 + (long long)blockIdx.y;
    const int s0 = blockIdx.z * per_group, s1 = min(CRT_S, s0 + per_group);
    const int nk = (g.k + 2 * CRT_KB - 1) / (2 * CRT_KB);        // 64-deep steps of this problem
    const unsigned char* gA = planes + ((prob * MT + tm) * CRT_S) * (long long)KB2 * 2 * CRT_A_BLOCK;
    const unsigned char* gB = planes + a_bytes + ((prob * NT + tn) * CRT_S) * (long long)KB2 * 2 * CRT_B_BLOCK;

    unsigned char* stage_base =
        reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(crt_smem) + 1023) & ~uintptr_t(1023));
    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[CRT_STAGES]);
    const uint32_t accfull0 = smem_u32(&bars[2 * CRT_STAGES]), accempty0 = smem_u32(&bars[2 * CRT_STAGES + 2]);
    const uint32_t done_bar = smem_u32(&bars[2 * CRT_STAGES + 4]);
    if (tid == 0) {
        abort_flag = 0;
        for (int q = 0; q < CRT_STAGES; ++q) {
            mbar_init(full0 + 8 * q, 1);
            mbar_init(empty0 + 8 * q, 1);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(accfull0 + 8 * q, 1);
            mbar_init(accempty0 + 8 * q, CRT_EPI);
        }
        mbar_init(done_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        // ---------------- producer: both blocks of a step, then the next, through the moduli -----------------
        bool ok = true;
        int it = 0;
        for (int s = s0; s < s1 && ok; ++s) {
            const unsigned char* a = gA + (long long)s * KB2 * 2 * CRT_A_BLOCK;
            const unsigned char* b = gB + (long long)s * KB2 * 2 * CRT_B_BLOCK;
            for (int kb = 0; kb < nk; ++kb) {
                const int q = it % CRT_STAGES, u = it / CRT_STAGES;
                if (u > 0) {
                    ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * q, (uint32_t)((u - 1) & 1), &abort_flag));
                    if (!ok) break;
                }
                if (lane == 0) {
                    const uint32_t st = smem_u32(stage_base + (size_t)q * CRT_STAGE);
                    mbar_arrive_expect_tx(full0 + 8 * q, (uint32_t)CRT_STAGE);
                    bulk_g2s(st, a + (long long)kb * 2 * CRT_A_BLOCK, 2 * CRT_A_BLOCK, full0 + 8 * q);
                    bulk_g2s(st + 2 * CRT_A_BLOCK, b + (long long)kb * 2 * CRT_B_BLOCK, 2 * CRT_B_BLOCK, full0 + 8 * q);
                }
                __syncwarp();
                ++it;
            }
        }
        if (!ok) {
            abort_flag = 1;
            if (lane == 0) atomicOr(status, RB_TC5_TIMEOUT);
            for (int i = max(0, it - CRT_STAGES); i < it; ++i)
                mbar_wait(full0 + 8 * (i % CRT_STAGES), (uint32_t)((i / CRT_STAGES) & 1), nullptr);
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer ------------------------------------------------------------------------
        constexpr uint32_t LBO_A = CRT_BM * 16, LBO_B = CRT_B_ROWS * 16, SBO = 128;
        constexpr uint32_t id2 = crt_idesc(2 * CRT_BN), id1 = crt_idesc(CRT_BN);
        bool ok = true;
        int it = 0;
        for (int s = s0; s < s1 && ok; ++s) {
            const int si = s - s0, buf = si & 1, ua = si >> 1;
            if (ua > 0) {
                ok = __all_sync(0xffffffffu, mbar_wait(accempty0 + 8 * buf, (uint32_t)((ua - 1) & 1), &abort_flag));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            const uint32_t acc = tmem + (uint32_t)(buf * 256);
            for (int kb = 0; kb < nk; ++kb, ++it) {
                const int q = it % CRT_STAGES;
                ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * q, (uint32_t)((it / CRT_STAGES) & 1), &abort_flag));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (lane == 0) {
                    const uint32_t st = smem_u32(stage_base + (size_t)q * CRT_STAGE);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t sa = st + (uint32_t)(h * CRT_A_BLOCK);
                        const uint32_t sb = st + (uint32_t)(2 * CRT_A_BLOCK + h * CRT_B_BLOCK);
                        const uint64_t ar = umma_desc(sa, LBO_A, SBO), ai = umma_desc(sa + CRT_A_BLOCK / 2, LBO_A, SBO);
                        const uint64_t bb = umma_desc(sb, LBO_B, SBO);
                        // columns: Ar Br | Ar Bi + Ai Br | Ai Bi
                        umma_i8(acc, ar, bb, id2, (kb > 0 || h > 0) ? 1u : 0u);
                        if (kb > 0 || h > 0) {
                            umma_i8(acc + CRT_BN, ai, bb, id2, 1u);
                        } else {
                            umma_i8(acc + CRT_BN, ai, bb, id1, 1u);
                            umma_i8(acc + 2 * CRT_BN, ai, umma_desc(sb + CRT_BN * 16, LBO_B, SBO), id1, 0u);
                        }
                    }
                    umma_commit(empty0 + 8 * q);
                    if (kb + 1 == nk) umma_commit(accfull0 + 8 * buf);
                }
                __syncwarp();
            }
        }
        if (!ok) {
            abort_flag = 1;
            if (lane == 0) atomicOr(status, RB_TC5_TIMEOUT);
        }
        if (lane == 0) umma_commit(done_bar);
        __syncwarp();
        mbar_wait(done_bar, 0u, nullptr);            // every MMA has ended before tensor memory is freed
    } else if (warp >= 4) {
        // ---------------- epilogue: residues of the accumulators -------------------------------------------
        const int quarter = warp & 3, half = (warp - 4) >> 2;
        const int row = quarter * 32 + lane;
        unsigned char* tile_out = out + ((prob * MT + tm) * NT + tn) * (long long)CRT_S * 2 * CRT_OUT;
        for (int s = s0; s < s1; ++s) {
            const int si = s - s0, buf = si & 1, ua = si >> 1;
            if (!__all_sync(0xffffffffu, mbar_wait(accfull0 + 8 * buf, (uint32_t)(ua & 1), &abort_flag))) {
                abort_flag = 1;
                if (lane == 0) atomicOr(status, RB_TC5_TIMEOUT);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int m = c_mod[s], mg = c_magic[s];
            const uint32_t acc = tmem + (uint32_t)(buf * 256) + ((uint32_t)(quarter * 32) << 16);
            unsigned char* o = tile_out + (long long)s * 2 * CRT_OUT + row * 8;
#pragma unroll
            for (int c = 0; c < CRT_BN / 16; ++c) {
                const int c8 = half * (CRT_BN / 16) + c;         // columns 8 c8 .. 8 c8 + 7
                int p1[8], p3[8], p2[8];
                tmem_ld8(acc + (uint32_t)(c8 * 8), p1);
                tmem_ld8(acc + (uint32_t)(CRT_BN + c8 * 8), p3);
                tmem_ld8(acc + (uint32_t)(2 * CRT_BN + c8 * 8), p2);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                uint32_t re[2] = {0u, 0u}, im[2] = {0u, 0u};
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int x = p1[e] - p2[e], y = p3[e];
                    const int rx = x - m * (__mulhi(x, mg) >> 6), ry = y - m * (__mulhi(y, mg) >> 6);
                    re[e >> 2] |= (uint32_t)rx << (8 * (e & 3));
                    im[e >> 2] |= (uint32_t)ry << (8 * (e & 3));
                }
                *reinterpret_cast<uint2*>(o + c8 * (CRT_BM * 8)) = make_uint2(re[0], re[1]);
                *reinterpret_cast<uint2*>(o + CRT_OUT + c8 * (CRT_BM * 8)) = make_uint2(im[0], im[1]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(accempty0 + 8 * buf);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
    }
}

// Outputs from their residues: a thread takes 8 columns of one row of a tile.
__global__ void __launch_bounds__(256) crt_combine_kernel(const GemmDesc* __restrict__ descs, int prob0, int MT, int NT,
                                                          const unsigned char* __restrict__ out, const int* __restrict__ ea,
                                                          const int* __restrict__ fb) {
    const GemmDesc& g = descs[blockIdx.y];
    const long long prob = prob0 + (long long)blockIdx.y;
    const int tiles_m = (g.m + CRT_BM - 1) / CRT_BM;
    // blockIdx.x: pairs of column groups of a tile (tm fastest)
    const int per = CRT_BN / 16, t = blockIdx.x / per;
    const int tm = t % tiles_m, tn = t / tiles_m;
    const int row = threadIdx.x & 127, c8 = 2 * (blockIdx.x % per) + (threadIdx.x >> 7);
    const int i = tm * CRT_BM + row, j0 = tn * CRT_BN + 8 * c8;
    if (tn * CRT_BN >= g.n || i >= g.m || j0 >= g.n) return;
    const unsigned char* p = out + ((prob * MT + tm) * NT + tn) * (long long)CRT_S * 2 * CRT_OUT + c8 * (CRT_BM * 8) + row * 8;
    constexpr double magic = 4503599627370496.0;         // 2^52
    double hr[8], lr[8], hi[8], li[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) hr[e] = lr[e] = hi[e] = li[e] = 0.0;
#pragma unroll 4
    for (int s = 0; s < CRT_S; ++s) {
        const uint2 a = *reinterpret_cast<const uint2*>(p + (long long)s * 2 * CRT_OUT);
        const uint2 b = *reinterpret_cast<const uint2*>(p + (long long)s * 2 * CRT_OUT + CRT_OUT);
        const double wh = c_whi[s], wl = c_wlo[s];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const double x = __hiloint2double(0x43300000, (int)(((e < 4 ? a.x : a.y) >> (8 * (e & 3))) & 0xFFu)) - magic;
            const double y = __hiloint2double(0x43300000, (int)(((e < 4 ? b.x : b.y) >> (8 * (e & 3))) & 0xFFu)) - magic;
            hr[e] = __fma_rn(x, wh, hr[e]);
            lr[e] = __fma_rn(x, wl, lr[e]);
            hi[e] = __fma_rn(y, wh, hi[e]);
            li[e] = __fma_rn(y, wl, li[e]);
        }
    }
    const int er = crt_exp(ea[(prob * MT + tm) * CRT_BM + row]);
    const int* fc = fb + (prob * NT + tn) * CRT_BN + 8 * c8;
    const z alpha = g.alpha, beta = g.beta;
    const long long dro = vrow(g.D, i);
    const bool use_c = g.C.p && !(i >= g.nobeta_r0 && i < g.nobeta_r1);
    const long long cro = use_c ? (long long)vrow(g.C, i) : 0;
    constexpr double rm = 1.0 / CRT_MHI;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int j = j0 + e;
        if (j >= g.n) break;
        // the symmetric representative: minus the nearest multiple of M, exact in both parts
        const double qr = rint(hr[e] * rm), qi = rint(hi[e] * rm);
        double re = __fma_rn(-qr, CRT_MHI, hr[e]) + __fma_rn(-qr, CRT_MLO, lr[e]);
        double im = __fma_rn(-qi, CRT_MHI, hi[e]) + __fma_rn(-qi, CRT_MLO, li[e]);
        const int fj = crt_exp(fc[e]);
        const int p2 = er + fj - 2 * CRT_P + CRT_LO;
        re = ldexp(re, p2);
        im = ldexp(im, p2);
        if (er >= CRT_NONFINITE || fj >= CRT_NONFINITE) re = im = __longlong_as_double(0x7ff8000000000000LL);
        z v = gemm_alpha(alpha, zmk(re, im));
        if (use_c) v = gemm_beta(v, beta, g.C.p[cro + (long long)vcol(g.C, j) * g.C.ld]);
        g.D.p[dro + (long long)vcol(g.D, j) * g.D.ld] = v;
    }
}

size_t crt_bytes(const GemmBatch& b) {
    if (b.count == 0 || b.max_m == 0 || b.max_n == 0 || b.max_k == 0 || b.max_k > CRT_MAX_K) return 0;
    return (size_t)crt_geom(b).total;
}

cudaError_t launch_gemm_crt(const GemmBatch& b, int* status, cudaStream_t s) {
    if (b.count == 0 || b.max_m == 0 || b.max_n == 0) return cudaSuccess;
    const size_t need = crt_bytes(b);
    if (need == 0 || !status || !b.crt_ws || (reinterpret_cast<uintptr_t>(b.crt_ws) & 255) || need > b.crt_cap)
        return cudaErrorInvalidValue;
    static DeviceAttrCache attr;
    cudaError_t e = ensure_smem_attr(zgemm_crt_kernel, CRT_SMEM, attr, true);
    if (e != cudaSuccess) return e;
    const CrtGeom cg = crt_geom(b);
    unsigned char* ws = static_cast<unsigned char*>(b.crt_ws);
    int* ea = reinterpret_cast<int*>(ws + cg.ea_off);
    int* fb = reinterpret_cast<int*>(ws + cg.fb_off);
    const long long nA = (long long)b.count * cg.MT * cg.KB2 * 2, nB = (long long)b.count * cg.NT * cg.KB2 * 2;
    const long long tiles = (long long)cg.MT * cg.NT;
    if (nA + nB > 0x7FFFFFFFLL || tiles * (CRT_BN / 16) > 0x7FFFFFFFLL) return cudaErrorInvalidValue;
    if ((e = launch_operand_scales(b, cg.MT * CRT_BM, cg.NT * CRT_BN, ea, fb, s)) != cudaSuccess) return e;
    crt_split_kernel<<<(unsigned)(nA + nB), 256, 0, s>>>(b.d_desc, cg.MT, cg.NT, cg.KB2 * 2, nA, ws, cg.a_bytes, ea, fb);
    note_launch();
    // groups of moduli until there are about four CTAs per SM to even the last wave out
    int groups = 1;
    while (groups < 8 && tiles * b.count * groups < 4 * 148) groups *= 2;
    for (int off = 0; off < b.count; off += 65535) {
        const int cnt = std::min(b.count - off, 65535);
        zgemm_crt_kernel<<<dim3((unsigned)tiles, cnt, groups), CRT_THREADS, CRT_SMEM, s>>>(
            b.d_desc + off, off, status, ws, cg.MT, cg.NT, cg.KB2, cg.a_bytes, ws + cg.c_off, CRT_S / groups);
        note_launch();
        crt_combine_kernel<<<dim3((unsigned)(tiles * (CRT_BN / 16)), cnt), 256, 0, s>>>(b.d_desc + off, off, cg.MT, cg.NT,
                                                                                       ws + cg.c_off, ea, fb);
        note_launch();
    }
    return cudaGetLastError();
}

}  // namespace rb
