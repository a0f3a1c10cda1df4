// rb_gemm_crt.cu -- batched complex GEMM on the int8 tensor cores, for the FP64 factor's large maps: products
// modulo 16 coprime numbers, put together by the Chinese remainder theorem (the "Ozaki scheme II" of Ozaki,
// Uchino and Imamura, arXiv:2504.08009, here for complex operands).
//
// FP64 tensor cores give 37 TFLOP/s of real products, the int8 ones about 45 times that.  Every row of
// A and column of B is scaled by a power of two and rounded to integers of CRT_P = 57 bits (their largest
// entry below 2^56).  The integers are reduced modulo 16 numbers up to 256; the integer product, below
// 2^123, is known from its 16 residues, each an int8 product with exact int32 accumulation.
// Errors: an entry within 2^-4 of its row's or column's largest is held exactly, a smaller one to 2^-57 of
// that largest and so with fewer bits the smaller it is; the sum over k adds none; the weights that put
// the residues together are cut at 2^44, which leaves the integer up to 2^53.4 off, about 2^-57 of the
// product of the two largest entries; then one rounding of the result.  So an element is off by at most
// about 2^-56 (amax_i sum_k |b_kj| + bmax_j sum_k |a_ik|), where a chain of FP64 products is off by some
// 2^-53 sqrt(k) sum_k |a_ik| |b_kj|: less where the operands are even, more where both are graded along k.
// Which products of the factor are the one and which the other was measured (crt_level, rb_tree.cpp).
// Four passes:
//  1. launch_operand_scales: the row and column exponents;
//  2. crt_split_kernel: 16 residues of the real and imaginary parts, one byte each, laid out block by
//     block as the product kernel's shared memory holds them (K-major, 128-byte swizzle);
//  3. zgemm_crt_kernel: per modulus, the residues of B's column tile ([Br | Bi], 160 rows) stay in shared
//     memory (k up to 512; above, they stream too) while those of A (Ar, Ai) stream past through a ring
//     of bulk-copied stages.  MMAs of
//     128 x 160 x 32 accumulate Ar Br, the sum Ar Bi + Ai Br and Ai Bi in 240 tensor-memory columns
//     (Ai's columns overlap Ar's by half, so the sum forms by itself).  The next tile's MMAs run on the
//     other half of tensor memory while eight warps read the accumulators, reduce them and write one
//     byte per real output;
//  4. crt_combine_kernel: the 16 residues of an output to its value, sum_s r_s w_s mod M with the
//     cut weights in two parts of 41 bits (every sum of which is exact in FP64), the scales, and the usual
//     epilogue.
// Why N = 160: an MMA reads its operands from shared memory, and below N of about 128 that, not the
// tensor pipe, is its time; two accumulator sets of 3 x 80 columns fill tensor memory.
// A row or column that holds an infinity or a NaN gives NaN.
// Measured against the FP64 tensor-core tiles (complex m x n x k, count; us): 2048 x 2048 x 1024, 4: 3196 to
// 1376; 1536 x 1536 x 512, 8: 1874 to 1016; 512 x 1536 x 512, 4: 357 to 261; 1024 x 2048 x 1024, 1: 462 to 230;
// 768 x 768 x 256, 32: 988 to 826; 256 x 768 x 256, 16: 190 to 236; 384 x 384 x 128, 128: 548 to 808.  The first spends
// 29 + 26 us on scales, 294 on the split (its 16 residues per entry are issue bound), 829 on products
// (the tensor pipe alone would take 520) and 205 on the outputs (FP64 sums, issue
// bound too; DRAM 43% busy).
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
constexpr int CRT_KB = 128;                  // k of one plane block: a row is 128 bytes
constexpr int CRT_A_BLOCK = CRT_BM * CRT_KB;               // bytes per block of one part (Ar or Ai)
constexpr int CRT_B_ROWS = 2 * CRT_BN;                     // Br, Bi
constexpr int CRT_B_BLOCK = CRT_B_ROWS * CRT_KB;
constexpr int CRT_CHUNKS = 4;                              // blocks of a B tile that stay resident (k <= 512)
constexpr int CRT_STAGES = 4;                              // stages of Ar and Ai (and B's block, above) of 128 k
constexpr int CRT_SMEM = CRT_STAGES * (2 * CRT_A_BLOCK + CRT_B_BLOCK) + 1024;
static_assert(CRT_SMEM <= 227 * 1024 - 1024, "shared memory");
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
    int MT, NT, KB;                          // row tiles, column tiles, 128-deep blocks
    long long a_bytes, b_bytes, c_off, ea_off, fb_off, total;
};
CrtGeom crt_geom(const GemmBatch& b) {
    CrtGeom g;
    g.MT = (b.max_m + CRT_BM - 1) / CRT_BM;
    g.NT = (b.max_n + CRT_BN - 1) / CRT_BN;
    g.KB = (b.max_k + CRT_KB - 1) / CRT_KB;
    g.a_bytes = (long long)b.count * g.MT * CRT_S * g.KB * 2 * CRT_A_BLOCK;
    g.b_bytes = (long long)b.count * g.NT * CRT_S * g.KB * CRT_B_BLOCK;
    g.c_off = g.a_bytes + g.b_bytes;
    g.ea_off = g.c_off + (long long)b.count * g.MT * g.NT * CRT_S * 2 * CRT_OUT;
    g.fb_off = g.ea_off + 4LL * b.count * g.MT * CRT_BM;
    g.total = (g.fb_off + 4LL * b.count * g.NT * CRT_BN + 255) / 256 * 256;
    return g;
}

__host__ __device__ constexpr uint32_t crt_idesc(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(CRT_BM >> 4) << 24);
}

// UMMA shared-memory descriptor, K-major, 128-byte swizzle: rows of 128 bytes, 16-byte chunk c of row r
// at c ^ (r % 8), 8-row groups 1024 bytes apart and aligned; a k-step of 32 is 32 bytes further on.
// Version 1 (sm_100), base offset 0, layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t crt_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}

// 1 on one lane of a converged warp
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(p));
    return p;
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// a pair of moduli: their product, and each, with reciprocals
struct CrtPair {
    double mp, ip;
    float m0, i0, m1, i1;
};
constexpr CrtPair crt_pair(int p) {
    const double mp = (double)(crt_mod(2 * p) * crt_mod(2 * p + 1));
    const float m0 = (float)crt_mod(2 * p), m1 = (float)crt_mod(2 * p + 1);
    return CrtPair{mp, 1.0 / mp, m0, 1.0f / m0, m1, 1.0f / m1};
}
__constant__ CrtPair c_pair[CRT_S / 2] = {crt_pair(0), crt_pair(1), crt_pair(2), crt_pair(3),
                                          crt_pair(4), crt_pair(5), crt_pair(6), crt_pair(7)};

// residues of x (an integer below 2^56 in magnitude) modulo a pair of moduli, as signed bytes
__device__ __forceinline__ void crt_residues(double x, const CrtPair& c, uint32_t& r0, uint32_t& r1) {
    constexpr double magic = 6755399441055744.0;         // 1.5 * 2^52: rounds to an integer in the low word
    constexpr float fmagic = 12582912.0f;                // 1.5 * 2^23
    // modulo the product of the two first: |y| <= (1/2 + 2^-12) 2^16
    const double q = __dadd_rn(__fma_rn(x, c.ip, magic), -magic);
    const double y = __fma_rn(-q, c.mp, x);
    const float f = __fadd_rn(__int_as_float(0x4B400000 + __double2loint(__dadd_rn(y, magic))), -fmagic);
    const float t0 = __fadd_rn(__fmaf_rn(f, c.i0, fmagic), -fmagic), t1 = __fadd_rn(__fmaf_rn(f, c.i1, fmagic), -fmagic);
    // |f - t m| <= m / 2, in the low byte
    r0 = (uint32_t)__float_as_int(__fadd_rn(__fmaf_rn(-t0, c.m0, f), fmagic));
    r1 = (uint32_t)__float_as_int(__fadd_rn(__fmaf_rn(-t1, c.m1, f), fmagic));
}
// the low bytes of four words
__device__ __forceinline__ uint32_t crt_pack(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

// v 2^p in two factors: neither end of the exponent range has 2^p as one double
__device__ __forceinline__ double crt_scale(double v, int p) {
    const int p1 = p / 2;
    return v * oz_pow2(p1) * oz_pow2(p - p1);
}

// v 2^p for the outputs' wider range of p (both exponents): three factors
__device__ __forceinline__ double crt_ldexp(double v, int p) {
    const int p1 = p / 3, p2 = (p - p1) / 2;
    return v * oz_pow2(p1) * oz_pow2(p2) * oz_pow2(p - p1 - p2);
}

// The problem whose A planes problem p uses: the first of the run of neighbours with the same A as its
// own (the two column halves of Y1, Y2 and of a map's rows read one A: split once, 6 units of 8 of a map).
__device__ __forceinline__ int crt_a_owner(const GemmDesc* descs, int p) {
    const ZView a = descs[p].A;
    const int m = descs[p].m, k = descs[p].k;
    while (p > 0) {
        const GemmDesc& o = descs[p - 1];
        if (o.A.p != a.p || o.A.ld != a.ld || o.A.rmap != a.rmap || o.A.cmap != a.cmap || o.A.rs != a.rs || o.A.rl != a.rl ||
            o.A.cs != a.cs || o.A.cl != a.cl || o.m != m || o.k != k)
            break;
        --p;
    }
    return p;
}

// exponents of rows or columns with an infinity or a NaN (frexp exponent 1025) become the mark
__device__ __forceinline__ int crt_exp(int e) { return e > 1025 ? CRT_NONFINITE : e; }

}  // namespace

// Residue planes of one slab of 16 rows x 128 k: s < nA of A (problem, mt, kb, 16-row group), else of B
// (problem, nt, kb, 16-column group).  Blocks: A [problem][mt][modulus][kb][part], B
// [problem][nt][modulus][kb] with Br's 80 rows, then Bi's; chunk c (16 k) of row r of a block at
// r * 128 + (c ^ (r % 8)) * 16.  A thread takes one chunk of one part of one row, so that a warp's store
// of one modulus is 512 bytes in a row.
__global__ void __launch_bounds__(256, 3) crt_split_kernel(const GemmDesc* __restrict__ descs, int MT, int NT, int KB,
                                                           long long nA, unsigned char* __restrict__ planes,
                                                           long long a_bytes, const int* __restrict__ ea,
                                                           const int* __restrict__ fb) {
    __shared__ z S[16 * 8 * 17];             // [row][chunk][16 of 17]
    const int tid = threadIdx.x;
    long long s = blockIdx.x;
    const bool isA = s < nA;
    if (!isA) s -= nA;
    const int rows = isA ? CRT_BM : CRT_BN, groups = rows / 16;
    const int grp = (int)(s % groups);
    s /= groups;
    const int kb = (int)(s % KB);
    s /= KB;
    const int tiles = isA ? MT : NT;
    const int tile = (int)(s % tiles);
    const int prob = (int)(s / tiles);
    if (isA && crt_a_owner(descs, prob) != prob) return;
    const GemmDesc& g = descs[prob];
    const int i0 = tile * rows + grp * 16, k0 = kb * CRT_KB;
    for (int e = tid; e < 16 * CRT_KB; e += 256) {
        // rows of A run contiguously, k runs contiguously down a column of B
        const int r = isA ? e % 16 : e / CRT_KB, kk = isA ? e / 16 : e % CRT_KB;
        const int i = i0 + r, k = k0 + kk;
        z val = zmk(0.0, 0.0);
        if (k < g.k) {
            if (isA && i < g.m) val = g.A.p[vrow(g.A, i) + (long long)vcol(g.A, k) * g.A.ld];
            if (!isA && i < g.n) val = g.B.p[vrow(g.B, k) + (long long)vcol(g.B, i) * g.B.ld];
        }
        S[(r * 8 + (kk >> 4)) * 17 + (kk & 15)] = val;
    }
    __syncthreads();
    const int c = tid & 7, r = (tid >> 3) & 15, part = tid >> 7;
    const long long block = isA ? 2 * CRT_A_BLOCK : CRT_B_BLOCK, mstride = KB * block;      // per kb; between moduli
    const int e = crt_exp((isA ? ea : fb)[(long long)prob * tiles * rows + i0 + r]);
    const int rr = (isA ? 0 : part * CRT_BN) + grp * 16 + r;
    unsigned char* dst = planes + (isA ? part * CRT_A_BLOCK : a_bytes) + ((long long)prob * tiles + tile) * CRT_S * mstride +
                         kb * block + rr * CRT_KB + ((c ^ (rr & 7)) << 4);
    double x[16];
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
        const z v = S[(r * 8 + c) * 17 + kk];
        // 2^56 > |x|; zero for a marked row
        x[kk] = e >= CRT_NONFINITE ? 0.0 : rint(crt_scale(part ? v.y : v.x, CRT_P - e));
    }
    // rolled: eight unrolled pairs of 16 values hold too many registers for three CTAs per SM
#pragma unroll 1
    for (int p = 0; p < CRT_S / 2; ++p, dst += 2 * mstride) {
        const CrtPair pr = c_pair[p];
        uint32_t w0[4], w1[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            uint32_t a[4], b[4];
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) crt_residues(x[4 * w + kk], pr, a[kk], b[kk]);
            w0[w] = crt_pack(a[0], a[1], a[2], a[3]);
            w1[w] = crt_pack(b[0], b[1], b[2], b[3]);
        }
        *reinterpret_cast<uint4*>(dst) = make_uint4(w0[0], w0[1], w0[2], w0[3]);
        *reinterpret_cast<uint4*>(dst + mstride) = make_uint4(w1[0], w1[1], w1[2], w1[3]);
    }
}

// One CTA per column tile and run of up to R row tiles (blockIdx.x), problem (y) and group of moduli (z).
// Up to k = 512 B's column tile (160 rows x k) stays in shared memory for a modulus while the row tiles
// of A stream past it; its blocks are refilled for the next modulus as the last row tile lets go of
// them.  Above, B's blocks stream beside A's: a resident tile would leave room for two stages only
// (k = 1024: 1014 us of products for 4 x 2048 x 2048, 829 streaming).  Every mbarrier wait is bounded; a CTA that gives up sets RB_TC5_TIMEOUT; in every
// CTA the copies and MMAs it issued are waited for (bounded) before its tensor memory is freed and it returns.
__global__ void __launch_bounds__(CRT_THREADS, 1) zgemm_crt_kernel(const GemmDesc* __restrict__ descs, int* status,
                                                                  const unsigned char* __restrict__ planes, int MT, int NT,
                                                                  int KB, long long a_bytes, unsigned char* __restrict__ out,
                                                                  int R, int per_group) {
    extern __shared__ __align__(1024) unsigned char crt_smem[];
    __shared__ __align__(8) unsigned long long bars[2 * CRT_STAGES + 2 * CRT_CHUNKS + 5];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const GemmDesc& g = descs[blockIdx.y];
    const int tiles_m = (g.m + CRT_BM - 1) / CRT_BM, tiles_n = (g.n + CRT_BN - 1) / CRT_BN;
    const int runs = (MT + R - 1) / R;
    const int tn = blockIdx.x / runs, t0 = (blockIdx.x % runs) * R, t1 = min(tiles_m, t0 + R);
    if (tn >= tiles_n || t0 >= tiles_m) return;                  // the whole CTA
    const long long prob = blockIdx.y;
    const int s0 = blockIdx.z * per_group, s1 = min(CRT_S, s0 + per_group);
    const int nk = max(1, (g.k + CRT_KB - 1) / CRT_KB);          // blocks of this problem (k = 0: one of zeros)
    const long long a_mod = (long long)KB * 2 * CRT_A_BLOCK, b_mod = (long long)KB * CRT_B_BLOCK;
    const unsigned char* gB = planes + a_bytes + (prob * NT + tn) * CRT_S * b_mod;

    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(crt_smem) + 1023) & ~uintptr_t(1023));
    // resident: four blocks of B, then the stages of A; streaming: stages of A and a block of B each
    const bool resident = nk <= CRT_CHUNKS;
    const uint32_t sB = smem_u32(base) + (resident ? 0u : (uint32_t)(2 * CRT_A_BLOCK));
    const uint32_t sA = smem_u32(base) + (resident ? (uint32_t)(CRT_CHUNKS * CRT_B_BLOCK) : 0u);
    const uint32_t stage_bytes = 2 * CRT_A_BLOCK + (resident ? 0 : CRT_B_BLOCK);
    const uint32_t afull0 = smem_u32(&bars[0]), aempty0 = afull0 + 8 * CRT_STAGES;
    const uint32_t bfull0 = aempty0 + 8 * CRT_STAGES, bempty0 = bfull0 + 8 * CRT_CHUNKS;
    const uint32_t accfull0 = bempty0 + 8 * CRT_CHUNKS, accempty0 = accfull0 + 16, done_bar = accempty0 + 16;
    if (tid == 0) {
        abort_flag = 0;
        for (int q = 0; q < 2 * CRT_STAGES + 2 * CRT_CHUNKS + 2; ++q) mbar_init(afull0 + 8 * q, 1);
        mbar_init(accempty0, CRT_EPI);
        mbar_init(accempty0 + 8, CRT_EPI);
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
        // ---------------- producer, in the issuer's order ------------------------------------------------
        if (lane == 0) {
            bool ok = true;
            const unsigned char* gA = planes + (long long)crt_a_owner(descs, (int)prob) * MT * CRT_S * a_mod;
            uint32_t q = 0;                          // stage
            int it = 0, nb = 0;                      // stages and resident B blocks issued
            uint32_t par = 1u;                       // parity of the A stage's previous release
            for (int s = s0; s < s1 && ok; ++s) {
                const unsigned char* a = gA + ((long long)t0 * CRT_S + s) * a_mod;
                const unsigned char* bsrc = gB + s * b_mod;
                for (int tm = t0; tm < t1 && ok; ++tm, a += CRT_S * a_mod) {
                    for (int kb = 0; kb < nk && ok; ++kb) {
                        if (resident && tm == t0) {
                            if (s > s0) ok = mbar_wait(bempty0 + 8 * kb, (uint32_t)((s - s0 - 1) & 1), &abort_flag);
                            if (!ok) break;
                            mbar_arrive_expect_tx(bfull0 + 8 * kb, CRT_B_BLOCK);
                            bulk_g2s(sB + (uint32_t)(kb * CRT_B_BLOCK), bsrc + kb * CRT_B_BLOCK, CRT_B_BLOCK, bfull0 + 8 * kb);
                            ++nb;
                        }
                        if (it >= CRT_STAGES) ok = mbar_wait(aempty0 + 8 * q, par, &abort_flag);
                        if (!ok) break;
                        mbar_arrive_expect_tx(afull0 + 8 * q, stage_bytes);
                        bulk_g2s(sA + q * stage_bytes, a + kb * 2 * CRT_A_BLOCK, 2 * CRT_A_BLOCK, afull0 + 8 * q);
                        if (!resident) bulk_g2s(sB + q * stage_bytes, bsrc + kb * CRT_B_BLOCK, CRT_B_BLOCK, afull0 + 8 * q);
                        ++it;
                        if (++q == CRT_STAGES) {
                            q = 0;
                            par ^= 1u;
                        }
                    }
                }
            }
            if (!ok) {
                abort_flag = 1;
                atomicOr(status, RB_TC5_TIMEOUT);
            }
            // no copy may still target this CTA's memory when it exits, whichever warp gave up: wait
            // (bounded) for the last fill of every stage and resident block
            for (int i = max(0, it - CRT_STAGES); i < it; ++i)
                mbar_wait(afull0 + 8 * (i % CRT_STAGES), (uint32_t)((i / CRT_STAGES) & 1), nullptr);
            for (int i = max(0, nb - nk); i < nb; ++i) mbar_wait(bfull0 + 8 * (i % nk), (uint32_t)((i / nk) & 1), nullptr);
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer ------------------------------------------------------------------------
        // the whole warp runs the loop (the descriptors then live in uniform registers); one elected lane
        // issues.  Both parts of a k block are one wait and one commit: 640 cycles of MMAs.
        constexpr uint32_t id2 = crt_idesc(2 * CRT_BN), id1 = crt_idesc(CRT_BN);
        const uint32_t elected = elect_one();
        const uint64_t da0 = crt_desc(sA), db0 = crt_desc(sB);
        bool ok = true;
        uint32_t q = 0;                              // stage
        int ai = 0;                                  // accumulator sets begun
        uint32_t par = 0u;                           // parity of the A stage's fill
        for (int s = s0; s < s1 && ok; ++s) {
            for (int tm = t0; tm < t1 && ok; ++tm, ++ai) {
                const int buf = ai & 1, ua = ai >> 1;
                if (ua > 0) ok = mbar_wait(accempty0 + 8 * buf, (uint32_t)((ua - 1) & 1), &abort_flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + (uint32_t)(buf * 256);
                for (int kb = 0; kb < nk; ++kb) {
                    if (resident && tm == t0) ok = mbar_wait(bfull0 + 8 * kb, (uint32_t)((s - s0) & 1), &abort_flag);
                    ok = ok && mbar_wait(afull0 + 8 * q, par, &abort_flag);
                    if (!ok) break;
                    if (elected) {
                        // Ar: columns Ar Br | Ar Bi; Ai: columns Ai Br (onto Ar Bi) | Ai Bi
                        const uint64_t da = da0 + q * (stage_bytes >> 4), dai = da + (CRT_A_BLOCK >> 4);
                        const uint64_t db = db0 + (resident ? (uint32_t)kb * (CRT_B_BLOCK >> 4) : q * (stage_bytes >> 4));
                        umma_i8(acc, da, db, id2, kb > 0 ? 1u : 0u);
#pragma unroll
                        for (int j = 1; j < CRT_KB / 32; ++j) umma_i8(acc, da + 2 * j, db + 2 * j, id2, 1u);
                        if (kb > 0) {
                            umma_i8(acc + CRT_BN, dai, db, id2, 1u);
                        } else {
                            umma_i8(acc + CRT_BN, dai, db, id1, 1u);
                            umma_i8(acc + 2 * CRT_BN, dai, db + (CRT_BN * CRT_KB >> 4), id1, 0u);
                        }
#pragma unroll
                        for (int j = 1; j < CRT_KB / 32; ++j) umma_i8(acc + CRT_BN, dai + 2 * j, db + 2 * j, id2, 1u);
                        umma_commit(aempty0 + 8 * q);
                        if (resident && tm + 1 == t1) umma_commit(bempty0 + 8 * kb);
                        if (kb + 1 == nk) umma_commit(accfull0 + 8 * buf);
                    }
                    __syncwarp();
                    if (++q == CRT_STAGES) {
                        q = 0;
                        par ^= 1u;
                    }
                }
            }
        }
        if (!ok) {
            abort_flag = 1;
            if (elected) atomicOr(status, RB_TC5_TIMEOUT);
        }
        if (elected) umma_commit(done_bar);
        __syncwarp();
        mbar_wait(done_bar, 0u, nullptr);            // every MMA has ended before tensor memory is freed
    } else if (warp >= 4) {
        // ---------------- epilogue: residues of the accumulators -------------------------------------------
        const int quarter = warp & 3, half = (warp - 4) >> 2;
        const int row = quarter * 32 + lane;
        int ai = 0;
        bool ok = true;
        for (int s = s0; s < s1 && ok; ++s) {
            const int m = c_mod[s], mg = c_magic[s];
            for (int tm = t0; tm < t1; ++tm, ++ai) {
                const int buf = ai & 1, ua = ai >> 1;
                ok = __all_sync(0xffffffffu, mbar_wait(accfull0 + 8 * buf, (uint32_t)(ua & 1), &abort_flag));
                if (!ok) {
                    abort_flag = 1;
                    if (lane == 0) atomicOr(status, RB_TC5_TIMEOUT);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + (uint32_t)(buf * 256) + ((uint32_t)(quarter * 32) << 16);
                unsigned char* o = out + (((prob * MT + tm) * NT + tn) * CRT_S + s) * 2LL * CRT_OUT + row * 8;
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
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
    }
}

// Outputs from their residues: a thread takes 4 columns of one row of a tile; two neighbours share the
// 8 residues a row has in a column group.
__global__ void __launch_bounds__(256, 4) crt_combine_kernel(const GemmDesc* __restrict__ descs, int MT, int NT,
                                                          const unsigned char* __restrict__ out, const int* __restrict__ ea,
                                                          const int* __restrict__ fb) {
    const GemmDesc& g = descs[blockIdx.y];
    const long long prob = blockIdx.y;
    const int tiles_m = max(1, (g.m + CRT_BM - 1) / CRT_BM);
    // blockIdx.x: column groups of a tile (tm fastest)
    const int c8 = blockIdx.x % (CRT_BN / 8), t = blockIdx.x / (CRT_BN / 8);
    const int tm = t % tiles_m, tn = t / tiles_m;
    const int row = threadIdx.x >> 1, c4 = 2 * c8 + (threadIdx.x & 1);
    const int i = tm * CRT_BM + row, j0 = tn * CRT_BN + 4 * c4;
    if (i >= g.m || j0 >= g.n) return;
    const unsigned char* p = out + ((prob * MT + tm) * NT + tn) * (long long)CRT_S * 2 * CRT_OUT + c8 * (CRT_BM * 8) +
                             threadIdx.x * 4;
    constexpr double magic = 4503599627370496.0;         // 2^52
    double hr[4], lr[4], hi[4], li[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) hr[e] = lr[e] = hi[e] = li[e] = 0.0;
#pragma unroll 8
    for (int s = 0; s < CRT_S; ++s) {
        const uint32_t a = *reinterpret_cast<const uint32_t*>(p + (long long)s * 2 * CRT_OUT);
        const uint32_t b = *reinterpret_cast<const uint32_t*>(p + (long long)s * 2 * CRT_OUT + CRT_OUT);
        const double wh = c_whi[s], wl = c_wlo[s];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const double x = __hiloint2double(0x43300000, (int)((a >> (8 * e)) & 0xFFu)) - magic;
            const double y = __hiloint2double(0x43300000, (int)((b >> (8 * e)) & 0xFFu)) - magic;
            hr[e] = __fma_rn(x, wh, hr[e]);
            lr[e] = __fma_rn(x, wl, lr[e]);
            hi[e] = __fma_rn(y, wh, hi[e]);
            li[e] = __fma_rn(y, wl, li[e]);
        }
    }
    const int er = crt_exp(ea[(prob * MT + tm) * CRT_BM + row]);
    const int* fc = fb + (prob * NT + tn) * CRT_BN + 4 * c4;
    const z alpha = g.alpha, beta = g.beta;
    const long long dro = vrow(g.D, i);
    const bool use_c = g.C.p && !(i >= g.nobeta_r0 && i < g.nobeta_r1);
    const long long cro = use_c ? (long long)vrow(g.C, i) : 0;
    constexpr double rm = 1.0 / CRT_MHI;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int j = j0 + e;
        if (j >= g.n) break;
        // the symmetric representative: minus the nearest multiple of M, exact in both parts
        const double qr = rint(hr[e] * rm), qi = rint(hi[e] * rm);
        double re = __fma_rn(-qr, CRT_MHI, hr[e]) + __fma_rn(-qr, CRT_MLO, lr[e]);
        double im = __fma_rn(-qi, CRT_MHI, hi[e]) + __fma_rn(-qi, CRT_MLO, li[e]);
        const int fj = crt_exp(fc[e]);
        const int p2 = er + fj - 2 * CRT_P + CRT_LO;
        if (er >= CRT_NONFINITE || fj >= CRT_NONFINITE) {
            re = im = __longlong_as_double(0x7ff8000000000000LL);
        } else {
            re = crt_ldexp(re, p2);
            im = crt_ldexp(im, p2);
        }
        z v = gemm_alpha(alpha, zmk(re, im));
        if (use_c) v = gemm_beta(v, beta, g.C.p[cro + (long long)vcol(g.C, j) * g.C.ld]);
        g.D.p[dro + (long long)vcol(g.D, j) * g.D.ld] = v;
    }
}

// problems a workspace of cap bytes takes at a time, 0 for a batch the engine does not take: all of them, or
// an even number, so that the neighbours that share an A stay together, or one
static int crt_part(const GemmBatch& b, size_t cap) {
    if (b.count == 0 || b.max_m == 0 || b.max_n == 0 || b.max_k == 0 || b.max_k > CRT_MAX_K) return 0;
    GemmBatch c = b;
    c.count = 1;
    const CrtGeom g = crt_geom(c);
    // the split and combine grids take one block per slab and per column group, the product's y a problem
    const long long slabs = (long long)g.KB * (g.MT * (CRT_BM / 16) + g.NT * (CRT_BN / 16));
    if (slabs > INT_MAX || (long long)g.MT * g.NT * (CRT_BN / 8) > INT_MAX) return 0;
    const long long fit = std::min<long long>((long long)cap / g.total, std::min<long long>(INT_MAX / slabs, 65535));
    if (fit >= b.count) return b.count;
    return fit >= 2 ? (int)(fit / 2 * 2) : (int)fit;
}
size_t crt_bytes(const GemmBatch& b, size_t cap) {
    GemmBatch c = b;
    c.count = 1;
    if (crt_part(c, SIZE_MAX / 2) == 0) return 0;
    c.count = std::max(1, crt_part(b, cap));
    return (size_t)crt_geom(c).total;
}

// a sub-batch whose planes and residues fit the workspace
static cudaError_t launch_crt_part(const GemmBatch& b, int* status, cudaStream_t s) {
    const CrtGeom cg = crt_geom(b);
    unsigned char* ws = static_cast<unsigned char*>(b.crt_ws);
    int* ea = reinterpret_cast<int*>(ws + cg.ea_off);
    int* fb = reinterpret_cast<int*>(ws + cg.fb_off);
    const long long nA = (long long)b.count * cg.MT * cg.KB * (CRT_BM / 16), nB = (long long)b.count * cg.NT * cg.KB * (CRT_BN / 16);
    const long long tiles = (long long)cg.MT * cg.NT;
    cudaError_t e = launch_operand_scales(b, cg.MT * CRT_BM, cg.NT * CRT_BN, ea, fb, s);
    if (e != cudaSuccess) return e;
    crt_split_kernel<<<(unsigned)(nA + nB), 256, 0, s>>>(b.d_desc, cg.MT, cg.NT, cg.KB, nA, ws, cg.a_bytes, ea, fb);
    note_launch();
    // runs of up to 8 row tiles per CTA (a resident B tile serves them all), and groups of moduli until there
    // are about six CTAs per SM to even the last wave out
    const int R = std::min(cg.MT, 8), runs = (cg.MT + R - 1) / R;
    int groups = 1;
    while (groups < CRT_S && (long long)runs * cg.NT * b.count * groups < 6 * 148) groups *= 2;
    zgemm_crt_kernel<<<dim3((unsigned)(runs * cg.NT), b.count, groups), CRT_THREADS, CRT_SMEM, s>>>(
        b.d_desc, status, ws, cg.MT, cg.NT, cg.KB, cg.a_bytes, ws + cg.c_off, R, CRT_S / groups);
    note_launch();
    crt_combine_kernel<<<dim3((unsigned)(tiles * (CRT_BN / 8)), b.count), 256, 0, s>>>(b.d_desc, cg.MT, cg.NT, ws + cg.c_off, ea,
                                                                                      fb);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_gemm_crt(const GemmBatch& b, int* status, cudaStream_t s) {
    if (b.count == 0 || b.max_m == 0 || b.max_n == 0) return cudaSuccess;
    // as many problems at a time as the workspace holds; an element's result does not depend on it
    const int part = crt_part(b, b.crt_cap);
    if (part == 0 || !status || !b.crt_ws || (reinterpret_cast<uintptr_t>(b.crt_ws) & 255)) return cudaErrorInvalidValue;
    static DeviceAttrCache attr;
    cudaError_t e = ensure_smem_attr(zgemm_crt_kernel, CRT_SMEM, attr, true);
    if (e != cudaSuccess) return e;
    GemmBatch c = b;
    for (int off = 0; off < b.count; off += part) {
        c.count = std::min(part, b.count - off);
        c.d_desc = b.d_desc + off;
        if ((e = launch_crt_part(c, status, s)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace rb
