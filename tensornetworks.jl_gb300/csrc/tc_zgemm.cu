// FP64 complex GEMM on the tensor cores: the Chinese remainder theorem over
// sixteen small moduli (the modular form of Ozaki's error-free splitting:
// K. Ozaki, Y. Uchino, T. Imamura, "Ozaki Scheme II", arXiv:2504.08009).
//
// GB300 issues FP64 at two FMAs per clock per SM (1.1 TFLOP/s measured), its
// tensor cores multiply BF16 at 1,934 TFLOP/s measured, and a BF16 product of
// integers below 128 accumulates in FP32 without rounding while the sum stays
// within 2^24.  Measured against the FP64 SIMT tile kernel: 256 x 256 x 256
// 1,031 -> 31 us, 1024 x 1280 x 512 6.1 ms -> 0.13 ms, and 5120 x 4096 x 1024 at
// 68 TFLOP/s of FP64 work; relative error 5e-17 against 5e-16 at K = 97 and
// 600 of normal entries.  The steps:
//
//   1. every row of op(A) and column of op(B) gets its own power-of-two scale
//      and becomes integers of T <= 57 bits relative to its largest entry
//      (FP64 holds 53 relative to each entry).  The result is good to
//      4 K max_k|a_ik| max_k|b_kj| 2^-T in either part: where large entries of one side meet small
//      ones of the other all along K, that is more than FP64's
//      K 2^-53 sum_k |a_ik||b_kj|.  A caller that knows the operands' grading along K
//      gives it as kexp: op(A) then counts as op(A) D and op(B) as D^-1 op(B), D = 2^kexp,
//      in that bound;
//   2. the integers are reduced modulo p_0 .. p_15 <= 251 (pairwise coprime,
//      product P = 2^124.9) into BF16 planes, real and imaginary;
//   3. per modulus, tcgen05 forms the four real products of the complex
//      product exactly: |sum| <= 2 * 512 * 127^2 < 2^24 for 512-element K
//      chunks, each chunk reduced modulo p in the epilogue;
//   4. the residues determine the integer product (2 K 2^2T < P / 2): its
//      fraction of P is sum_i r_i inv_i / p_i modulo 1, evaluated in 96-bit
//      fixed point, scaled back and rounded once to FP64.
//
// Rows or columns that hold an infinity or NaN, or nothing but denormals, have
// no scale: outputs they meet are recomputed by the plain FP64 dot product, as
// the SIMT kernels give them.
//
// Four real products instead of three (Karatsuba is free modulo p): with four,
// each operand plane in shared memory feeds two products, so a 128 x 128 tile
// needs half the L2 traffic per flop, and conversion writes two planes per
// modulus instead of three.
#include <climits>

#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include "common.cuh"

namespace tn {

namespace {

constexpr int NP = 16;                        // moduli
constexpr int BM = 128, BN = 128, BK = 64;    // CTA tile, K elements per stage
constexpr int STAGES = 3;
constexpr int KCHUNK = 512;                   // exact FP32 accumulation length
constexpr int KT_CHUNK = KCHUNK / BK;
constexpr int TILE_BYTES = BM * BK * 2;       // 16 KB, BM == BN
constexpr int STAGE_BYTES = 4 * TILE_BYTES;   // A re, A im, B re, B im
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
constexpr int EPI_T = 256;                    // epilogue threads
constexpr int GEMM_T = 64 + EPI_T;
constexpr uint32_t TMEM_COLS = 512;           // two accumulator pairs (re, im)
constexpr uint64_t WAIT_NS = 2000000000ull;   // 2 s bound on any wait

typedef unsigned __int128 u128;

constexpr int MODULI[NP] = {251, 250, 249, 247, 241, 239, 233, 229,
                            227, 223, 217, 211, 199, 197, 193, 191};

struct Tables {
    float p[NP], rp[NP];
    float c1[NP], c2[NP], c3[NP];  // 2^15, 2^30, 2^45 modulo p, symmetric
    uint32_t w0[NP], w1[NP], w2[NP];  // (inv_i / p_i) 2^96 modulo 2^96
    uint32_t o0, o1, o2;              // 128 sum_i W_i modulo 2^96
    uint64_t p64;                     // P = p64 2^pexp, p64 in [2^63, 2^64)
    int pexp;
};

constexpr int symmod(u128 v, int p) {
    int r = (int)(v % (u128)p);
    return r > p / 2 ? r - p : r;
}

constexpr Tables make_tables() {
    Tables t{};
    u128 P = 1;
    for (int i = 0; i < NP; ++i) P *= (u128)MODULI[i];
    u128 off = 0;
    const u128 mask96 = (((u128)1) << 96) - 1;
    for (int i = 0; i < NP; ++i) {
        const int p = MODULI[i];
        t.p[i] = (float)p;
        t.rp[i] = 1.0f / (float)p;
        t.c1[i] = (float)symmod((u128)1 << 15, p);
        t.c2[i] = (float)symmod((u128)1 << 30, p);
        t.c3[i] = (float)symmod((u128)1 << 45, p);
        const int m = (int)((P / (u128)p) % (u128)p);
        int inv = 1;
        while ((m * inv) % p != 1) ++inv;
        const u128 num = ((u128)inv) << 96;
        const u128 w = ((num + (u128)(p / 2)) / (u128)p) & mask96;
        t.w0[i] = (uint32_t)w;
        t.w1[i] = (uint32_t)(w >> 32);
        t.w2[i] = (uint32_t)(w >> 64);
        off = (off + 128 * w) & mask96;
    }
    t.o0 = (uint32_t)off;
    t.o1 = (uint32_t)(off >> 32);
    t.o2 = (uint32_t)(off >> 64);
    int e = 0;
    u128 q = P;
    while (q >= (((u128)1) << 64)) {
        q >>= 1;
        ++e;
    }
    t.p64 = (uint64_t)q;
    t.pexp = e;
    return t;
}

constexpr Tables HT = make_tables();
__constant__ Tables KT = make_tables();

// ---- operands ----------------------------------------------------------------
// One operand as rows x K: entry (r, k) at src[k + ld r] when kmajor, else at
// src[r + ld k]; conj negates the imaginary part.
struct Side {
    const cplx* src;
    int64_t rows, K, ld;
    int kmajor, conj;
    unsigned* hmax;          // rows: largest high word of |re|, |im|
    const int* kexp;         // K: entry (r, k) counts as itself 2^(ksign kexp[k]); null: as itself
    int ksign;
    int* ex;                 // rows: largest biased exponent with that, when kexp
    __nv_bfloat16* planes;   // [NP][re, im][rows][ldp]
    int64_t ldp;
    int blocks_max, blocks_cvt;  // grid shares of the two kernels
};

// the high word of |x|, at least 1 unless x is zero
__device__ __forceinline__ unsigned hi_abs(double x) {
    return ((unsigned)__double2hiint(x) & 0x7fffffffu) | (__double2loint(x) != 0 ? 1u : 0u);
}
// a row without a scale of its own: infinities, NaN, or nothing but denormals
__device__ __forceinline__ bool unscaled(unsigned h) {
    return h >= 0x7ff00000u || (h != 0 && h < 0x00100000u);
}

// biased exponent of the larger part of an entry whose high word of both is h
__device__ __forceinline__ int exponent(unsigned h, int shift) {
    return h ? max((int)(h >> 20), 1) + shift : INT_MIN;
}
template <bool GRADED>  // with kexp
__device__ __forceinline__ int row_exponent(const Side& s, int64_t r) {
    if (GRADED) return s.ex[r] < -100000 ? 1 : s.ex[r];  // a row of zeros: any
    return max(1, min((int)(s.hmax[r] >> 20), 0x7fe));
}

constexpr int SEG = 512;    // K per block of the row-maximum kernel
constexpr int MAX_T = 512;  // its threads

// Largest high word of every row's entries.  Integer maxima, so the order of
// the atomics that merge several segments does not matter (hmax then starts
// at zero); one segment stores directly.
template <bool GRADED>
__global__ void __launch_bounds__(MAX_T) zrow_max_kernel(Side a, Side b) {
    const bool first = (int)blockIdx.x < a.blocks_max;
    const Side& s = first ? a : b;
    const int blk = first ? blockIdx.x : blockIdx.x - a.blocks_max;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nseg = (int)((s.K + SEG - 1) / SEG);
    const int64_t k0 = (int64_t)(blk % nseg) * SEG, k1 = min(s.K, k0 + SEG);
    if (s.kmajor) {  // a row per warp
        const int64_t r = (int64_t)(blk / nseg) * (MAX_T / 32) + warp;
        if (r >= s.rows) return;
        unsigned m = 0;
        int e = INT_MIN;
#pragma unroll 4
        for (int64_t k = k0 + lane; k < k1; k += 32) {
            const cplx v = s.src[k + s.ld * r];
            const unsigned h = max(hi_abs(v.x), hi_abs(v.y));
            m = max(m, h);
            if (GRADED) e = max(e, exponent(h, s.ksign * s.kexp[k]));
        }
        m = __reduce_max_sync(0xffffffffu, m);
        if (GRADED) e = __reduce_max_sync(0xffffffffu, e);
        if (lane == 0) {
            if (nseg > 1) atomicMax(s.hmax + r, m);
            else s.hmax[r] = m;
            if (GRADED) {
                if (nseg > 1) atomicMax(s.ex + r, e);
                else s.ex[r] = e;
            }
        }
    } else {  // 32 rows per block, a lane each; the warps share the segment
        __shared__ unsigned sm[MAX_T / 32][32];
        __shared__ int se[GRADED ? MAX_T / 32 : 1][32];
        const int64_t r = (int64_t)(blk / nseg) * 32 + lane;
        unsigned m = 0;
        int e = INT_MIN;
        if (r < s.rows)
#pragma unroll 8
            for (int64_t k = k0 + warp; k < k1; k += MAX_T / 32) {
                const cplx v = s.src[r + s.ld * k];
                const unsigned h = max(hi_abs(v.x), hi_abs(v.y));
                m = max(m, h);
                if (GRADED) e = max(e, exponent(h, s.ksign * s.kexp[k]));
            }
        sm[warp][lane] = m;
        if (GRADED) se[warp][lane] = e;
        __syncthreads();
        if (warp == 0 && r < s.rows) {
#pragma unroll
            for (int w = 1; w < MAX_T / 32; ++w) {
                m = max(m, sm[w][lane]);
                if (GRADED) e = max(e, se[w][lane]);
            }
            if (nseg > 1) atomicMax(s.hmax + r, m);
            else s.hmax[r] = m;
            if (GRADED) {
                if (nseg > 1) atomicMax(s.ex + r, e);
                else s.ex[r] = e;
            }
        }
    }
}

// x 2^(T - 1 - e) rounded to an integer, |x| < 2^(e+1) with e the row's exponent less
// what the entry's K index adds
__device__ __forceinline__ int64_t to_int(double x, int E, int T) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    int e = (int)((b >> 52) & 0x7ff);
    uint64_t m = b & 0xfffffffffffffull;
    if (e) m |= 0x10000000000000ull;
    else e = 1;
    const int sh = e - E + T - 53;
    if (sh >= 0) m <<= sh;  // sh <= T - 53 <= 4
    else if (sh < -54) m = 0;
    else m = (m + (1ull << (-sh - 1))) >> -sh;
    return (int64_t)b < 0 ? -(int64_t)m : (int64_t)m;
}

struct Limbs {
    float x0, x1, x2, x3;
    __device__ __forceinline__ Limbs(int64_t x) {
        x0 = (float)(int)(x & 0x7fff);
        x1 = (float)(int)((x >> 15) & 0x7fff);
        x2 = (float)(int)((x >> 30) & 0x7fff);
        x3 = (float)(int)(x >> 45);
    }
};

// v - p rint(v / p) for an integer |v| <= 2^24: FP32 throughout, exact (the
// quotient may be off by one near a half, which the bound 127 allows)
__device__ __forceinline__ float mod_p(float v, float p, float rp) {
    const float magic = 12582912.0f;  // 1.5 * 2^23
    const float q = __fsub_rn(__fmaf_rn(v, rp, magic), magic);
    return __fmaf_rn(-q, p, v);
}

// Residues of four consecutive K entries of one row, eight bytes per plane;
// parts [lo, hi) of (real, imaginary).
__device__ __forceinline__ void convert4(const cplx* v, int lo, int hi, const int* E, int T, int conj,
                                         __nv_bfloat16* __restrict__ dst, size_t plane) {
#pragma unroll 1
    for (int part = lo; part < hi; ++part) {
        Limbs l[4] = {Limbs(0), Limbs(0), Limbs(0), Limbs(0)};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double x = part ? (conj ? -v[i].y : v[i].y) : v[i].x;
            l[i] = Limbs(to_int(x, E[i], T));
        }
        __nv_bfloat16* d = dst + part * plane;
#pragma unroll
        for (int m = 0; m < NP; ++m) {
            float r[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                r[i] = mod_p(__fmaf_rn(l[i].x3, KT.c3[m],
                                       __fmaf_rn(l[i].x2, KT.c2[m], __fmaf_rn(l[i].x1, KT.c1[m], l[i].x0))),
                             KT.p[m], KT.rp[m]);
            __nv_bfloat162 a = __floats2bfloat162_rn(r[0], r[1]), c = __floats2bfloat162_rn(r[2], r[3]);
            uint2 w;
            w.x = *reinterpret_cast<unsigned*>(&a);
            w.y = *reinterpret_cast<unsigned*>(&c);
            *reinterpret_cast<uint2*>(d + (size_t)(2 * m) * plane) = w;
        }
    }
}

// the row's exponent for K entries k .. k + 3
template <bool GRADED>
__device__ __forceinline__ void exponents(const Side& s, int64_t r, int64_t k, int* E) {
    const int e = row_exponent<GRADED>(s, r);
#pragma unroll
    for (int i = 0; i < 4; ++i) E[i] = GRADED && k + i < s.K ? e - s.ksign * s.kexp[k + i] : e;
}

// Residue planes.  A half-warp converts 64 consecutive K entries of a row, so
// that every plane gets 128-byte stores; operands whose rows are contiguous
// pass through a shared-memory tile of 32 rows x 64 K.
template <bool GRADED>
__global__ void __launch_bounds__(256, 2) zconvert_kernel(Side a, Side b, int T) {
    __shared__ cplx tile[32][65];  // row r, K entry k at (k & 3) * 16 + k / 4: no bank conflicts
    const bool first = (int)blockIdx.x < a.blocks_cvt;
    const Side& s = first ? a : b;
    const int blk = first ? blockIdx.x : blockIdx.x - a.blocks_cvt;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int hl = threadIdx.x & 15, half = threadIdx.x >> 4;
    // two grid rows take a part each where one row would leave SMs idle
    const int lo = gridDim.y == 2 ? blockIdx.y : 0, hi = gridDim.y == 2 ? lo + 1 : 2;
    const int nk = (int)((s.ldp + 63) / 64);
    const size_t plane = (size_t)s.rows * s.ldp;
    if (s.kmajor) {  // sixteen rows x 64 K per block
        const int64_t r = (int64_t)(blk / nk) * 16 + half;
        const int64_t k = (int64_t)(blk % nk) * 64 + 4 * hl;
        if (r >= s.rows || k >= s.ldp) return;
        int E[4];
        exponents<GRADED>(s, r, k, E);
        cplx v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = k + i < s.K ? s.src[k + i + s.ld * r] : cmk(0, 0);
        convert4(v, lo, hi, E, T, s.conj, s.planes + (size_t)r * s.ldp + k, plane);
    } else {
        const int64_t r0 = (int64_t)(blk / nk) * 32, k0 = (int64_t)(blk % nk) * 64;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int64_t k = k0 + warp + 8 * j, r = r0 + lane;
            const int kl = warp + 8 * j;
            tile[lane][(kl & 3) * 16 + (kl >> 2)] =
                (k < s.K && r < s.rows) ? s.src[r + s.ld * k] : cmk(0, 0);
        }
        __syncthreads();
        const int64_t k = k0 + 4 * hl;
        if (k >= s.ldp) return;
        for (int rl = half; rl < 32; rl += 16) {
            const int64_t r = r0 + rl;
            if (r >= s.rows) continue;
            int E[4];
            exponents<GRADED>(s, r, k, E);
            cplx v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = tile[rl][16 * i + hl];
            convert4(v, lo, hi, E, T, s.conj, s.planes + (size_t)r * s.ldp + k, plane);
        }
    }
}

// ---- the modular products ------------------------------------------------------
struct Params {
    int64_t M, N;
    int ktiles;            // BK slices of K
    int mt, nt, tiles;     // tile grid; tiles per modulus (lower: the triangle)
    int lower;
    uchar2* q;             // [NP][N][ldq] residues + 128
    int64_t ldq;
    int* err;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint64_t gtimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait: false when the limit runs out or another role gave up
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* abort_flag) {
    if (mbar_try(bar, parity)) return true;
    const uint64_t t0 = gtimer();
    while (!mbar_try(bar, parity)) {
        if (*(volatile int*)abort_flag) return false;
        if (gtimer() - t0 > WAIT_NS) {
            atomicExch(abort_flag, 1);
            return false;
        }
    }
    return true;
}
// the same, whatever the other roles did
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity) {
    const uint64_t t0 = gtimer();
    while (!mbar_try(bar, parity))
        if (gtimer() - t0 > WAIT_NS) return;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar,
                                            int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                       uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

// K-major operand tile of 128-byte rows, 128-byte swizzle (tc_gemm.cu's layout)
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// kind::f16: D fp32 (bits 4-5 = 1), A and B bf16 (bits 7-9, 10-12 = 1),
// bit 13 negates A
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n, bool negA) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (negA ? (1u << 13) : 0u) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

#define TN_TMEM_LD32(taddr, r)                                                                   \
    asm volatile(                                                                                \
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "  \
        "%11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, "   \
        "%28, %29, %30, %31}, [%32];"                                                            \
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),    \
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),             \
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),          \
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),          \
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),          \
          "=r"(r[31])                                                                            \
        : "r"(taddr))

struct Item {
    int mod, m0, n0;
};
// item order: modulus by modulus, so that one modulus' planes stay in L2 while
// its tiles run; lower: tiles (i, j) with j <= i of a square grid
__device__ __forceinline__ Item item_of(const Params& p, int it) {
    Item r;
    r.mod = it / p.tiles;
    const int t = it - r.mod * p.tiles;
    int i, j;
    if (p.lower) {
        i = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
        while ((i + 1) * (i + 2) / 2 <= t) ++i;
        while (i * (i + 1) / 2 > t) --i;
        j = t - i * (i + 1) / 2;
    } else {
        i = t % p.mt;
        j = t / p.mt;
    }
    r.m0 = i * BM;
    r.n0 = j * BN;
    return r;
}

// Persistent: CTA b takes items b, b + gridDim.x, ...; an item is one tile of
// one modulus.  Warp 0 loads by TMA, one lane of warp 1 issues the MMAs, warps
// 2-9 reduce the accumulators modulo p; two accumulator pairs in TMEM let the
// next chunk's MMAs run under the epilogue.  A 512-element chunk is 4.3 us of
// MMAs at the dense rate of one SM; with four epilogue warps its modular
// reduction took 14 us and the tensor pipe was 30 % busy (1.52 ms at 4096 x 2048
// x 1024), with eight, each residue of the chunks before loaded ahead of the
// accumulator, 59 % (0.77 ms).
__global__ void __launch_bounds__(GEMM_T, 1)
    zmod_gemm_kernel(const __grid_constant__ CUtensorMap mapA,
                     const __grid_constant__ CUtensorMap mapB, Params p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
    uint64_t* empty = full + STAGES;
    uint64_t* accf = empty + STAGES;
    uint64_t* acce = accf + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acce + 2);
    int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int items = NP * p.tiles;
    const int nch = (p.ktiles + KT_CHUNK - 1) / KT_CHUNK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&accf[s], 1);
            mbar_init(&acce[s], EPI_T);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mapA)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mapB)) : "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int n = 0;  // stages filled so far
            bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                const Item w = item_of(p, it);
                for (int kt = 0; kt < p.ktiles; ++kt) {
                    const int s = n % STAGES;
                    if (!mbar_wait(&empty[s], ((uint32_t)(n / STAGES) & 1u) ^ 1u, abort_flag)) {
                        ok = false;
                        break;
                    }
                    uint8_t* st = smem + s * STAGE_BYTES;
                    mbar_expect_tx(&full[s], STAGE_BYTES);
                    const int x = kt * BK;  // BK bf16 = 128 bytes: 16-byte aligned
                    tma_load_3d(st + 0 * TILE_BYTES, &mapA, &full[s], x, w.m0, 2 * w.mod + 0);
                    tma_load_3d(st + 1 * TILE_BYTES, &mapA, &full[s], x, w.m0, 2 * w.mod + 1);
                    tma_load_3d(st + 2 * TILE_BYTES, &mapB, &full[s], x, w.n0, 2 * w.mod + 0);
                    tma_load_3d(st + 3 * TILE_BYTES, &mapB, &full[s], x, w.n0, 2 * w.mod + 1);
                    ++n;
                }
            }
            // copies still in flight land before the CTA can retire
            for (int i = (n > STAGES ? n - STAGES : 0); i < n; ++i)
                mbar_drain(&full[i % STAGES], (uint32_t)(i / STAGES) & 1u);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t id_pos = idesc_bf16(BM, BN, false);
            const uint32_t id_neg = idesc_bf16(BM, BN, true);
            int n = 0, c = 0;  // stages consumed, chunks started
            bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                for (int kt = 0; kt < p.ktiles; ++kt) {
                    const bool start = kt % KT_CHUNK == 0;
                    if (start) {
                        if (!mbar_wait(&acce[c & 1], ((uint32_t)(c >> 1) & 1u) ^ 1u, abort_flag)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                    }
                    const int s = n % STAGES;
                    if (!mbar_wait(&full[s], (uint32_t)(n / STAGES) & 1u, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t base = smem_u32(smem + s * STAGE_BYTES);
                    const uint64_t dAr = sw128_desc(base + 0 * TILE_BYTES);
                    const uint64_t dAi = sw128_desc(base + 1 * TILE_BYTES);
                    const uint64_t dBr = sw128_desc(base + 2 * TILE_BYTES);
                    const uint64_t dBi = sw128_desc(base + 3 * TILE_BYTES);
                    const uint32_t dr = tmem + 256u * (uint32_t)(c & 1), di = dr + 128u;
#pragma unroll
                    for (int j = 0; j < BK / 16; ++j) {
                        const uint64_t o = (uint64_t)(j * 32) >> 4;  // 16 bf16 = 32 bytes along K
                        const uint32_t acc = (start && j == 0) ? 0u : 1u;
                        tc_mma(dr, dAr + o, dBr + o, id_pos, acc);
                        tc_mma(di, dAr + o, dBi + o, id_pos, acc);
                        tc_mma(dr, dAi + o, dBi + o, id_neg, 1u);
                        tc_mma(di, dAi + o, dBr + o, id_pos, 1u);
                    }
                    tc_commit(&empty[s]);
                    ++n;
                    if (kt % KT_CHUNK == KT_CHUNK - 1 || kt == p.ktiles - 1) {
                        tc_commit(&accf[c & 1]);
                        ++c;
                    }
                }
            }
            // after an abort products in flight end before their TMEM goes back
            if (!ok && n > 0) mbar_drain(&empty[(n - 1) % STAGES], (uint32_t)((n - 1) / STAGES) & 1u);
        }
    } else {
        // two warps per TMEM lane quarter, 64 columns each
        const int q = warp & 3, h = (warp - 2) >> 2;
        int c = 0;
        bool ok = true;
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            const Item w = item_of(p, it);
            const float pm = KT.p[w.mod], rp = KT.rp[w.mod];
            const int64_t m = w.m0 + 32 * q + lane, nb = w.n0 + 64 * h;
            const int ncol = (int)min((int64_t)64, p.N - nb);
            uchar2* out = p.q + ((int64_t)w.mod * p.N + nb) * p.ldq + m;
            for (int ch = 0; ch < nch; ++ch, ++c) {
                // a warp leaves or goes on as a whole: the loads below are the warp's
                if (!__all_sync(0xffffffffu, mbar_wait(&accf[c & 1], (uint32_t)(c >> 1) & 1u, abort_flag))) {
                    atomicExch(abort_flag, 1);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t ta =
                    tmem + ((uint32_t)(32 * q) << 16) + 256u * (uint32_t)(c & 1) + 64u * (uint32_t)h;
#pragma unroll 1
                for (int c0 = 0; c0 < 64; c0 += 32) {
                    uint32_t a[32], b[32];
                    unsigned short prev[32];
                    const int nc = m < p.M ? ncol - c0 : 0;
                    uchar2* o = out + (int64_t)c0 * p.ldq;
                    if (ch > 0) {  // this thread's residues of the chunks before
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (j < nc)
                                prev[j] = *reinterpret_cast<unsigned short*>(o + (int64_t)j * p.ldq);
                    }
                    __syncwarp();
                    TN_TMEM_LD32(ta + c0, a);
                    TN_TMEM_LD32(ta + 128 + c0, b);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        float r = mod_p(__uint_as_float(a[j]), pm, rp);
                        float s = mod_p(__uint_as_float(b[j]), pm, rp);
                        if (ch > 0) {  // stored biased by 128
                            r = mod_p(r + (float)((int)(prev[j] & 0xff) - 128), pm, rp);
                            s = mod_p(s + (float)((int)(prev[j] >> 8) - 128), pm, rp);
                        }
                        // the byte r + 128 in the low bits of 1.5 2^23 + r + 128
                        const uint32_t x = __float_as_uint(r + 12583040.0f);
                        const uint32_t y = __float_as_uint(s + 12583040.0f);
                        if (j < nc)
                            *reinterpret_cast<unsigned short*>(o + (int64_t)j * p.ldq) =
                                (unsigned short)__byte_perm(x, y, 0x0040);
                    }
                }
                tc_fence_before();
                mbar_arrive(&acce[c & 1]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(TMEM_COLS));
    }
    if (threadIdx.x == 0 && *(volatile int*)abort_flag) *(volatile int*)p.err = 1;  // host memory
}

// ---- reconstruction --------------------------------------------------------------
// mag / 2^96 P 2^sc rounded to FP64, mag = the 96-bit magnitude (h, l)
__device__ __forceinline__ double fixed_to_double(uint64_t h, uint32_t l, bool neg, int sc) {
    int lz;
    uint64_t m;
    if (h) {
        lz = __clzll(h);
        m = lz ? (h << lz) | ((((uint64_t)l) << 32) >> (64 - lz)) : h;
    } else if (l) {
        lz = 64 + __clz(l);
        m = (uint64_t)l << (lz - 32);
    } else {
        return 0.0;
    }
    m = __umul64hi(m, KT.p64);  // value: m 2^(64 + 32 - lz + pexp - 96)
    int e = KT.pexp - lz + sc;  // value: m 2^e
    const int s = __clzll(m);   // 0 or 1
    m <<= s;
    e += 63 - s;
    uint64_t mant = m >> 11;
    const uint32_t rem = (uint32_t)m & 0x7ffu;
    mant += (rem > 0x400u) || (rem == 0x400u && (mant & 1));
    const int be = e + 1023;
    double v;
    if (be > 0 && be < 2046)
        v = __longlong_as_double((long long)(((uint64_t)(be - 1) << 52) + mant));
    else  // overflow or gradual underflow
        v = scalbn((double)mant, e - 52);
    return neg ? -v : v;
}

struct Out {
    int64_t M, N, ldc, ldq;
    cplx alpha, beta;
    cplx* C;
    const uchar2* q;
    int lower, T, plain;  // plain: alpha = 1, beta = 0
};

// plain FP64 dot product of one output, for rows or columns without a scale
__device__ __noinline__ cplx dot64(const Side& a, const Side& b, int64_t m, int64_t n) {
    cplx acc = cmk(0, 0);
    for (int64_t k = 0; k < a.K; ++k) {
        cplx x = a.kmajor ? a.src[k + a.ld * m] : a.src[m + a.ld * k];
        cplx y = b.kmajor ? b.src[k + b.ld * n] : b.src[n + b.ld * k];
        if (a.conj) x.y = -x.y;
        if (b.conj) y.y = -y.y;
        acc = cfma(x, y, acc);
    }
    return acc;
}

constexpr int CRT_T = 128;

// C = alpha X + beta C from the residues, four consecutive rows per thread.
// All-integer up to the last scaling: sixteen 32 x 8 bit products per word
// where FP64 would wait on its two lanes per clock.
template <bool GRADED>
__global__ void __launch_bounds__(CRT_T) zcrt_kernel(Out o, Side a, Side b) {
    const int64_t mq = (o.M + 3) / 4, total = mq * o.N;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n = e / mq, m0 = 4 * (e - n * mq);
        if (o.lower && m0 + 3 < n) continue;
        uint64_t acc[8][3];
#pragma unroll
        for (int u = 0; u < 8; ++u) acc[u][0] = acc[u][1] = acc[u][2] = 0;
        const uchar2* q = o.q + n * o.ldq + m0;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            const uint2 w = __ldcs(reinterpret_cast<const uint2*>(q + (int64_t)i * o.N * o.ldq));
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const uint32_t r = ((u < 4 ? w.x : w.y) >> (8 * (u & 3))) & 0xffu;
                acc[u][0] += (uint64_t)r * KT.w0[i];
                acc[u][1] += (uint64_t)r * KT.w1[i];
                acc[u][2] += (uint64_t)r * KT.w2[i];
            }
        }
        const unsigned hb = b.hmax[n];
        const int eb = row_exponent<GRADED>(b, n);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int64_t m = m0 + v;
            if (m >= o.M || (o.lower && m < n)) continue;
            const unsigned ha = a.hmax[m];
            const int ea = row_exponent<GRADED>(a, m);
            const int sc = ea + eb - 2044 - 2 * o.T;
            double x[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint64_t* A = acc[2 * v + u];
                // 96-bit sum of the words, minus the offset 128 sum W
                const uint64_t t0 = (A[0] & 0xffffffffull) + (0x100000000ull - KT.o0);
                const uint64_t t1 = (A[0] >> 32) + A[1] + (0xffffffffull - KT.o1) + (t0 >> 32);
                const uint64_t t2 = (t1 >> 32) + A[2] + (0xffffffffull - KT.o2);
                uint32_t l = (uint32_t)t0;
                uint64_t h = (uint64_t)(uint32_t)t1 | (t2 << 32);
                const bool neg = (int64_t)h < 0;
                if (neg) {  // two's complement magnitude
                    l = ~l + 1u;
                    h = ~h + (l == 0u);
                }
                x[u] = fixed_to_double(h, l, neg, sc);
            }
            cplx r = cmk(x[0], x[1]);
            if (unscaled(ha) || unscaled(hb)) r = dot64(a, b, m, n);
            cplx* c = o.C + m + n * o.ldc;
            if (!o.plain) {
                r = cmul(o.alpha, r);
                if (o.beta.x != 0.0 || o.beta.y != 0.0) r = cfma(o.beta, *c, r);
            }
            *c = r;
        }
    }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        cudaDriverEntryPointQueryResult q;
        void* f = nullptr;
        TN_CHECK_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000,
                                                       cudaEnableDefault, &q));
        TN_REQUIRE(q == cudaDriverEntryPointSuccess && f, "cuTensorMapEncodeTiled unavailable");
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    }();
    return fn;
}

void make_map(const Side& s, CUtensorMap* map) {
    cuuint64_t dims[3] = {(cuuint64_t)s.K, (cuuint64_t)s.rows, 2 * NP};
    cuuint64_t strides[2] = {(cuuint64_t)s.ldp * 2, (cuuint64_t)(s.rows * s.ldp) * 2};
    cuuint32_t box[3] = {BK, BM, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r =
        encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, s.planes, dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        throw Error(TN_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
}

void grids(Side& s) {
    const int64_t nk = (s.ldp + 63) / 64, nseg = (s.K + SEG - 1) / SEG;
    s.blocks_max = (int)((s.kmajor ? (s.rows + MAX_T / 32 - 1) / (MAX_T / 32) : (s.rows + 31) / 32) * nseg);
    s.blocks_cvt = (int)((s.kmajor ? (s.rows + 15) / 16 : (s.rows + 31) / 32) * nk);
}

}  // namespace

bool zgemm_tc(Ctx* ctx, Op opa, Op opb, int64_t m, int64_t n, int64_t k, cplx alpha, const cplx* A,
              int64_t lda, const cplx* B, int64_t ldb, cplx beta, cplx* C, int64_t ldc,
              bool lower_only, const int* kexp, int ksign) {
    if (m > (1 << 24) || n > (1 << 24) || k > (1 << 16)) return false;
    const int64_t ldp = (k + 7) / 8 * 8, ldq = (m + 3) / 4 * 4;
    auto r256 = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t bA = r256(sizeof(__nv_bfloat16) * 2 * NP * (size_t)m * ldp);
    const size_t bB = r256(sizeof(__nv_bfloat16) * 2 * NP * (size_t)n * ldp);
    const size_t bQ = r256(sizeof(uchar2) * NP * (size_t)n * ldq);
    const size_t bH = r256(2 * sizeof(unsigned) * (size_t)(m + n));
    char* base;
    try {
        base = static_cast<char*>(ctx->s_tcz.get(ctx, bA + bB + bQ + bH));
    } catch (const Error& e) {
        if (e.code != TN_ERR_OOM) throw;
        // the FP64 kernels need no planes; up to thirty times slower, so it is said once
        if (!ctx->told_oom)
            fprintf(stderr, "tngpu: no room for %zu MB of residue planes, product of %lld x %lld x %lld on the FP64 units\n",
                    (bA + bB + bQ + bH) >> 20, (long long)m, (long long)n, (long long)k);
        ctx->told_oom = true;
        return false;
    }
    unsigned* hmax = reinterpret_cast<unsigned*>(base + bA + bB + bQ);
    Side a{A, m, k, lda, (opa == OP_T || opa == OP_C) ? 1 : 0, (opa == OP_C || opa == OP_R) ? 1 : 0,
           hmax, kexp, ksign, reinterpret_cast<int*>(hmax + m + n), reinterpret_cast<__nv_bfloat16*>(base), ldp, 0, 0};
    Side b{B, n, k, ldb, (opb == OP_N || opb == OP_R) ? 1 : 0, (opb == OP_C || opb == OP_R) ? 1 : 0,
           hmax + m, kexp, -ksign, a.ex + m, reinterpret_cast<__nv_bfloat16*>(base + bA), ldp, 0, 0};
    grids(a);
    grids(b);
    // 2 k 2^2T <= P / 2 with P > 2^124
    int lk = 0;
    while (((int64_t)1 << lk) < k) ++lk;
    const int T = std::min(57, (124 - 2 - lk) / 2);
    if (k > SEG) {
        TN_CHECK_CUDA(cudaMemsetAsync(hmax, 0, sizeof(unsigned) * (size_t)(m + n), ctx->stream));
        if (kexp)  // below any exponent
            TN_CHECK_CUDA(cudaMemsetAsync(a.ex, 0x80, sizeof(int) * (size_t)(m + n), ctx->stream));
    }
    auto row_max = kexp ? zrow_max_kernel<true> : zrow_max_kernel<false>;
    row_max<<<a.blocks_max + b.blocks_max, MAX_T, 0, ctx->stream>>>(a, b);
    ctx->count();
    const int ncvt = a.blocks_cvt + b.blocks_cvt;
    auto convert = kexp ? zconvert_kernel<true> : zconvert_kernel<false>;
    convert<<<dim3(ncvt, ncvt < 2 * ctx->sm_count ? 2 : 1), 256, 0, ctx->stream>>>(a, b, T);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
    CUtensorMap ma, mb;
    make_map(a, &ma);
    make_map(b, &mb);
    Params p{};
    p.M = m;
    p.N = n;
    p.ktiles = (int)((k + BK - 1) / BK);
    p.mt = (int)((m + BM - 1) / BM);
    p.nt = (int)((n + BN - 1) / BN);
    p.lower = (lower_only && m == n) ? 1 : 0;
    p.tiles = p.lower ? p.mt * (p.mt + 1) / 2 : p.mt * p.nt;
    p.q = reinterpret_cast<uchar2*>(base + bA + bB);
    p.ldq = ldq;
    p.err = ctx->h_err;
    TN_CHECK_CUDA(cudaFuncSetAttribute(zmod_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       SMEM_BYTES));
    const int grid = std::min(NP * p.tiles, ctx->sm_count);
    zmod_gemm_kernel<<<grid, GEMM_T, SMEM_BYTES, ctx->stream>>>(ma, mb, p);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
    const bool plain = alpha.x == 1.0 && alpha.y == 0.0 && beta.x == 0.0 && beta.y == 0.0;
    Out o{m, n, ldc, ldq, alpha, beta, C, p.q, lower_only ? 1 : 0, T, plain ? 1 : 0};
    const int64_t blocks = ((m + 3) / 4 * n + CRT_T - 1) / CRT_T;
    auto crt = kexp ? zcrt_kernel<true> : zcrt_kernel<false>;
    crt<<<(unsigned)std::min<int64_t>(blocks, (int64_t)ctx->sm_count * 16), CRT_T, 0,
                  ctx->stream>>>(o, a, b);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
    return true;
}

}  // namespace tn
