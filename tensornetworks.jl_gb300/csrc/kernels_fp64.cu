// FP64 kernels of the plain (parity) path: complex GEMM, the small-operator
// contraction used for MPO/gate legs, Lanczos vector reductions (warp
// shuffles) and the truncation keep rule.
//
// GB300 executes FP64 on the SIMT pipes at a small fraction of its tensor
// rate.  Large products of the library's own paths therefore run on the
// tensor cores (tc_zgemm.cu, chosen by tc_sized).  Here are the small ones,
// one output per thread or group of lanes, and a 64x64 complex tile per
// 256-thread block with a 4x4 complex register tile per thread, which keeps
// the DFMA pipe busy: it serves products that a caller wants on FP64 units
// and those whose operand planes find no room.
#include "common.cuh"
#include "grid_dev.cuh"

namespace tn {

namespace {

constexpr int GB_M = 64, GB_N = 64, GB_K = 16;

template <int OPA, int OPB>
__global__ void __launch_bounds__(256) zgemm_kernel(int64_t M, int64_t N, int64_t K, cplx alpha,
                                                    const cplx* __restrict__ A, int64_t lda,
                                                    int64_t sA, const cplx* __restrict__ B,
                                                    int64_t ldb, int64_t sB, cplx beta,
                                                    cplx* __restrict__ C, int64_t ldc, int64_t sC,
                                                    int lower, int64_t kc) {
    __shared__ cplx As[GB_K][GB_M + 1];
    __shared__ cplx Bs[GB_K][GB_N + 1];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    // kc > 0: split K; blockIdx.z is the chunk and C the chunk's partial
    // (M x N, ld M); otherwise blockIdx.z is the batch index
    const int64_t bz = kc > 0 ? 0 : blockIdx.z;
    const int64_t k_lo = kc > 0 ? (int64_t)blockIdx.z * kc : 0;
    const int64_t k_hi = kc > 0 ? min(K, k_lo + kc) : K;
    A += bz * sA;
    B += bz * sB;
    C += kc > 0 ? (int64_t)blockIdx.z * M * N : bz * sC;
    const int64_t m0 = (int64_t)blockIdx.x * GB_M, n0 = (int64_t)blockIdx.y * GB_N;
    // lower: only the lower triangle is wanted (a Hermitian Gram matrix read
    // by the eigensolver, which reads the lower triangle); tiles strictly
    // above the diagonal skip
    if (lower && n0 >= m0 + GB_M) return;
    cplx acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = cmk(0.0, 0.0);

    for (int64_t k0 = k_lo; k0 < k_hi; k0 += GB_K) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int mm, kk;
            if (OPA == OP_N || OPA == OP_R) {
                mm = tid & 63;
                kk = (tid >> 6) + 4 * i;
            } else {
                kk = tid & 15;
                mm = (tid >> 4) + 16 * i;
            }
            const int64_t gm = m0 + mm, gk = k0 + kk;
            cplx v = cmk(0.0, 0.0);
            if (gm < M && gk < k_hi) {
                v = (OPA == OP_N || OPA == OP_R) ? A[gm + gk * lda] : A[gk + gm * lda];
                if (OPA == OP_C || OPA == OP_R) v.y = -v.y;
            }
            As[kk][mm] = v;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int kk, nn;
            if (OPB == OP_N || OPB == OP_R) {
                kk = tid & 15;
                nn = (tid >> 4) + 16 * i;
            } else {
                nn = tid & 63;
                kk = (tid >> 6) + 4 * i;
            }
            const int64_t gn = n0 + nn, gk = k0 + kk;
            cplx v = cmk(0.0, 0.0);
            if (gn < N && gk < k_hi) {
                v = (OPB == OP_N || OPB == OP_R) ? B[gk + gn * ldb] : B[gn + gk * ldb];
                if (OPB == OP_C || OPB == OP_R) v.y = -v.y;
            }
            Bs[kk][nn] = v;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < GB_K; ++kk) {
            cplx a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][tx + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][ty + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = cfma(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
    const bool use_beta = (beta.x != 0.0 || beta.y != 0.0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int64_t gn = n0 + ty + 16 * j;
        if (gn >= N) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t gm = m0 + tx + 16 * i;
            if (gm >= M) continue;
            cplx v = cmul(alpha, acc[i][j]);
            if (use_beta) v = cfma(beta, C[gm + gn * ldc], v);
            C[gm + gn * ldc] = v;
        }
    }
}

// Small and thin products: one thread per output element and K slice, a plain
// dot product; blockDim = (outputs, S) and the S slices of an element are added
// in slice order through shared memory.  GB300 issues one FP64 warp instruction
// per 16 clocks and SM, so operands read straight from L1/L2 keep that pipe
// busy and no tile is padded: what counts is that the outputs, times the
// slices where they are few, reach every SM.
constexpr int ZS_T = 512;  // most threads of a block

template <int OPA, int OPB>
__global__ void __launch_bounds__(ZS_T)
    zgemm_small_kernel(int64_t M, int64_t N, int64_t K, cplx alpha, const cplx* __restrict__ A,
                       int64_t lda, int64_t sA, const cplx* __restrict__ B, int64_t ldb, int64_t sB,
                       cplx beta, cplx* __restrict__ C, int64_t ldc, int64_t sC, int64_t batch,
                       int lower) {
    __shared__ cplx part[ZS_T];
    const int tx = threadIdx.x, ty = threadIdx.y, OX = blockDim.x, S = blockDim.y;
    const int64_t total = M * N * batch;
    const bool use_beta = (beta.x != 0.0 || beta.y != 0.0);
    const int64_t kc = (K + S - 1) / S, l0 = ty * kc, l1 = min(K, l0 + kc);
    for (int64_t base = blockIdx.x * (int64_t)OX; base < total; base += (int64_t)gridDim.x * OX) {
        const int64_t idx = base + tx;
        const int64_t i = idx % M, j = (idx / M) % N, b = idx / (M * N);
        const bool on = idx < total && !(lower && i < j);  // only the lower triangle is wanted
        cplx acc = cmk(0.0, 0.0);
        if (on) {
            const cplx* a = A + b * sA + ((OPA == OP_N || OPA == OP_R) ? i : i * lda);
            const cplx* bb = B + b * sB + ((OPB == OP_N || OPB == OP_R) ? j * ldb : j);
            const int64_t da = (OPA == OP_N || OPA == OP_R) ? lda : 1;
            const int64_t db = (OPB == OP_N || OPB == OP_R) ? 1 : ldb;
            auto step = [&](cplx x, cplx y) {
                if (OPA == OP_C || OPA == OP_R) x.y = -x.y;
                if (OPB == OP_C || OPB == OP_R) y.y = -y.y;
                acc = cfma(x, y, acc);
            };
            int64_t l = l0;
            for (; l + 3 < l1; l += 4) {  // four loads in flight
                cplx x[4], y[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    x[u] = a[(l + u) * da];
                    y[u] = bb[(l + u) * db];
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) step(x[u], y[u]);
            }
            for (; l < l1; ++l) step(a[l * da], bb[l * db]);
        }
        if (S > 1) {
            part[ty * OX + tx] = acc;
            __syncthreads();
            if (ty == 0)
                for (int s = 1; s < S; ++s) acc = cadd(acc, part[s * OX + tx]);
        }
        if (on && ty == 0) {
            cplx* c = C + b * sC + i + j * ldc;
            cplx v = cmul(alpha, acc);
            if (use_beta) v = cfma(beta, *c, v);
            *c = v;
        }
        if (S > 1) __syncthreads();
    }
}

// C = alpha sum_z P[z] + beta C over the split-K partials in chunk order
// (deterministic); lower: entries above the diagonal are left alone.
__global__ void splitk_reduce_kernel(const cplx* __restrict__ P, int64_t M, int64_t N, int S,
                                     cplx alpha, cplx beta, cplx* __restrict__ C, int64_t ldc,
                                     int lower) {
    const int64_t total = M * N;
    const bool use_beta = (beta.x != 0.0 || beta.y != 0.0);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = e % M, j = e / M;
        if (lower && i < j) continue;
        cplx acc = cmk(0, 0);
        for (int z = 0; z < S; ++z) acc = cadd(acc, P[e + (int64_t)z * total]);
        cplx v = cmul(alpha, acc);
        if (use_beta) v = cfma(beta, C[i + j * ldc], v);
        C[i + j * ldc] = v;
    }
}

template <int OPA>
void zgemm_small_dispatch_b(Ctx* ctx, Op opb, int64_t m, int64_t n, int64_t k, cplx alpha,
                            const cplx* A, int64_t lda, int64_t sA, const cplx* B, int64_t ldb,
                            int64_t sB, cplx beta, cplx* C, int64_t ldc, int64_t sC, int64_t batch,
                            int lower) {
    // Outputs per block: 32, fewer while the blocks would not reach every SM
    // twice (16 x 16 outputs, K = 1024: 37 us on 8 SMs, 7 us on 128); then K
    // slices of at least 16 terms up to a full warp, and on to eight warps per
    // SM.
    const int64_t outs = m * n * batch;
    // DMRG's sums of up to 192 terms stay in one piece (eig_fp64.cu).
    int OX = 32, S = 1;
    const bool whole = ctx->ordered && k <= 192;
    while (!whole && OX > 2 && outs < 2 * OX * (int64_t)ctx->sm_count && k >= 16 * (64 / OX)) OX /= 2;
    while (!whole && OX * S < 32 && k >= 32 * S) S *= 2;
    while (!whole && OX * S < ZS_T && outs / OX * ((OX * S + 31) / 32) < 8 * (int64_t)ctx->sm_count && k >= 32 * S) S *= 2;
    const unsigned g = (unsigned)std::min<int64_t>((outs + OX - 1) / OX, (int64_t)ctx->sm_count * 64);
    const dim3 th((unsigned)OX, (unsigned)S);
    switch (opb) {
#define TN_ZS(OB) case OB: zgemm_small_kernel<OPA, OB><<<g, th, 0, ctx->stream>>>(m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, lower); break;
        TN_ZS(OP_N) TN_ZS(OP_T) TN_ZS(OP_C) TN_ZS(OP_R)
#undef TN_ZS
    }
}

template <int OPA>
void zgemm_dispatch_b(Ctx* ctx, Op opb, dim3 grid, int64_t m, int64_t n, int64_t k, cplx alpha,
                      const cplx* A, int64_t lda, int64_t sA, const cplx* B, int64_t ldb,
                      int64_t sB, cplx beta, cplx* C, int64_t ldc, int64_t sC, int lower,
                      int64_t kc) {
    switch (opb) {
        case OP_N:
            zgemm_kernel<OPA, OP_N><<<grid, 256, 0, ctx->stream>>>(m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, lower, kc);
            break;
        case OP_T:
            zgemm_kernel<OPA, OP_T><<<grid, 256, 0, ctx->stream>>>(m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, lower, kc);
            break;
        case OP_C:
            zgemm_kernel<OPA, OP_C><<<grid, 256, 0, ctx->stream>>>(m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, lower, kc);
            break;
        case OP_R:
            zgemm_kernel<OPA, OP_R><<<grid, 256, 0, ctx->stream>>>(m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, lower, kc);
            break;
    }
}

// -------------------------------------------------------------------------
// out[a, J, c] = sum_I in[a, I, c] M[I, J].  Two-site MPO tensors are mostly zero (28
// of 144 entries for the transverse-field Ising chain, 52 of 400 for XXZ), and FP64
// is what bounds this kernel, so every block lists the nonzero entries of M's
// columns, real ones, imaginary ones (two multiply-adds either) and the rest (four),
// and a thread multiplies those; a column of the input with an infinity or NaN takes
// all entries, as 0 times it is NaN.  IN_ORDER: by their index instead, which gives the
// full sum's bits, for small bonds of DMRG (eig_fp64.cu); at bond dimension 256 a sweep
// of the XXZ chain takes 138 ms that way, 130 by kinds.  parts threads share a column's J.
// Against all entries of four J at a time by one thread: bond dimension 64, 12 x 12:
// 41.0 -> 8.2 us; 20 x 20: 104.5 -> 13.4, at 256 204 -> 30.7 (10.7 of them FP64).
template <bool IN_ORDER>
__global__ void __launch_bounds__(128, 8) small_apply_kernel(const cplx* __restrict__ in, cplx* __restrict__ out,
                                                          const cplx* __restrict__ M, int nI, int nJ, int64_t na,
                                                          int64_t nc, int64_t lda_i, int64_t ldc_i, int64_t lda_o,
                                                          int64_t ldc_o, int accumulate, int parts) {
    extern __shared__ cplx sM[];
    unsigned short* li = reinterpret_cast<unsigned short*>(sM + nI * nJ);  // nonzero I of column J, with their kind
    unsigned short* cnt = li + nI * nJ;  // 3 to a column: where each kind ends
    const int lane = threadIdx.x & 31;
    for (int t = threadIdx.x; t < nI * nJ; t += blockDim.x) sM[t] = M[t];
    __syncthreads();
    for (int J = threadIdx.x >> 5; J < nJ; J += blockDim.x >> 5) {
        int c = 0;
        for (int pass = 1; pass <= (IN_ORDER ? 1 : 3); ++pass) {
            for (int I0 = 0; I0 < nI; I0 += 32) {
                const int I = I0 + lane;
                int kind = 0;  // 1 real, 2 imaginary, 3 neither
                if (I < nI) {
                    const cplx v = sM[I + nI * J];
                    kind = (v.x != 0.0 ? 1 : 0) | (v.y != 0.0 ? 2 : 0);
                }
                const bool on = IN_ORDER ? kind != 0 : kind == pass;
                const unsigned m = __ballot_sync(0xffffffffu, on);
                if (on) li[nI * J + c + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(I | kind << 13);
                c += __popc(m);
            }
            if (lane == 0) cnt[3 * J + pass - 1] = (unsigned short)c;
        }
    }
    __syncthreads();
    const int64_t total = na * nc * parts;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = idx % na, c = idx / na % nc;
        const int part = (int)(idx / (na * nc));
        const cplx* x = in + a + ldc_i * c;
        cplx* y = out + a + ldc_o * c;
        bool bad = false;
        for (int I = 0; I < nI; ++I) {
            const cplx v = x[lda_i * I];
            bad |= (__double2hiint(v.x) & 0x7ff00000) == 0x7ff00000 || (__double2hiint(v.y) & 0x7ff00000) == 0x7ff00000;
        }
        for (int J = part; J < nJ; J += parts) {
            cplx s = cmk(0, 0);
            if (bad) {
                for (int I = 0; I < nI; ++I) s = cfma(x[lda_i * I], sM[I + nI * J], s);
            } else {
                const unsigned short* l = li + nI * J;
                const cplx* m = sM + nI * J;
                const int n0 = cnt[3 * J];
                if (IN_ORDER) {
#pragma unroll 4
                    for (int t = 0; t < n0; ++t) {
                        const int I = l[t] & 0x1fff, kind = l[t] >> 13;
                        const cplx v = x[lda_i * I], w = m[I];
                        if (kind == 1) s = cmk(fma(v.x, w.x, s.x), fma(v.y, w.x, s.y));
                        else if (kind == 2) s = cmk(fma(-v.y, w.y, s.x), fma(v.x, w.y, s.y));
                        else s = cfma(v, w, s);
                    }
                } else {
                    const int n1 = cnt[3 * J + 1], n2 = cnt[3 * J + 2];
#pragma unroll 4
                    for (int t = 0; t < n0; ++t) {
                        const int I = l[t] & 0x1fff;
                        const cplx v = x[lda_i * I];
                        const double r = m[I].x;
                        s = cmk(fma(v.x, r, s.x), fma(v.y, r, s.y));
                    }
#pragma unroll 2
                    for (int t = n0; t < n1; ++t) {
                        const int I = l[t] & 0x1fff;
                        const cplx v = x[lda_i * I];
                        const double r = m[I].y;
                        s = cmk(fma(-v.y, r, s.x), fma(v.x, r, s.y));
                    }
#pragma unroll 2
                    for (int t = n1; t < n2; ++t) {
                        const int I = l[t] & 0x1fff;
                        s = cfma(x[lda_i * I], m[I], s);
                    }
                }
            }
            cplx* dst = y + lda_o * J;
            *dst = accumulate ? cadd(*dst, s) : s;
        }
    }
}

// The same for nI <= 4 (gates and operators on one or two spin-1/2 legs), a thread per
// output and all loads at once: what takes the time there is one load's latency, and
// lists of nonzeros would be two more (2 x 2: 5.2 us with them, 4.1 without;
// 4 x 4 at bond dimension 32: 6.2 and 4.1).
__global__ void __launch_bounds__(128) dense_apply_kernel(const cplx* __restrict__ in, cplx* __restrict__ out,
                                                          const cplx* __restrict__ M, int nI, int nJ, int64_t na,
                                                          int64_t nc, int64_t lda_i, int64_t ldc_i, int64_t lda_o,
                                                          int64_t ldc_o, int accumulate) {
    const int64_t total = na * nc * nJ;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = idx % na, c = idx / na / nJ;
        const int J = (int)(idx / na % nJ);
        const cplx* x = in + a + ldc_i * c;
        cplx v[4], m[4];
#pragma unroll
        for (int I = 0; I < 4; ++I)
            if (I < nI) {
                v[I] = x[lda_i * I];
                m[I] = M[I + nI * J];
            }
        cplx s = cmk(0, 0);
#pragma unroll
        for (int I = 0; I < 4; ++I)
            if (I < nI) s = cfma(v[I], m[I], s);
        cplx* dst = out + a + ldc_o * c + lda_o * J;
        *dst = accumulate ? cadd(*dst, s) : s;
    }
}

// -------------------------------------------------------------------------
constexpr int MAXV = 8;
struct PtrPack {
    const cplx* p[MAXV];
};

__device__ inline cplx warp_sum(cplx v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_down_sync(0xffffffffu, v.x, o);
        v.y += __shfl_down_sync(0xffffffffu, v.y, o);
    }
    return v;
}

// Sum of all blocks' partials of K outputs by the block that comes last, one warp per
// output in fixed order (a launch of its own for that took 3.3 us).  red: the
// block's partials, in shared memory; count is zero before and after.
__device__ inline void last_block_sum(const cplx* red, int K, cplx* __restrict__ partial, cplx* __restrict__ out,
                                      unsigned* __restrict__ count) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (gridDim.x == 1) {
        if (t < K) out[t] = red[t];
        return;
    }
    __shared__ bool s_last;
    if (t < K) {
        partial[blockIdx.x * K + t] = red[t];
        __threadfence();
    }
    __syncthreads();
    if (t == 0) s_last = atomicInc(count, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int j = warp; j < K; j += blockDim.x >> 5) {
        cplx s = cmk(0, 0);
        for (int b = lane; b < (int)gridDim.x; b += 32) {
            const double2 v = __ldcg(reinterpret_cast<const double2*>(partial) + b * K + j);
            s = cadd(s, cmk(v.x, v.y));
        }
        s = warp_sum(s);
        if (lane == 0) out[j] = s;
    }
}

// out[j] = sum of conj(v_j[i]) * w[i]
template <int K>
__global__ void __launch_bounds__(256) multi_dot_kernel(PtrPack V, const cplx* __restrict__ w,
                                                        int64_t n, cplx* __restrict__ partial,
                                                        cplx* __restrict__ out, unsigned* __restrict__ count) {
    cplx acc[K];
#pragma unroll
    for (int j = 0; j < K; ++j) acc[j] = cmk(0, 0);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const cplx wi = w[i];
#pragma unroll
        for (int j = 0; j < K; ++j) acc[j] = cfma(cconj(V.p[j][i]), wi, acc[j]);
    }
    __shared__ cplx red[8][K];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < K; ++j) {
        cplx s = warp_sum(acc[j]);
        if (lane == 0) red[warp][j] = s;
    }
    __syncthreads();
    __shared__ cplx sum[K];
    if (threadIdx.x < K) {
        cplx s = cmk(0, 0);
        for (int wp = 0; wp < (int)(blockDim.x >> 5); ++wp) s = cadd(s, red[wp][threadIdx.x]);
        sum[threadIdx.x] = s;
    }
    last_block_sum(sum, K, partial, out, count);
}

__global__ void __launch_bounds__(256) bilinear_dot_kernel(const cplx* __restrict__ x,
                                                           const cplx* __restrict__ y, int64_t n,
                                                           cplx* __restrict__ partial, cplx* __restrict__ out,
                                                           unsigned* __restrict__ count) {
    cplx acc = cmk(0, 0);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        acc = cfma(x[i], y[i], acc);
    __shared__ cplx red[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    acc = warp_sum(acc);
    if (lane == 0) red[warp] = acc;
    __syncthreads();
    __shared__ cplx sum;
    if (threadIdx.x == 0) {
        cplx s = cmk(0, 0);
        for (int wp = 0; wp < (int)(blockDim.x >> 5); ++wp) s = cadd(s, red[wp]);
        sum = s;
    }
    last_block_sum(&sum, 1, partial, out, count);
}

template <int K>
__global__ void multi_axpy_kernel(cplx* __restrict__ w, PtrPack V, const cplx* __restrict__ coef,
                                  int64_t n, double sign) {
    cplx c[K];
#pragma unroll
    for (int j = 0; j < K; ++j) c[j] = cmk(sign * coef[j].x, sign * coef[j].y);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        cplx acc = w[i];
#pragma unroll
        for (int j = 0; j < K; ++j) acc = cfma(c[j], V.p[j][i], acc);
        w[i] = acc;
    }
}

// ---- one Lanczos step's orthogonalisation ------------------------------------
// w <- w minus its components along v_0 .. v_{K-1}, twice (classical Gram-Schmidt);
// w <- w / |w|.  coef: the K components of either pass, |w|^2 and a mark that the
// kernel ran to its end.  One cooperative grid in place of nine launches and a host
// round trip: a thread keeps to its entries of w, so only the K + K + 1 sums cross
// blocks, in fixed order, at a barrier each (1.2 us).  On average over a DMRG run at
// bond dimension 64 (vectors up to 16,384, K up to 8): 47 us of kernels and nine
// gaps -> 17.6 us.  FP64 bounds long vectors (16 K instructions an entry), as before.
constexpr int LMAX = 49, LG = 8;
struct LanczosArgs {
    const cplx* v[LMAX];
    cplx *w, *partial, *coef;  // partial: gridDim.x x (2 LMAX + 1); coef: host memory
    int64_t n;
    int K;
    double mark;
    unsigned *bar, *exits;  // zero at launch and after
    int* err;
};

// Sums over a warp of LG complex values: halves change lanes, so that 16 additions
// do for 16 sums (64 clocks each; five a sum otherwise).  Lane 2 r gets value r of
// (re_0, im_0, re_1, ...).
__device__ __forceinline__ double warp_sums(const cplx* acc) {
    const int lane = threadIdx.x & 31;
    double v[2 * LG];
#pragma unroll
    for (int j = 0; j < LG; ++j) {
        v[2 * j] = acc[j].x;
        v[2 * j + 1] = acc[j].y;
    }
#pragma unroll
    for (int h = LG, o = 16; h >= 1; h >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int j = 0; j < h; ++j) {
            const double give = up ? v[j] : v[j + h], keep = up ? v[j + h] : v[j];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

__global__ void __launch_bounds__(512) lanczos_orth_kernel(LanczosArgs p) {
    __shared__ double red[16][2 * LG];
    __shared__ cplx c[LMAX];
    const int nw = blockDim.x >> 5, t = threadIdx.x, lane = t & 31, warp = t >> 5, C = gridDim.x, K = p.K;
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + t, di = (int64_t)C * blockDim.x;
    unsigned arrivals = 0;
    // this block's sum of nv values a thread to slot s of the partials
    auto put = [&](const cplx* acc, int nv, int s) {
        const double v = warp_sums(acc);
        if (!(lane & 1)) red[warp][lane >> 1] = v;
        __syncthreads();
        if (t < 2 * nv) {
            double u = red[0][t];
            for (int k = 1; k < nw; ++k) u += red[k][t];
            reinterpret_cast<double*>(p.partial)[2 * ((int64_t)blockIdx.x * (2 * LMAX + 1) + s) + t] = u;
        }
        __syncthreads();
    };
    // all blocks' partials of slots s .. s + nv - 1, to c and (block 0) to coef
    auto gather = [&](int nv, int s) -> bool {
        arrivals += (unsigned)C;
        if (C > 1 && !griddev::grid_sync(p.bar, p.err, arrivals)) return false;
        for (int j = warp; j < nv; j += nw) {
            cplx v = cmk(0, 0);
            for (int b = lane; b < C; b += 32) {
                const double2 x = __ldcg(reinterpret_cast<const double2*>(p.partial) + (int64_t)b * (2 * LMAX + 1) + s + j);
                v = cadd(v, cmk(x.x, x.y));
            }
            v = warp_sum(v);
            if (lane == 0) {
                c[j] = v;
                if (blockIdx.x == 0) p.coef[s + j] = v;
            }
        }
        __syncthreads();
        return true;
    };
    // subtract the components c and, in the same pass, take the products for the next
    // sums with the vectors of group j0 (the last group holds the finished entries)
    for (int j0 = 0; j0 < K; j0 += LG) {
        const int kk = min(LG, K - j0);
        cplx acc[LG];
#pragma unroll
        for (int j = 0; j < LG; ++j) acc[j] = cmk(0, 0);
        for (int64_t i = i0; i < p.n; i += di) {
            const cplx w = p.w[i];
#pragma unroll
            for (int j = 0; j < LG; ++j)
                if (j < kk) acc[j] = cfma(cconj(p.v[j0 + j][i]), w, acc[j]);
        }
        put(acc, kk, j0);
    }
    for (int pass = 0; pass < 2; ++pass) {
        if (!gather(K, pass * LMAX)) return;
        for (int j0 = 0; j0 < K; j0 += LG) {
            const int kk = min(LG, K - j0);
            const bool last = j0 + LG >= K;
            cplx acc[LG];
#pragma unroll
            for (int j = 0; j < LG; ++j) acc[j] = cmk(0, 0);
            for (int64_t i = i0; i < p.n; i += di) {
                cplx w = p.w[i], v[LG];
#pragma unroll
                for (int j = 0; j < LG; ++j)
                    if (j < kk) {
                        v[j] = p.v[j0 + j][i];
                        w = cfma(cmk(-c[j0 + j].x, -c[j0 + j].y), v[j], w);
                    }
                p.w[i] = w;
                if (pass == 1) {
                    if (last) acc[0].x = fma(w.x, w.x, fma(w.y, w.y, acc[0].x));
                } else if (K <= LG) {
#pragma unroll
                    for (int j = 0; j < LG; ++j)
                        if (j < kk) acc[j] = cfma(cconj(v[j]), w, acc[j]);
                }
            }
            if (pass == 0 && K <= LG) put(acc, kk, LMAX);
            if (pass == 1 && last) put(acc, 1, 2 * LMAX);
        }
        if (pass == 0 && K > LG)  // components of the finished w
            for (int j0 = 0; j0 < K; j0 += LG) {
                const int kk = min(LG, K - j0);
                cplx acc[LG];
#pragma unroll
                for (int j = 0; j < LG; ++j) acc[j] = cmk(0, 0);
                for (int64_t i = i0; i < p.n; i += di) {
                    const cplx w = p.w[i];
#pragma unroll
                    for (int j = 0; j < LG; ++j)
                        if (j < kk) acc[j] = cfma(cconj(p.v[j0 + j][i]), w, acc[j]);
                }
                put(acc, kk, LMAX + j0);
            }
    }
    if (!gather(1, 2 * LMAX)) return;
    const double b2 = c[0].x, s = b2 > 0.0 ? 1.0 / sqrt(b2) : 0.0;
    for (int64_t i = i0; i < p.n; i += di) p.w[i] = cmk(p.w[i].x * s, p.w[i].y * s);
    if (t == 0) {
        if (blockIdx.x == 0) p.coef[2 * LMAX + 1] = cmk(p.mark, 0.0);
        // everybody has passed the last barrier once the last block is here
        if (atomicInc(p.exits, C - 1) == (unsigned)C - 1) *p.bar = 0;
    }
}

__global__ void zaxpy_kernel(cplx* __restrict__ y, const cplx* __restrict__ x, int64_t n, cplx a) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        y[i] = cfma(a, x[i], y[i]);
}

__global__ void zscale_kernel(cplx* x, int64_t n, cplx a) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        x[i] = cmul(a, x[i]);
}

__global__ void zscale_dev_kernel(cplx* x, int64_t n, const double* dnorm2, int invert_sqrt) {
    const double s = invert_sqrt ? 1.0 / sqrt(*dnorm2) : *dnorm2;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        x[i] = cmk(x[i].x * s, x[i].y * s);
}

__global__ void zfill_kernel(cplx* x, int64_t n, cplx v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        x[i] = v;
}

__global__ void top_eigvecs_kernel(const cplx* __restrict__ G, int64_t n, int64_t k,
                                   int64_t ncols, cplx* __restrict__ dst) {
    const int64_t total = n * k;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = idx % n, j = idx / n;
        dst[i + n * j] = G[i + n * (ncols - 1 - j)];
    }
}

__global__ void grading_kernel(const cplx* __restrict__ G, int64_t n, int* __restrict__ out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = (int)((((unsigned)__double2hiint(G[i + n * i].x) >> 20) & 0x7ffu) / 2);
}

__global__ void scale_cols_kernel(cplx* X, int64_t m, int64_t k, const double* s, int invert) {
    const int64_t total = m * k;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = idx / m;
        const double f = invert ? (s[j] > 0 ? 1.0 / s[j] : 0.0) : s[j];
        X[idx] = cmk(X[idx].x * f, X[idx].y * f);
    }
}

__global__ void scale_rows_kernel(cplx* X, int64_t k, int64_t n, const double* s, int invert) {
    const int64_t total = k * n;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = idx % k;
        const double f = invert ? (s[j] > 0 ? 1.0 / s[j] : 0.0) : s[j];
        X[idx] = cmk(X[idx].x * f, X[idx].y * f);
    }
}

__global__ void conj_transpose_kernel(const cplx* __restrict__ src, int64_t r, int64_t c,
                                      cplx* __restrict__ dst) {
    __shared__ cplx tile[32][33];
    const int64_t r0 = (int64_t)blockIdx.x * 32, c0 = (int64_t)blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int64_t gr = r0 + threadIdx.x, gc = c0 + j;
        if (gr < r && gc < c) tile[j][threadIdx.x] = src[gr + r * gc];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int64_t gc = c0 + threadIdx.x, gr = r0 + j;
        if (gr < r && gc < c) dst[gc + c * gr] = cconj(tile[threadIdx.x][j]);
    }
}

// out[j] = ||X[:, j]||, one warp per column
__global__ void col_norms_kernel(const cplx* __restrict__ X, int64_t m, int64_t k,
                                 double* __restrict__ out) {
    const int64_t j = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (j >= k) return;
    double s = 0.0;
    for (int64_t i = lane; i < m; i += 32) {
        const cplx v = X[i + m * j];
        s = fma(v.x, v.x, fma(v.y, v.y, s));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) out[j] = sqrt(s);
}

// out[i] = ||Y[i, :]|| for a column-major k x n matrix, one thread per row
__global__ void row_norms_kernel(const cplx* __restrict__ Y, int64_t k, int64_t n,
                                 double* __restrict__ out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= k) return;
    double s = 0.0;
    for (int64_t j = 0; j < n; ++j) {
        const cplx v = Y[i + k * j];
        s = fma(v.x, v.x, fma(v.y, v.y, s));
    }
    out[i] = sqrt(s);
}

// -------------------------------------------------------------------------
// Keep rule (src/tensors.jl:200-215) on ascending Gram eigenvalues.  One
// block; thread t owns a contiguous chunk of the descending squared singular
// values; suffix sums come from a warp-shuffle scan over chunk totals.
struct KeepDev {
    int64_t k;
    double total, discarded;
    int64_t err;  // the eigensolver's barriers ran out
};

__device__ inline double s2_at(const double* lam, int64_t n, int64_t i) {
    const double v = lam[n - 1 - i];
    return v > 0.0 ? v : 0.0;
}

__global__ void __launch_bounds__(1024) keep_rule_kernel(const double* __restrict__ lam, int64_t n,
                                                         int64_t sz, double cutoff, int64_t maxdim,
                                                         int64_t mindim, double* __restrict__ S_out,
                                                         const cplx* __restrict__ G, int64_t g,
                                                         const int* __restrict__ dinfo,
                                                         KeepDev* __restrict__ res) {
    __shared__ double wsum[32];
    __shared__ long long wcnt[32];
    __shared__ double s_total, s_rest;
    __shared__ int64_t s_k;
    const int T = blockDim.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nw = T >> 5;
    const int64_t per = (sz + T - 1) / T;
    const int64_t lo = min((int64_t)t * per, sz), hi = min(lo + per, sz);
    // the whole spectrum's weight: the trace of the Gram matrix
    __shared__ double wtr[32];
    if (G) {
        double tr = 0.0;
        for (int64_t i = t; i < g; i += T) tr += G[i + g * i].x;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tr += __shfl_down_sync(0xffffffffu, tr, o);
        if (lane == 0) wtr[warp] = tr;
    }
    double local = 0.0;
    for (int64_t i = hi - 1; i >= lo; --i) local += s2_at(lam, n, i);
    // inclusive suffix scan over threads: incl(t) = sum_{t' >= t} local(t')
    double v = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_down_sync(0xffffffffu, v, o);
        if (lane + o < 32) v += u;
    }
    if (lane == 0) wsum[warp] = v;  // warp total
    __syncthreads();
    if (t == 0) {
        double acc = 0.0;
        for (int w = nw - 1; w >= 0; --w) {
            const double tw = wsum[w];
            wsum[w] = acc;  // sum of warps after w
            acc += tw;
        }
        // partial spectrum: the weight below the available values is the
        // trace minus their sum
        double tr = 0.0;
        for (int w = 0; G && w < nw; ++w) tr += wtr[w];
        const double rest = G ? fmax(tr - acc, 0.0) : 0.0;
        s_rest = rest;
        s_total = acc + rest;
    }
    __syncthreads();
    const double rest = s_rest;
    const double after = v - local + wsum[warp] + rest;  // weight after chunk t
    const double total = s_total;
    long long cnt = 0;
    double tail = after;
    for (int64_t i = hi - 1; i >= lo; --i) {
        tail += s2_at(lam, n, i);
        if (tail / total > cutoff) ++cnt;  // NaN (total 0) compares false
        if (S_out) S_out[i] = sqrt(s2_at(lam, n, i));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    if (lane == 0) wcnt[warp] = cnt;
    __syncthreads();
    if (t == 0) {
        long long c = 0;
        for (int w = 0; w < nw; ++w) c += wcnt[w];
        int64_t mind = min(mindim, sz);
        int64_t maxd = (maxdim == 0 || maxdim > sz) ? sz : maxdim;
        if (maxd == 0) maxd = 1;
        if (cutoff != 0.0) {
            const int64_t idxs = c > 0 ? (int64_t)c : 1;
            maxd = min(maxd, idxs);
        }
        s_k = max(maxd, mind);
    }
    __syncthreads();
    // discarded weight = sum_{i >= k} s2 / total
    const int64_t k = s_k;
    double disc = 0.0;
    for (int64_t i = max(lo, k); i < hi; ++i) disc += s2_at(lam, n, i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) disc += __shfl_down_sync(0xffffffffu, disc, o);
    __syncthreads();
    if (lane == 0) wsum[warp] = disc;
    __syncthreads();
    if (t == 0) {
        double d = rest;
        for (int w = 0; w < nw; ++w) d += wsum[w];
        res->k = k;
        res->total = total;
        res->discarded = total > 0 ? d / total : 0.0;
        res->err = dinfo ? *dinfo : 0;
    }
}

// Multiply-adds from which the tensor-core product is the faster one: it takes
// five stream operations (27 us at any size up to 256 x 128 x 128 = 4.2 M, where
// the per-output kernel takes 37 us; at 128^3 = 2.1 M it is 27 us against 23).
constexpr double ZTC_MIN = 2.5e6;
inline double gemm_work(int64_t m, int64_t n, int64_t k, int64_t batch, bool lower) {
    return (lower ? 0.5 : 1.0) * (double)m * n * k * batch;
}

// Threads of a kernel of one block that scans n values: no more warps than there are
// values for, as every FP64 instruction of every warp holds its scheduler for 64
// clocks (the keep rule of 32 values takes 6.7 us with one warp, 13 with 32).
inline unsigned one_block(int64_t n) { return (unsigned)std::min<int64_t>(1024, (n + 31) / 32 * 32); }

inline int grid_for(Ctx* ctx, int64_t n, int threads = 256) {
    int64_t g = (n + threads - 1) / threads;
    const int64_t cap = (int64_t)ctx->sm_count * 8;
    if (g > cap) g = cap;
    return (int)(g < 1 ? 1 : g);
}

}  // namespace

// -------------------------------------------------------------------------
// Large products run on the tensor cores.  Thin ones (a side below 16) read more than
// they multiply: there the operand conversion (64 bytes written per entry) costs more
// than the FP64 pipe.
bool tc_sized(const Ctx* ctx, int64_t m, int64_t n, int64_t k, bool lower) {
    return ctx->splitk && std::min(m, n) >= 16 && k >= 8 && gemm_work(m, n, k, 1, lower) >= ZTC_MIN;
}

void zgemm(Ctx* ctx, Op opa, Op opb, int64_t m, int64_t n, int64_t k, cplx alpha, const cplx* A,
           int64_t lda, int64_t sA, const cplx* B, int64_t ldb, int64_t sB, cplx beta, cplx* C,
           int64_t ldc, int64_t sC, int64_t batch, bool lower_only, const int* kexp, int ksign) {
    if (batch == 1 && tc_sized(ctx, m, n, k, lower_only)) {
        ProfScope ps(ctx, 1, 8.0 * gemm_work(m, n, k, 1, lower_only), 16.0 * (double)(m * k + k * n + m * n));
        if (zgemm_tc(ctx, opa, opb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, lower_only, kexp, ksign)) return;
    }
    zgemm_fp64(ctx, opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, lower_only);
}

void zgemm_fp64(Ctx* ctx, Op opa, Op opb, int64_t m, int64_t n, int64_t k, cplx alpha, const cplx* A,
                int64_t lda, int64_t sA, const cplx* B, int64_t ldb, int64_t sB, cplx beta, cplx* C,
                int64_t ldc, int64_t sC, int64_t batch, bool lower_only) {
    if (m <= 0 || n <= 0 || batch <= 0) return;
    const int lower = lower_only ? 1 : 0;
    TN_REQUIRE((n + GB_N - 1) / GB_N <= 65535 && batch <= 65535, "zgemm: grid too large");
    dim3 grid((unsigned)((m + GB_M - 1) / GB_M), (unsigned)((n + GB_N - 1) / GB_N), (unsigned)batch);
    if (k <= 0) {  // C = beta * C
        alpha = cmk(0, 0);
    }
    const double work = gemm_work(m, n, std::max<int64_t>(k, 0), batch, lower_only);
    ProfScope ps(ctx, 1, 8.0 * work, 16.0 * (double)(m * k + k * n + m * n) * batch);
    // A 64 x 64 tile keeps one SM busy for 4.1 us per K entry at two FP64 FMAs per clock
    // (64^3: 263 us), the per-output kernel spreads the same work over the SMs
    // (64^3: 7 us).  Tiles, with their reuse, pay once they fill the SMs.
    if (std::min(m, n) < 48 || work < 6.0e7) {
        switch (opa) {
            case OP_N: zgemm_small_dispatch_b<OP_N>(ctx, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, lower); break;
            case OP_T: zgemm_small_dispatch_b<OP_T>(ctx, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, lower); break;
            case OP_C: zgemm_small_dispatch_b<OP_C>(ctx, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, lower); break;
            case OP_R: zgemm_small_dispatch_b<OP_R>(ctx, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, lower); break;
        }
        ctx->count();
        TN_CHECK_CUDA(cudaGetLastError());
        return;
    }
    // Split K when the tiles cannot fill the SMs (a long
    // inner dimension under a small result): S chunks of at least 128, each
    // into its own partial, summed in chunk order by a second kernel.
    const int64_t tiles = (int64_t)grid.x * grid.y;
    int64_t S = 1;
    if (ctx->splitk && batch == 1 && k >= 512 && tiles < ctx->sm_count)
        S = std::min<int64_t>((2 * ctx->sm_count + tiles - 1) / tiles, k / 128);
    if (S > 1) {
        const int64_t kc = ((k + S - 1) / S + GB_K - 1) / GB_K * GB_K;
        S = (k + kc - 1) / kc;
        cplx* P = ctx->s_splitk.c(ctx, (size_t)(S * m * n));
        dim3 g2(grid.x, grid.y, (unsigned)S);
        const cplx one = cmk(1, 0), zero = cmk(0, 0);
        switch (opa) {
            case OP_N: zgemm_dispatch_b<OP_N>(ctx, opb, g2, m, n, k, one, A, lda, 0, B, ldb, 0, zero, P, m, 0, lower, kc); break;
            case OP_T: zgemm_dispatch_b<OP_T>(ctx, opb, g2, m, n, k, one, A, lda, 0, B, ldb, 0, zero, P, m, 0, lower, kc); break;
            case OP_C: zgemm_dispatch_b<OP_C>(ctx, opb, g2, m, n, k, one, A, lda, 0, B, ldb, 0, zero, P, m, 0, lower, kc); break;
            case OP_R: zgemm_dispatch_b<OP_R>(ctx, opb, g2, m, n, k, one, A, lda, 0, B, ldb, 0, zero, P, m, 0, lower, kc); break;
        }
        ctx->count();
        TN_CHECK_CUDA(cudaGetLastError());
        const int64_t blocks = std::min<int64_t>((m * n + 255) / 256, (int64_t)ctx->sm_count * 8);
        splitk_reduce_kernel<<<(unsigned)blocks, 256, 0, ctx->stream>>>(P, m, n, (int)S, alpha, beta,
                                                                        C, ldc, lower);
        ctx->count();
        TN_CHECK_CUDA(cudaGetLastError());
        return;
    }
    switch (opa) {
        case OP_N: zgemm_dispatch_b<OP_N>(ctx, opb, grid, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, lower, 0); break;
        case OP_T: zgemm_dispatch_b<OP_T>(ctx, opb, grid, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, lower, 0); break;
        case OP_C: zgemm_dispatch_b<OP_C>(ctx, opb, grid, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, lower, 0); break;
        case OP_R: zgemm_dispatch_b<OP_R>(ctx, opb, grid, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, lower, 0); break;
    }
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

void small_apply(Ctx* ctx, const cplx* in, cplx* out, const cplx* M, int nI, int nJ, int64_t na,
                 int64_t nc, int64_t lda_i, int64_t ldc_i, int64_t lda_o, int64_t ldc_o,
                 bool accumulate) {
    if (na <= 0 || nc <= 0) return;
    TN_REQUIRE(nI * nJ <= 4096, "small_apply: operator too large");
    ProfScope ps(ctx, 3, 8.0 * na * nc * nI * nJ, 16.0 * na * nc * (nI + nJ));
    if (nI <= 4) {
        dense_apply_kernel<<<grid_for(ctx, na * nc * nJ, 128), 128, 0, ctx->stream>>>(
            in, out, M, nI, nJ, na, nc, lda_i, ldc_i, lda_o, ldc_o, accumulate ? 1 : 0);
        ctx->count();
        TN_CHECK_CUDA(cudaGetLastError());
        return;
    }
    const size_t smem = (sizeof(cplx) + 2) * nI * nJ + 6 * nJ;
    // the whole operator is staged in shared memory: up to 96 KiB, above the
    // 48 KiB a launch gets without opting in
    auto kernel = ctx->ordered && na * nc <= 4096 ? small_apply_kernel<true> : small_apply_kernel<false>;
    if (smem > 48 * 1024)
        TN_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           18 * 4096 + 6 * 4096));
    // threads to a column until two warps are on every scheduler
    int parts = 1;
    while (parts < nJ && na * nc * parts < (int64_t)ctx->sm_count * 256) parts *= 2;
    parts = std::min(parts, nJ);
    kernel<<<grid_for(ctx, na * nc * parts, 128), 128, smem, ctx->stream>>>(
        in, out, M, nI, nJ, na, nc, lda_i, ldc_i, lda_o, ldc_o, accumulate ? 1 : 0, parts);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

void multi_dot(Ctx* ctx, const cplx* const* hV, int K, const cplx* w, int64_t n, cplx* dout) {
    ProfScope ps(ctx, 6, 8.0 * n * K, 16.0 * n * (K + 1));
    const int nblk = grid_for(ctx, n);
    cplx* partial = ctx->s_dot.c(ctx, (size_t)nblk * MAXV);
    for (int j0 = 0; j0 < K; j0 += MAXV) {
        const int kk = std::min(MAXV, K - j0);
        PtrPack P{};
        for (int j = 0; j < kk; ++j) P.p[j] = hV[j0 + j];
        switch (kk) {
#define TN_MD(KK) case KK: multi_dot_kernel<KK><<<nblk, 256, 0, ctx->stream>>>(P, w, n, partial, dout + j0, ctx->d_bar + 3); break;
            TN_MD(1) TN_MD(2) TN_MD(3) TN_MD(4) TN_MD(5) TN_MD(6) TN_MD(7) TN_MD(8)
#undef TN_MD
        }
        ctx->count();
    }
    TN_CHECK_CUDA(cudaGetLastError());
}

void bilinear_dot(Ctx* ctx, const cplx* x, const cplx* y, int64_t n, cplx* dout) {
    const int nblk = grid_for(ctx, n);
    cplx* partial = ctx->s_dot.c(ctx, (size_t)nblk * MAXV);
    bilinear_dot_kernel<<<nblk, 256, 0, ctx->stream>>>(x, y, n, partial, dout, ctx->d_bar + 3);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

void multi_axpy(Ctx* ctx, cplx* w, const cplx* const* hV, const cplx* dcoef, int K, int64_t n,
                double sign) {
    ProfScope ps(ctx, 6, 8.0 * n * K, 16.0 * n * (K + 2));
    const int nblk = grid_for(ctx, n);
    for (int j0 = 0; j0 < K; j0 += MAXV) {
        const int kk = std::min(MAXV, K - j0);
        PtrPack P{};
        for (int j = 0; j < kk; ++j) P.p[j] = hV[j0 + j];
        switch (kk) {
#define TN_MA(KK) case KK: multi_axpy_kernel<KK><<<nblk, 256, 0, ctx->stream>>>(w, P, dcoef + j0, n, sign); break;
            TN_MA(1) TN_MA(2) TN_MA(3) TN_MA(4) TN_MA(5) TN_MA(6) TN_MA(7) TN_MA(8)
#undef TN_MA
        }
        ctx->count();
    }
    TN_CHECK_CUDA(cudaGetLastError());
}

// The components of both passes (c1[j] + c2[j] to comp[j]) and |w| of the result, w
// divided by it; one host synchronisation.
double lanczos_orth(Ctx* ctx, const cplx* const* hV, int K, cplx* w, int64_t n, cplx* comp) {
    TN_REQUIRE(K >= 1 && K <= LMAX, "lanczos_orth: too many vectors");
    ProfScope ps(ctx, 6, 32.0 * n * K, 16.0 * n * (3 * K + 5));
    LanczosArgs a{};
    for (int j = 0; j < K; ++j) a.v[j] = hV[j];
    // Up to 256 entries an SM a thread has one entry and the sums are those of
    // multi_dot's blocks, in its order (DMRG's results rest on it, eig_fp64.cu).  Above,
    // one warp on every scheduler keeps the FP64 units busy and has the fewest sums;
    // vectors beyond L2 want more loads in flight.
    const int threads = n <= 256 * (int64_t)ctx->sm_count ? 256 : n <= (1 << 20) ? 128 : 512;
    const int C = (int)std::min<int64_t>(ctx->sm_count, (n + threads - 1) / threads);
    a.partial = ctx->s_dot.c(ctx, (size_t)C * (2 * LMAX + 1));
    double* h = ctx->pinned(2 * (2 * LMAX + 2));
    unset(h, 2 * (2 * LMAX + 2));
    a.coef = reinterpret_cast<cplx*>(h);
    a.w = w;
    a.n = n;
    a.K = K;
    a.mark = (double)++ctx->lanczos_calls;
    a.bar = ctx->d_bar + 4;
    a.exits = ctx->d_bar + 5;
    a.err = reinterpret_cast<int*>(ctx->d_bar + 6);
    void* args[] = {&a};
    TN_CHECK_CUDA(cudaLaunchCooperativeKernel((void*)lanczos_orth_kernel, dim3((unsigned)C), dim3(threads), args, 0,
                                              ctx->stream));
    ctx->count();
    ctx->sync();
    if (h[2 * (2 * LMAX + 1)] != a.mark) {
        TN_CHECK_CUDA(cudaMemsetAsync(ctx->d_bar + 4, 0, 3 * sizeof(unsigned), ctx->stream));
        throw Error(TN_ERR_TIMEOUT, "Lanczos: a bounded grid barrier ran out");
    }
    check_set(h, 2 * K);
    check_set(h + 2 * LMAX, 2 * K);
    check_set(h + 4 * LMAX, 2);
    for (int j = 0; j < K; ++j)
        comp[j] = cmk(h[2 * j] + h[2 * (LMAX + j)], h[2 * j + 1] + h[2 * (LMAX + j) + 1]);
    return std::sqrt(h[4 * LMAX]);
}

void zaxpy(Ctx* ctx, cplx* y, const cplx* x, int64_t n, cplx a) {
    if (n <= 0) return;
    ProfScope ps(ctx, 6, 8.0 * n, 48.0 * n);
    zaxpy_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(y, x, n, a);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

void zscale(Ctx* ctx, cplx* x, int64_t n, cplx a) {
    if (n <= 0) return;
    zscale_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(x, n, a);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

void zscale_dev(Ctx* ctx, cplx* x, int64_t n, const double* dnorm2, int invert) {
    if (n <= 0) return;
    zscale_dev_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(x, n, dnorm2, invert);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

void zcopy(Ctx* ctx, cplx* dst, const cplx* src, int64_t n) {
    if (n <= 0) return;
    TN_CHECK_CUDA(cudaMemcpyAsync(dst, src, n * sizeof(cplx), cudaMemcpyDeviceToDevice, ctx->stream));
}

void zfill(Ctx* ctx, cplx* dst, int64_t n, cplx v) {
    if (n <= 0) return;
    zfill_kernel<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(dst, n, v);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

double znorm2(Ctx* ctx, const cplx* x, int64_t n) {
    const cplx* V[1] = {x};
    double* h = ctx->pinned(2);  // the kernel writes there
    unset(h, 2);
    multi_dot(ctx, V, 1, x, n, reinterpret_cast<cplx*>(h));
    ctx->sync();
    check_set(h, 2);
    return h[0];
}

void grading(Ctx* ctx, const cplx* G, int64_t n, int* out) {
    grading_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(G, n, out);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

void take_top_eigvecs(Ctx* ctx, const cplx* G, int64_t n, int64_t k, cplx* dst, int64_t ncols) {
    if (n <= 0 || k <= 0) return;
    if (ncols < 0) ncols = n;
    TN_REQUIRE(k <= ncols, "take_top_eigvecs: k exceeds the available eigenvectors");
    top_eigvecs_kernel<<<grid_for(ctx, n * k), 256, 0, ctx->stream>>>(G, n, k, ncols, dst);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

void conj_transpose(Ctx* ctx, const cplx* src, int64_t r, int64_t c, cplx* dst) {
    if (r <= 0 || c <= 0) return;
    TN_REQUIRE((c + 31) / 32 <= 65535, "conj_transpose: too many columns");
    dim3 grid((unsigned)((r + 31) / 32), (unsigned)((c + 31) / 32));
    conj_transpose_kernel<<<grid, dim3(32, 8), 0, ctx->stream>>>(src, r, c, dst);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

void col_norms(Ctx* ctx, const cplx* X, int64_t m, int64_t k, double* out) {
    if (m <= 0 || k <= 0) return;
    col_norms_kernel<<<(unsigned)((k + 7) / 8), 256, 0, ctx->stream>>>(X, m, k, out);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

void row_norms(Ctx* ctx, const cplx* Y, int64_t k, int64_t n, double* out) {
    if (n <= 0 || k <= 0) return;
    row_norms_kernel<<<(unsigned)((k + 127) / 128), 128, 0, ctx->stream>>>(Y, k, n, out);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

void scale_cols(Ctx* ctx, cplx* X, int64_t m, int64_t k, const double* s, int invert) {
    if (m <= 0 || k <= 0) return;
    scale_cols_kernel<<<grid_for(ctx, m * k), 256, 0, ctx->stream>>>(X, m, k, s, invert);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

void scale_rows(Ctx* ctx, cplx* X, int64_t k, int64_t n, const double* s, int invert) {
    if (n <= 0 || k <= 0) return;
    scale_rows_kernel<<<grid_for(ctx, n * k), 256, 0, ctx->stream>>>(X, k, n, s, invert);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

KeepResult keep_rule(Ctx* ctx, const double* dlam, int64_t n, int64_t sz, double cutoff,
                     int64_t maxdim, int64_t mindim, double* dS, const cplx* G, int64_t g,
                     const int* dinfo) {
    TN_REQUIRE(sz <= n, "keep_rule: more singular values than eigenvalues");
    // the result goes to host memory (a copy of its own takes 5 us)
    static_assert(sizeof(KeepDev) == 4 * sizeof(double), "four words");
    double* h = ctx->pinned(4);
    KeepDev* dres = reinterpret_cast<KeepDev*>(h);
    unset(h, 4);
    // the trace is summed by a thread an entry where its last bit counts
    const unsigned threads = one_block(ctx->ordered ? std::max(sz, g) : sz);
    keep_rule_kernel<<<1, threads, 0, ctx->stream>>>(dlam, n, sz, cutoff, maxdim, mindim, dS, G, g,
                                                  dinfo, dres);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
    ctx->sync();
    check_set(h, 4);
    KeepDev r;
    memcpy(&r, h, sizeof(KeepDev));
    if (r.err != 0) {
        TN_CHECK_CUDA(cudaMemsetAsync(const_cast<int*>(dinfo), 0, sizeof(int), ctx->stream));
        throw Error(TN_ERR_TIMEOUT, "eigensolver: a bounded barrier ran out");
    }
    return KeepResult{r.k, r.total, r.discarded};
}

}  // namespace tn
