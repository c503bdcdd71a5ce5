// Hermitian eigensolver of the truncated split, FP64 accurate, on the device.
//
// The reference's svd(x, idx; cutoff, maxdim, mindim) (src/tensors.jl:168-227)
// calls LAPACK gesdd on the grouped tensor.  This library forms the Gram
// matrix of the isometric side instead and needs its top eigenpairs:
//
//   1. Householder reduction G = Q T Q^H to a real symmetric tridiagonal T, in
//      fixed point (hetrd.cu).
//   2. Divide and conquer on T (dc.cu): eigenvalues and orthonormal vectors Z.
//   3. Back-transformation X = Q Z by the reflectors of step 1, panels of them
//      as two matrix products around a triangular solve.
//
// GB300 issues FP64 at two FMAs per clock per SM and each FP64 instruction of a
// warp takes 64 clocks, so serial recurrences and reductions cost most; steps 1
// and 2 say how each avoids them.  Order 16 with 8 vectors takes 0.15 ms, 64 with 32
// 0.43, 128 with 64 0.86, 256 with 128 2.3 (reduction 1.8), 512 with 256 5.1 (4.2).
// Small splits of FP64 DMRG keep another solver, for their values (eig_fp64.cu).
#include <cmath>

#include "common.cuh"

namespace tn {

namespace {

constexpr int64_t EIG_MAXN = 4096;  // step 1 keeps three vectors in shared memory

// ---- 3. back-transformation ----------------------------------------------------
// X = H_0 ... H_{n-2} [Z], panels of reflectors from the last: a panel's product
// is I - V T V^H with T^-1 = the strict upper triangle of V^H V plus diag(1/tau)
// (LAPACK zlarft's T), so a panel is a product W = V^H X, the triangular solve
// Y = T W and the product X -= V Y.

// perm is clamped wherever it is read, for it is not set after a reduction that a
// barrier ended
__device__ __forceinline__ int64_t clamped(int p, int64_t n) { return min((unsigned)p, (unsigned)n - 1u); }

// X[perm[l], :] = Y[l, :]
__global__ void bt_perm_kernel(const cplx* __restrict__ Y, const int* __restrict__ perm, int64_t n, int64_t total,
                               cplx* __restrict__ X) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x)
        X[i / n * n + clamped(perm[i % n], n)] = Y[i];
}

// X (n x k) = Z (real); zeros above the reflectors in V (n x n)
__global__ void bt_init_kernel(const double* __restrict__ Z, int64_t total, cplx* __restrict__ X, int64_t n,
                               cplx* __restrict__ V) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < max(total, n * n);
         i += (int64_t)gridDim.x * blockDim.x) {
        if (i < total) X[i] = cmk(Z[i], 0.0);
        if (i < n * n && i % n <= i / n) V[i] = cmk(0, 0);
    }
}

// Small orders: all reflectors on one column by one warp, E entries a lane, and the
// rows' order undone: 20 FP64 instructions a reflector, one after the other (order 16:
// 12 us, 32: 20, 64: 65), where the panel takes eight launches (40 us at order 32, 66
// at 64).
template <int E>
__global__ void __launch_bounds__(32) bt_small_kernel(const double* __restrict__ Z, const cplx* __restrict__ V,
                                                      const cplx* __restrict__ tau, const int* __restrict__ perm,
                                                      int n, cplx* __restrict__ X) {
    const int lane = threadIdx.x;
    const int64_t c = blockIdx.x;
    cplx x[E], v[E], nv[E];
    auto load = [&](int j, cplx* w) {
#pragma unroll
        for (int t = 0; t < E; ++t) {
            const int i = lane + 32 * t;
            w[t] = j >= 0 && i > j && i < n ? V[i + (int64_t)n * j] : cmk(0, 0);
        }
    };
#pragma unroll
    for (int t = 0; t < E; ++t) x[t] = lane + 32 * t < n ? cmk(Z[lane + 32 * t + n * c], 0.0) : cmk(0, 0);
    load(n - 2, v);
    cplx ta = tau[n - 2];
    for (int j = n - 2; j >= 0; --j) {
        load(j - 1, nv);
        const cplx nt = j > 0 ? tau[j - 1] : cmk(0, 0);
        cplx s = cmk(0, 0);
#pragma unroll
        for (int t = 0; t < E; ++t) s = cfma(cconj(v[t]), x[t], s);
        // real parts to the lower half of the warp, imaginary ones to the upper
        const bool up = lane & 16;
        double r = (up ? s.y : s.x) + __shfl_xor_sync(0xffffffffu, up ? s.x : s.y, 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        const double q = __shfl_xor_sync(0xffffffffu, r, 16);
        const cplx y = cmul(ta, up ? cmk(q, r) : cmk(r, q));
#pragma unroll
        for (int t = 0; t < E; ++t) x[t] = cfma(cmk(-y.x, -y.y), v[t], x[t]);
#pragma unroll
        for (int t = 0; t < E; ++t) v[t] = nv[t];
        ta = nt;
    }
#pragma unroll
    for (int t = 0; t < E; ++t) {
        const int i = lane + 32 * t;
        if (i < n) X[(perm ? clamped(perm[i], n) : i) + n * c] = x[t];
    }
}
constexpr int64_t BT_SMALL = 48;

// Strict upper triangle of V^H V times diag(tau), from the lower triangle of S:
// U[i + nr r] = conj(S[r + nr i]) tau_r.
__global__ void bt_scale_kernel(const cplx* __restrict__ S, int nr, const cplx* __restrict__ tau,
                                cplx* __restrict__ U) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nr * nr; t += gridDim.x * blockDim.x) {
        const int i = t % nr, r = t / nr;
        if (i < r) U[t] = cmul(cconj(S[r + (int64_t)nr * i]), tau[r]);
    }
}

// W[:, c] <- T W[:, c], one block per column and a thread per reflector: back
// substitution, row r = nr-1 .. 1 broadcast through shared memory.  A step is
// four FP64 instructions of the row's warps (256 clocks) and a barrier.
__global__ void bt_solve_kernel(const cplx* __restrict__ U, int nr, const cplx* __restrict__ tau,
                                int64_t k, cplx* __restrict__ W) {
    __shared__ cplx sw[2];
    const int i = threadIdx.x;
    for (int64_t c = blockIdx.x; c < k; c += gridDim.x) {
        cplx* wc = W + c * nr;
        cplx w = i < nr ? wc[i] : cmk(0, 0);
        if (i == nr - 1) sw[(nr - 1) & 1] = w;
        cplx f = i < nr - 1 ? U[i + (int64_t)nr * (nr - 1)] : cmk(0, 0);
        for (int r = nr - 1; r > 0; --r) {
            const cplx fn = i < r - 1 ? U[i + (int64_t)nr * (r - 1)] : cmk(0, 0);  // next step's
            __syncthreads();
            if (i < r) {
                const cplx y = sw[r & 1];
                w.x = fma(-f.x, y.x, fma(f.y, y.y, w.x));
                w.y = fma(-f.x, y.y, fma(-f.y, y.x, w.y));
                if (i == r - 1) sw[(r - 1) & 1] = w;
            }
            f = fn;
        }
        if (i < nr) wc[i] = cmul(tau[i], w);
        __syncthreads();
    }
}

constexpr int64_t BT_MAXNB = 128;

inline unsigned nblk(int64_t n, int threads) { return (unsigned)std::max<int64_t>(1, (n + threads - 1) / threads); }

}  // namespace

// Top `want` eigenpairs of the Hermitian n x n matrix G (lower triangle
// read).  lam_asc[want-1-g] and X[:, g] (n x want,
// column-major) hold the g-th largest eigenvalue and its eigenvector.
// Everything runs on the context's stream without host synchronisation; a
// barrier that timed out leaves a nonzero word at ctx->d_bar[2],
// which the caller reads with its next synchronisation (keep_rule's dinfo).
void eig_top(Ctx* ctx, const cplx* G, int64_t n, int64_t want, double* lam_asc, cplx* X, bool psd) {
    TN_REQUIRE(n >= 1 && want >= 1 && want <= n, "eig_top: bad sizes");
    TN_REQUIRE(n <= EIG_MAXN, "eig_top: matrix order above 4096");
    ProfScope ps(ctx, 2, 16.0 / 3.0 * n * n * n + 8.0 * n * n * want, 16.0 * n * n);
    const bool small = n <= BT_SMALL;
    // scratch: d, e, tau, perm, Z, V, X
    const size_t n8 = (sizeof(double) * n + 255) / 256 * 256;
    const size_t nz = (sizeof(double) * (size_t)n * want + 255) / 256 * 256;
    const size_t nv = (sizeof(cplx) * (size_t)n * n + 255) / 256 * 256;
    char* base = static_cast<char*>(ctx->s_eig.get(ctx, 5 * n8 + nz + nv + (psd && !small ? 2 * nz : 0)));
    double* d = reinterpret_cast<double*>(base);
    double* e = reinterpret_cast<double*>(base + n8);
    cplx* tau = reinterpret_cast<cplx*>(base + 2 * n8);
    int* perm = reinterpret_cast<int*>(base + 4 * n8);
    double* Z = reinterpret_cast<double*>(base + 5 * n8);
    cplx* Vs = reinterpret_cast<cplx*>(base + 5 * n8 + nz);
    cplx* Xout = X;
    if (psd && !small) X = reinterpret_cast<cplx*>(base + 5 * n8 + nz + nv);  // rows in perm's order
    TN_CHECK_CUDA(cudaMemsetAsync(ctx->d_bar, 0, 3 * sizeof(unsigned), ctx->stream));
    if (n == 1) {
        TN_CHECK_CUDA(cudaMemcpyAsync(lam_asc, G, sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream));
        zfill(ctx, Xout, 1, cmk(1, 0));
        return;
    }
    hetrd(ctx, G, n, d, e, tau, Vs, psd, perm);
    tridiag_top(ctx, n, d, e, want, lam_asc, Z);
    if (small) {
        auto k = n <= 32 ? bt_small_kernel<1> : bt_small_kernel<2>;
        k<<<(unsigned)want, 32, 0, ctx->stream>>>(Z, Vs, tau, psd ? perm : nullptr, (int)n, Xout);
        ctx->count();
        TN_CHECK_CUDA(cudaGetLastError());
        return;
    }
    const unsigned nb256 = std::min<unsigned>(nblk(n * n, 256), (unsigned)ctx->sm_count * 8);
    bt_init_kernel<<<nb256, 256, 0, ctx->stream>>>(Z, n * want, X, n, Vs);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
    // Panels of 64 reflectors up to n = 192: their three products and 64 solve
    // steps (10 us) are shortest there; 128 above, where a panel's products cost
    // the same 27 us for twice the reflectors.
    const int64_t nref = n - 1, nb = n <= 192 ? 64 : BT_MAXNB;
    const cplx one = cmk(1, 0), zero = cmk(0, 0);
    cplx* S = ctx->s_bt.c(ctx, (size_t)(2 * nb * nb + nb * want));
    cplx* U = S + nb * nb;
    cplx* W = U + nb * nb;
    for (int64_t p = (nref + nb - 1) / nb - 1; p >= 0; --p) {
        const int64_t a = p * nb, nr = std::min(nb, nref - a), rows = n - 1 - a;
        const cplx* V = Vs + (a + 1) + n * a;  // rows a+1.. of columns a..: zeros above each reflector
        zgemm(ctx, OP_C, OP_N, nr, nr, rows, one, V, n, 0, V, n, 0, zero, S, nr, 0, 1, true);
        zgemm(ctx, OP_C, OP_N, nr, want, rows, one, V, n, 0, X + a + 1, n, 0, zero, W, nr, 0);
        bt_scale_kernel<<<nblk(nr * nr, 256), 256, 0, ctx->stream>>>(S, (int)nr, tau + a, U);
        ctx->count();
        bt_solve_kernel<<<(unsigned)std::min<int64_t>(want, 65535), (unsigned)((nr + 31) / 32 * 32), 0,
                          ctx->stream>>>(U, (int)nr, tau + a, want, W);
        ctx->count();
        TN_CHECK_CUDA(cudaGetLastError());
        zgemm(ctx, OP_N, OP_N, rows, want, nr, cmk(-1, 0), V, n, 0, W, nr, 0, one, X + a + 1, n, 0);
    }
    if (psd) {
        bt_perm_kernel<<<nb256, 256, 0, ctx->stream>>>(X, perm, n, n * want, Xout);
        ctx->count();
        TN_CHECK_CUDA(cudaGetLastError());
    }
}

}  // namespace tn
