// FP64 eigensolver of small Gram matrices (order up to 64): Householder
// tridiagonalisation, bisection, inverse iteration, QR of the vectors,
// back-transformation, every sum in one fixed order.
//
// A DMRG cut at a discarded weight of 1e-10 can pass between a pair of
// Schmidt vectors whose weights differ by less than FP64 resolves in the Gram matrix.
// Which combination is kept then follows the last bit of all arithmetic before it, and
// where the state is still far from converged (a domain wall in the ordered Ising
// chain, after two sweeps from a random state: 16 of 200 starts) energies and
// observables differ in the ninth digit or earlier between two solvers that are both
// right to rounding.  So that a run gives what it gave before eig.cu's solver came,
// FP64 DMRG's splits up to order 64, and the gauge moves without truncation up to
// order 16 that its start states come from, keep this solver and its order of operations;
// the Lanczos step and products of short sums keep theirs too (Ctx::ordered).
// Everything else takes eig.cu, which is closer to the exact vectors and faster.
//
// Four launches: the matrix to both triangles, the reduction by one cluster of
// n / 8 blocks (a cluster barrier a step, where a cooperative grid's took 1.9 us),
// eigenvalues to QR by one block, a warp per vector for the rest.
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "eig_dev.cuh"
#include "grid_dev.cuh"

namespace tn {

namespace {

using namespace eigdev;

constexpr int T = 256;  // threads of a block; the order of the sums depends on it
constexpr int MAXN = EIG_FP64_MAX;
constexpr int BIS_W = 4;  // lanes per eigenvalue in the bisection

__device__ __forceinline__ double block_sum(double v, double* ws) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
    __syncthreads();
    if (lane == 0) ws[w] = v;
    __syncthreads();
    double t = lane < nw ? ws[lane] : 0.0;
    t = warp_sum(t);
    return __shfl_sync(0xffffffffu, t, 0);
}


__device__ __forceinline__ void qr_form_column(int64_t w, int lane, const double* __restrict__ Zr,
                                               int64_t t, int64_t k,
                                               const double* __restrict__ qtau,
                                               const double* __restrict__ rdiag,
                                               double* __restrict__ Q) {
    const int64_t c = k - 1 - w;  // column c costs c+1 reflectors: the heaviest start first
    double* q = Q + c * t;
    for (int64_t i = lane; i < t; i += 32) q[i] = (i == c) ? 1.0 : 0.0;
    __syncwarp();
    for (int64_t j = c; j >= 0; --j) {
        const double tau = qtau[j];
        if (tau == 0.0) continue;
        const double* v = Zr + j * t;  // v[j] = 1 implicit
        double s0 = (lane == 0) ? q[j] : 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        int64_t i = j + 1 + lane;
        for (; i + 96 < t; i += 128) {
            s0 = fma(v[i], q[i], s0);
            s1 = fma(v[i + 32], q[i + 32], s1);
            s2 = fma(v[i + 64], q[i + 64], s2);
            s3 = fma(v[i + 96], q[i + 96], s3);
        }
        for (; i < t; i += 32) s0 = fma(v[i], q[i], s0);
        double s = warp_sum((s0 + s1) + (s2 + s3));
        s = __shfl_sync(0xffffffffu, s, 0) * tau;
        for (int64_t i = j + lane; i < t; i += 32) q[i] -= s * (i == j ? 1.0 : v[i]);
        __syncwarp();
    }
    // R's diagonal carries the sign that maps the input column onto Q's column
    if (rdiag[c] < 0.0)
        for (int64_t i = lane; i < t; i += 32) q[i] = -q[i];

}


__device__ __forceinline__ void wy_group(int64_t q, int lane, const cplx* __restrict__ A, int64_t n,
                                         const cplx* __restrict__ tau,
                                         cplx* __restrict__ Tg) {
    const int64_t a = q * BT_G;
    const int nr = (int)min((int64_t)BT_G, (n - 1) - a);
    // S[c][r] = v_c^H v_r for c < r
    double sre[BT_G][BT_G], sim[BT_G][BT_G];
#pragma unroll
    for (int c = 0; c < BT_G; ++c)
#pragma unroll
        for (int r = 0; r < BT_G; ++r) sre[c][r] = sim[c][r] = 0.0;
    for (int64_t i = a + 1 + lane; i < n; i += 32) {
        cplx v[BT_G];
#pragma unroll
        for (int r = 0; r < BT_G; ++r) v[r] = r < nr ? refl(A, n, a + r, i) : cmk(0, 0);
#pragma unroll
        for (int c = 0; c < BT_G; ++c)
#pragma unroll
            for (int r = c + 1; r < BT_G; ++r) {
                sre[c][r] = fma(v[c].x, v[r].x, fma(v[c].y, v[r].y, sre[c][r]));
                sim[c][r] = fma(v[c].x, v[r].y, fma(-v[c].y, v[r].x, sim[c][r]));
            }
    }
#pragma unroll
    for (int c = 0; c < BT_G; ++c)
#pragma unroll
        for (int r = c + 1; r < BT_G; ++r) {
            sre[c][r] = warp_sum(sre[c][r]);
            sim[c][r] = warp_sum(sim[c][r]);
        }
    if (lane != 0) return;
    cplx T[BT_G][BT_G];
#pragma unroll
    for (int c = 0; c < BT_G; ++c)
#pragma unroll
        for (int r = 0; r < BT_G; ++r) T[c][r] = cmk(0, 0);
    for (int r = 0; r < nr; ++r) {
        const cplx tr = tau[a + r];
        T[r][r] = tr;
        cplx z[BT_G];
        for (int c = 0; c < r; ++c) z[c] = cmul(cmk(-tr.x, -tr.y), cmk(sre[c][r], sim[c][r]));
        for (int c = 0; c < r; ++c) {  // T[0:r, r] = T[0:r, 0:r] z
            cplx acc = cmk(0, 0);
            for (int u = c; u < r; ++u) acc = cfma(T[c][u], z[u], acc);
            T[c][r] = acc;
        }
    }
    for (int c = 0; c < BT_G; ++c)
        for (int r = 0; r < BT_G; ++r) Tg[q * BT_G * BT_G + c + BT_G * r] = T[c][r];

}


__device__ __forceinline__ void bt_column(int64_t c, int lane, const cplx* __restrict__ A, int64_t n,
                                          const cplx* __restrict__ Tg, int64_t ngroups,
                                          const double* __restrict__ Z,
                                          cplx* __restrict__ X) {
    cplx* x = X + c * n;
    const double* z = Z + c * n;
    for (int64_t i = lane; i < n; i += 32) x[i] = cmk(z[i], 0.0);
    __syncwarp();
    for (int64_t q = ngroups - 1; q >= 0; --q) {
        const int64_t a = q * BT_G;
        const int nr = (int)min((int64_t)BT_G, (n - 1) - a);
        double sr[BT_G], si[BT_G];
#pragma unroll
        for (int r = 0; r < BT_G; ++r) sr[r] = si[r] = 0.0;
        for (int64_t i = a + 1 + lane; i < n; i += 32) {
            const cplx xi = x[i];
#pragma unroll
            for (int r = 0; r < BT_G; ++r) {
                if (r < nr) {
                    const cplx v = refl(A, n, a + r, i);  // conj(v) x as two FMA chains
                    sr[r] = fma(v.x, xi.x, fma(v.y, xi.y, sr[r]));
                    si[r] = fma(v.x, xi.y, fma(-v.y, xi.x, si[r]));
                }
            }
        }
#pragma unroll
        for (int r = 0; r < BT_G; ++r) {
            sr[r] = __shfl_sync(0xffffffffu, warp_sum(sr[r]), 0);
            si[r] = __shfl_sync(0xffffffffu, warp_sum(si[r]), 0);
        }
        // coefficients u = T s
        const cplx* T = Tg + q * BT_G * BT_G;
        cplx u[BT_G];
#pragma unroll
        for (int r = 0; r < BT_G; ++r) {
            cplx acc = cmk(0, 0);
#pragma unroll
            for (int v = r; v < BT_G; ++v) acc = cfma(T[r + BT_G * v], cmk(sr[v], si[v]), acc);
            u[r] = acc;
        }
        for (int64_t i = a + 1 + lane; i < n; i += 32) {
            cplx xi = x[i];
#pragma unroll
            for (int r = 0; r < BT_G; ++r)
                if (r < nr) {  // x -= u v, fused
                    const cplx v = refl(A, n, a + r, i);
                    xi.x = fma(-u[r].x, v.x, fma(u[r].y, v.y, xi.x));
                    xi.y = fma(-u[r].x, v.y, fma(-u[r].y, v.x, xi.y));
                }
            x[i] = xi;
        }
        __syncwarp();
    }

}


// both triangles of G, with a real diagonal, to A
__global__ void __launch_bounds__(T) hermitian_kernel(const cplx* __restrict__ G, int n, cplx* __restrict__ A) {
    for (int t = blockIdx.x * T + threadIdx.x; t < n * n; t += gridDim.x * T) {
        const int i = t % n, l = t / n;
        A[t] = i > l ? G[t] : i < l ? cconj(G[l + n * i]) : cmk(G[t].x, 0.0);
    }
}

struct Args {
    cplx* A;  // n x n; reflector j in A[j+2:, j] on exit
    int n, want;
    double *d, *e;       // the tridiagonal
    cplx *tau, *y;       // reflectors' scalars (H_j = I - tau_j v_j v_j^H, v_j[j+1] = 1); a step's product
    cplx* dpart;         // blocks' shares of y^H v
    double *bounds, *shift, *qtau, *rdiag, *lam_desc, *lam_asc, *e2;
    float *d32, *e2f;
    double *f1, *f2, *f3, *fl, *zw;  // inverse iteration, n x want
    unsigned char* piv;
    double *Z, *Q;       // n x want
    cplx* Tw;            // compact-WY factors
    cplx* X;             // n x want
};

// Rows of the unreduced block are split over the cluster's blocks; one pass applies the
// last step's rank-2 update and sums this step's product; every block forms the
// reflector and the next column itself.
__global__ void __launch_bounds__(T) reduce_kernel(Args p) {
    __shared__ cplx sv[3][MAXN], red[T];
    __shared__ double ws[32];
    __shared__ cplx s_c[2];
    cplx *vp = sv[0], *wp = sv[1], *vc = sv[2];  // v, w of the step before; v of this one
    const int n = p.n, tid = threadIdx.x, B = gridDim.x, b = blockIdx.x;
    bool pend = false;
    double nrm2 = 0.0;
    for (int i = tid; i < n; i += T) {
        const cplx a = __ldcg(p.A + i);
        vc[i] = a;
        if (i >= 2) nrm2 += a.x * a.x + a.y * a.y;
    }
    nrm2 = block_sum(nrm2, ws);
    for (int j = 0; j + 1 < n; ++j) {
        if (tid == 0) {  // H^H x = beta e_1, beta real
            const cplx al = vc[j + 1];
            cplx tau = cmk(0, 0), scale = cmk(0, 0);
            double beta = al.x;
            if (nrm2 != 0.0 || al.y != 0.0) {
                beta = -copysign(sqrt(al.x * al.x + al.y * al.y + nrm2), al.x);
                const double rb = 1.0 / beta;
                tau = cmk((beta - al.x) * rb, -al.y * rb);
                const double ur = al.x - beta, ui = al.y, rd = 1.0 / (ur * ur + ui * ui);
                scale = cmk(ur * rd, -ui * rd);
            }
            s_c[0] = tau;
            s_c[1] = scale;
            if (b == 0) {
                p.d[j] = vc[j].x;
                p.e[j] = beta;
                p.tau[j] = tau;
            }
        }
        __syncthreads();
        const cplx tau = s_c[0], scale = s_c[1];
        for (int i = j + 2 + tid; i < n; i += T) vc[i] = cmul(vc[i], scale);
        if (tid == 0) vc[j + 1] = cmk(1, 0);
        __syncthreads();
        const int m = n - j - 1, c = (m + B - 1) / B;
        const int r0 = j + 1 + b * c, r1 = min(r0 + c, n);
        double dre = 0.0, dim = 0.0;
        if (r0 < r1) {
            const int cr = r1 - r0, cs = T / cr;  // rows, threads to a row
            double ar = 0.0, ai = 0.0;
            if (tid < cs * cr) {
                const int i = r0 + tid % cr;
                const cplx vpi = pend ? vp[i] : cmk(0, 0), wpi = pend ? wp[i] : cmk(0, 0);
                for (int l = j + 1 + tid / cr; l < n; l += cs) {
                    cplx a = __ldcg(p.A + i + n * l);
                    if (pend) {  // a -= w_i conj(v_l) + v_i conj(w_l)
                        const cplx vl = vp[l], wl = wp[l];
                        a.x = fma(-wpi.x, vl.x, fma(-wpi.y, vl.y, fma(-vpi.x, wl.x, fma(-vpi.y, wl.y, a.x))));
                        a.y = fma(-wpi.y, vl.x, fma(wpi.x, vl.y, fma(-vpi.y, wl.x, fma(vpi.x, wl.y, a.y))));
                        p.A[i + n * l] = a;
                    }
                    const cplx x = vc[l];
                    ar = fma(a.x, x.x, fma(-a.y, x.y, ar));
                    ai = fma(a.x, x.y, fma(a.y, x.x, ai));
                }
            }
            red[tid] = cmk(ar, ai);
            __syncthreads();
            int span = 1;
            while (span < cs) span <<= 1;
            for (int h = span >> 1; h > 0; h >>= 1) {
                if (tid < h * cr && tid + h * cr < cs * cr) red[tid] = cadd(red[tid], red[tid + h * cr]);
                __syncthreads();
            }
            if (tid < cr) {
                const cplx yi = cmul(tau, red[tid]);
                p.y[r0 + tid] = yi;
                const cplx t = cmul(cconj(yi), vc[r0 + tid]);  // y^H v
                dre = t.x;
                dim = t.y;
            }
        }
        dre = block_sum(dre, ws);
        dim = block_sum(dim, ws);
        if (tid == 0) p.dpart[b] = cmk(dre, dim);
        __threadfence();  // results pass between blocks through L2
        __syncwarp();
        griddev::cluster_sync();
        const cplx q = tid < B ? __ldcg(p.dpart + tid) : cmk(0, 0);
        const int i = j + 1 + tid;  // n <= T: a thread has one entry of the vectors
        cplx yv = cmk(0, 0), cv = cmk(0, 0);
        if (i < n) {
            yv = __ldcg(p.y + i);
            cv = __ldcg(p.A + i + n * (j + 1));
        }
        // w = y - (tau/2) (y^H v) v, the same in every block
        const double sre = block_sum(q.x, ws), sim = block_sum(q.y, ws);
        const cplx al2 = cmul(cmk(-0.5 * tau.x, -0.5 * tau.y), cmk(sre, sim));
        if (i < n) {
            yv = cfma(al2, vc[i], yv);
            wp[i] = yv;
        }
        if (b == 0)
            for (int t = j + 2 + tid; t < n; t += T) p.A[t + n * j] = vc[t];
        cplx* t = vp;
        vp = vc;
        vc = t;
        pend = true;
        __syncthreads();
        // column j+1 with this step's update
        const cplx wj1 = wp[j + 1];
        nrm2 = 0.0;
        if (i < n) {
            const cplx vi = vp[i];
            cplx a = cv;
            a.x -= yv.x + (vi.x * wj1.x + vi.y * wj1.y);
            a.y -= yv.y + (vi.y * wj1.x - vi.x * wj1.y);
            vc[i] = a;
            if (i >= j + 3) nrm2 += a.x * a.x + a.y * a.y;
        }
        nrm2 = block_sum(nrm2, ws);
        // no block overwrites y, dpart or rows that another still reads
        __syncwarp();
        griddev::cluster_sync();
    }
    if (b == 0 && tid == 0) p.d[n - 1] = vc[n - 1].x;
}

// Eigenvalues by bisection (four lanes each), vectors by inverse iteration (a thread
// each), their Householder QR in descending order (a warp per column), so that
// multiplets come out orthonormal; and the compact-WY factors of the reduction.
__global__ void __launch_bounds__(T) vectors_kernel(Args p) {
    __shared__ double a0[T], a1[T], a2[T], sq[MAXN], ws[32];
    __shared__ double s_tau, s_scale;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, t = p.n, k = p.want;
    tri_bounds_block(p.d, p.e, t, p.bounds, p.d32, p.e2f, p.e2, a0, a1, a2);
    __syncthreads();
    if (tid / BIS_W < k)
        bisect_group_w<BIS_W>(tid / BIS_W, tid % BIS_W, 0xFu << (lane & ~(BIS_W - 1)), p.d, p.e2, p.d32, p.e2f, t, k,
                              p.bounds, p.lam_desc, p.lam_asc);
    __syncthreads();
    if (tid == 0) separate_shifts_serial(p.lam_desc, k, p.bounds, p.shift);
    __syncthreads();
    const int groups = (t - 1 + BT_G - 1) / BT_G;
    if (tid < k)
        stein_vector(tid, p.d, p.e, t, k, p.shift, p.bounds, p.f1, p.f2, p.f3, p.fl, p.piv, p.zw, p.Z);
    else if (warp >= 2)
        for (int q = warp - 2; q < groups; q += T / 32 - 2) wy_group(q, lane, p.A, t, p.tau, p.Tw);
    __syncthreads();
    if (k == 1) {
        for (int i = tid; i < t; i += T) p.Q[i] = p.Z[i];
        return;
    }
    for (int j = 0; j < k; ++j) {
        const double* zj = p.Z + j * t;
        double nrm2 = 0.0;
        for (int i = j + tid; i < t; i += T) {
            const double v = zj[i];
            sq[i] = v;
            if (i > j) nrm2 += v * v;
        }
        nrm2 = block_sum(nrm2, ws);
        if (tid == 0) {
            const double al = sq[j];
            double tau = 0.0, beta = al, scale = 0.0;
            if (nrm2 != 0.0) {
                beta = -copysign(sqrt(al * al + nrm2), al);
                tau = (beta - al) / beta;
                scale = 1.0 / (al - beta);
            }
            s_tau = tau;
            s_scale = scale;
            sq[j] = 1.0;
            p.qtau[j] = tau;
            p.rdiag[j] = beta;
        }
        __syncthreads();
        const double scale = s_scale, tau = s_tau;
        for (int i = j + 1 + tid; i < t; i += T) sq[i] *= scale;
        __syncthreads();
        for (int i = j + 1 + tid; i < t; i += T) p.Z[i + j * t] = sq[i];
        if (tau != 0.0)
            for (int c = j + 1 + warp; c < k; c += T / 32) {
                double* zc = p.Z + c * t;
                double s0 = 0.0;
                for (int i = j + lane; i < t; i += 32) s0 = fma(sq[i], zc[i], s0);
                double s = warp_sum(s0);
                s = __shfl_sync(0xffffffffu, s, 0) * tau;
                for (int i = j + lane; i < t; i += 32) zc[i] -= s * sq[i];
            }
        __syncthreads();
    }
}

// Column of the QR's orthonormal factor, then of X = H_0 .. H_{n-2} Q, by one warp.
__global__ void __launch_bounds__(32) transform_kernel(Args p) {
    if (p.want > 1) qr_form_column(blockIdx.x, threadIdx.x, p.Z, p.n, p.want, p.qtau, p.rdiag, p.Q);
    const int c = p.want > 1 ? p.want - 1 - blockIdx.x : 0;
    __syncwarp();
    bt_column(c, threadIdx.x, p.A, p.n, p.Tw, (p.n - 1 + BT_G - 1) / BT_G, p.Q, p.X);
}

}  // namespace

void eig_top_fp64(Ctx* ctx, const cplx* G, int64_t n, int64_t want, double* lam_asc, cplx* X) {
    TN_REQUIRE(n >= 1 && n <= MAXN && want >= 1 && want <= n, "eig_top_fp64: bad sizes");
    ProfScope ps(ctx, 2, 16.0 / 3.0 * n * n * n + 8.0 * n * n * want, 16.0 * n * n);
    TN_CHECK_CUDA(cudaMemsetAsync(ctx->d_bar, 0, 3 * sizeof(unsigned), ctx->stream));
    if (n == 1) {
        TN_CHECK_CUDA(cudaMemcpyAsync(lam_asc, G, sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream));
        zfill(ctx, X, 1, cmk(1, 0));
        return;
    }
    const size_t N = (size_t)n, nw = N * (size_t)want;
    const size_t bytes = sizeof(cplx) * (N * N + 2 * N + 8 + (N / BT_G + 1) * BT_G * BT_G) +
                         sizeof(double) * (3 * N + 8 + 4 * (size_t)want + 7 * nw) + sizeof(float) * 2 * N + nw;
    char* base = static_cast<char*>(ctx->s_eig.get(ctx, bytes));
    auto take = [&](auto*& q, size_t count) {
        q = reinterpret_cast<std::remove_reference_t<decltype(q)>>(base);
        base += sizeof(*q) * count;
    };
    Args a{};
    a.n = (int)n;
    a.want = (int)want;
    a.lam_asc = lam_asc;
    a.X = X;
    take(a.A, N * N);
    take(a.tau, N);
    take(a.y, N);
    take(a.dpart, 8);
    take(a.Tw, (N / BT_G + 1) * BT_G * BT_G);
    take(a.d, N);
    take(a.e, N);
    take(a.e2, N);
    take(a.bounds, 8);
    for (double** q : {&a.shift, &a.qtau, &a.rdiag, &a.lam_desc}) take(*q, want);
    for (double** q : {&a.Z, &a.Q, &a.f1, &a.f2, &a.f3, &a.fl, &a.zw}) take(*q, nw);
    take(a.d32, N);
    take(a.e2f, N);
    take(a.piv, nw);
    hermitian_kernel<<<(unsigned)((n * n + T - 1) / T), T, 0, ctx->stream>>>(G, (int)n, a.A);
    ctx->count();
    // one block to 8 rows: the split that the order of the sums rests on
    const unsigned B = (unsigned)std::max<int64_t>(1, n / 8);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = B;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3(B);
    cfg.blockDim = dim3(T);
    cfg.stream = ctx->stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    TN_CHECK_CUDA(cudaLaunchKernelEx(&cfg, reduce_kernel, a));
    ctx->count();
    vectors_kernel<<<1, T, 0, ctx->stream>>>(a);
    ctx->count();
    transform_kernel<<<(unsigned)want, 32, 0, ctx->stream>>>(a);
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

}  // namespace tn
