// Eigen-decomposition of a real symmetric tridiagonal T by divide and conquer
// (J. J. M. Cuppen, Numer. Math. 36, 1981; eigenvectors by M. Gu and
// S. C. Eisenstat, SIAM J. Matrix Anal. Appl. 16, 1995), steps 2-4 of the
// eigensolver (eig.cu): top `want` eigenvalues and orthonormal eigenvectors.
//
// T is cut into 1 x 1 blocks, T = blockdiag(T1 - rho.., T2 - rho..) + rho v v^T
// at every cut, and neighbouring blocks merge level by level.  A merge of two
// eigensystems (D, Q) is the rank-one problem D + rho z z^T with
// z = Q^T v: its eigenvalues are the roots of 1 / rho + sum z_i^2 / (d_i - x),
// one between each two poles.
//
// Every merge runs the same steps without deflation, so that no step is serial
// in its size: equal poles are moved an ulp apart and entries of z get a floor of
// 2^-56 (both a backward error of rounding size), after which all roots are
// simple.  Roots are kept as an offset from their nearest pole, to full relative
// accuracy, and z is recomputed from them (Loewner's formula), which makes the
// eigenvectors orthogonal to working precision however close the roots lie.
//
// What it replaced is serial in the order: a Sturm count is n steps of four FP64
// instructions of 64 clocks each, an inverse iteration six such sweeps, the QR
// of the vectors n grid barriers; at order 256, 128 vectors: bisection 1,071 us,
// inverse iteration 731, QR and its Q 1,114.  Here a level costs four barriers
// and the whole 250 us at order 64, 350 at 128, 430 at 256.
#include <climits>
#include <cmath>

#include "common.cuh"
#include "grid_dev.cuh"

namespace tn {

namespace {

using namespace griddev;

typedef long long ll;

constexpr int DT = 256;  // threads of a block
constexpr int DW = DT / 32;

struct DcArgs {
    int n, want;
    const double *d, *e;
    double* D;    // n: eigenvalues of the blocks, ascending in each
    double* ds;   // n: poles of a merge, ascending and distinct
    double* z;    // n: z in that order
    double* zh;   // n: recomputed z
    double* mu;   // n: root minus its nearest pole
    int* org;     // n: that pole
    int* idx;     // n: a pole's place in the unsorted merge
    double *Qa, *Qb;   // n x n, block diagonal
    double* Z;         // n x want
    double* lam_asc;   // want
    unsigned* bar;
    int* err;
    int warps2;        // warps of a block with room for a copy of the poles
};

// total order of doubles as signed integers
__device__ __forceinline__ ll okey(double x) {
    const ll b = __double_as_longlong(x);
    return b < 0 ? b ^ 0x7fffffffffffffffll : b;
}
__device__ __forceinline__ double unkey(ll k) {
    return __longlong_as_double(k < 0 ? k ^ 0x7fffffffffffffffll : k);
}
// Monotone map to integers whose unit step is an ulp, or 2^-82 below 2^-30.
constexpr ll B30 = (1023ll - 30) << 52;
__device__ __forceinline__ ll to_grid(double v) {
    const double a = fabs(v);
    const ll k = a < 0x1p-30 ? __double2ll_rn(a * 0x1p82) : (1ll << 52) + __double_as_longlong(a) - B30;
    return v < 0.0 ? -k : k;
}
__device__ __forceinline__ double from_grid(ll k) {
    const ll a = k < 0 ? -k : k;
    const double x = a < (1ll << 52) ? __ll2double_rn(a) * 0x1p-82 : __longlong_as_double(B30 + a - (1ll << 52));
    return k < 0 ? -x : x;
}
__device__ __forceinline__ ll shfl_up64(ll v, int o) {
    return __shfl_up_sync(0xffffffffu, v, o);
}
__device__ __forceinline__ double wsum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float wsumf(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// 1 / x for any normal x: recip() on the mantissa, the exponent by integers
__device__ __forceinline__ double rcp(double x) {
    const int h = __double2hiint(x), ex = (h >> 20) & 0x7ff;
    const double m = __hiloint2double((h & 0x800fffff) | 0x3ff00000, __double2loint(x));
    const double r = recip(m);  // in (1/2, 1]
    const int sh = 1023 - ex;   // exact while the result stays normal
    if (ex == 0 || ex >= 2045) return 1.0 / x;
    return __hiloint2double(__double2hiint(r) + (sh << 20), __double2loint(r));
}

template <bool GRID>
__global__ void __launch_bounds__(DT) dc_kernel(DcArgs p) {
    extern __shared__ __align__(16) unsigned char dsm[];
    __shared__ ll s_scan[DW];
    __shared__ unsigned s_max;
    const int n = p.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int C = (int)gridDim.x, b = (int)blockIdx.x;  // a cluster launch is one cluster
    const int W = C * DW, wid = b * DW + warp;
    unsigned arrivals = 0;
    auto sync = [&]() -> bool {
        if (GRID) {
            arrivals += (unsigned)C;
            return grid_sync(p.bar, p.err, arrivals);
        }
        __threadfence();
        cluster_sync();
        return true;
    };
    // power-of-two scale: |entries of T| < 1
    if (tid == 0) s_max = 0;
    __syncthreads();
    {
        unsigned m = 0;
        for (int i = tid; i < n; i += DT) {
            m = max(m, (unsigned)__double2hiint(p.d[i]) & 0x7fffffffu);
            if (i + 1 < n) m = max(m, (unsigned)__double2hiint(p.e[i]) & 0x7fffffffu);
        }
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) atomicMax(&s_max, m);
    }
    __syncthreads();
    const int ex = min(max((int)(s_max >> 20) - 1022, -900), 900);
    const double down = scalbn(1.0, -ex), up = s_max ? scalbn(1.0, ex) : 0.0;
    const double rho_min = 0x1p-58;
    // 1 x 1 blocks
    for (int i = b * DT + tid; i < n; i += C * DT) {
        double x = p.d[i] * down;
        if (i > 0) x -= fmax(fabs(p.e[i - 1] * down), rho_min);
        if (i + 1 < n) x -= fmax(fabs(p.e[i] * down), rho_min);
        p.D[i] = x;
        p.Qa[i + (size_t)n * i] = 1.0;
    }
    if (!sync()) return;
    double *Q = p.Qa, *Qn = p.Qb;
    for (int h = 1; h < n; h *= 2) {
        const int K0 = 2 * h, nm = (n + K0 - 1) / K0;
        const bool last = K0 >= n;
        // ---- poles of every merge: one block each -----------------------------
        for (int m = b; m < nm; m += C) {
            const int lo = m * K0, mid = lo + h, hi = min(lo + K0, n), K = hi - lo;
            if (mid >= n) continue;  // an unpaired block goes up as it is
            ll* key = reinterpret_cast<ll*>(dsm);
            ll* srt = key + K;
            const double ev = p.e[mid - 1];
            for (int i = tid; i < K; i += DT) key[i] = okey(__ldcg(p.D + lo + i));
            __syncthreads();
            for (int i = tid; i < K; i += DT) {
                const ll k = key[i];
                const int base = i < h ? h : 0;  // the other block; ties: first block first
                int l = 0, r = i < h ? K - h : h;
                while (l < r) {
                    const int c = (l + r) >> 1;
                    const ll o = key[base + c];
                    if (i < h ? o < k : o <= k) l = c + 1;
                    else r = c;
                }
                const int rk = min((i < h ? i : i - h) + l, K - 1);
                srt[rk] = k;
                double z = i < h ? __ldcg(Q + (mid - 1) + (size_t)n * (lo + i))
                                 : copysign(1.0, ev) * __ldcg(Q + mid + (size_t)n * (lo + i));
                if (!(fabs(z) >= 0x1p-56)) z = copysign(0x1p-56, z);
                p.z[lo + rk] = z;
                p.idx[lo + rk] = i;
            }
            __syncthreads();
            // distinct: on a grid of ulps, 2^-82 below 2^-30, pole r at least one
            // step above pole r-1 (a prefix maximum); poles that are distinct
            // already stay
            const int per = (K + DT - 1) / DT, r0 = min(tid * per, K), r1 = min(r0 + per, K);
            ll mx = LLONG_MIN / 2;
            for (int r = r0; r < r1; ++r) mx = max(mx, to_grid(unkey(srt[r])) - r);
            ll inc = mx;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const ll t = shfl_up64(inc, o);
                if (lane >= o) inc = max(inc, t);
            }
            if (lane == 31) s_scan[warp] = inc;
            __syncthreads();
            ll run = shfl_up64(inc, 1);
            if (lane == 0) run = LLONG_MIN / 2;
            for (int w = 0; w < warp; ++w) run = max(run, s_scan[w]);
            for (int r = r0; r < r1; ++r) {
                const double v = unkey(srt[r]);
                const ll k = to_grid(v);
                const double t = k < run + r ? from_grid(run + r) : v;
                p.ds[lo + r] = t;
                run = max(run, k - r);
            }
            __syncthreads();
        }
        if (!sync()) return;
        // ---- roots: a warp each ------------------------------------------------
        if (warp < p.warps2) {
            for (int g = b + C * warp; g < n; g += C * p.warps2) {
                const int lo = g / K0 * K0, mid = lo + h, hi = min(lo + K0, n), K = hi - lo, j = g - lo;
                if (mid >= n) continue;
                float2* pf = reinterpret_cast<float2*>(dsm) + (size_t)warp * K0;
                const double* ds = p.ds + lo;
                const double* zz = p.z + lo;
                const double rinv = rcp(fmax(fabs(p.e[mid - 1] * down), rho_min));
                const float rf = (float)rinv;
                const double dj = __ldcg(ds + j);
                __syncwarp();
                float sz = 0.f;
                for (int i = lane; i < K; i += 32) {
                    const float zf = (float)__ldcg(zz + i);
                    pf[i] = make_float2((float)(__ldcg(ds + i) - dj), zf * zf);
                    sz += zf * zf;
                }
                __syncwarp();
                auto evalf = [&](float x) {
                    float s = 0.f;
                    for (int i = lane; i < K; i += 32) s += __fdividef(pf[i].y, pf[i].x - x);
                    return wsumf(s) + rf;
                };
                // sum of the terms at x = sg m in FP64, its derivative and the terms' moduli
                double f, fp;
                float fa;
                auto eval = [&](double org, double x) {
                    double fl = 0.0, fr = 0.0;  // poles up to j, above j
                    fp = 0.0;
                    for (int i = lane; i < K; i += 32) {
                        const double r = rcp((__ldcg(ds + i) - org) - x), zi = __ldcg(zz + i);
                        const double t = zi * zi * r;
                        if (i <= j) fl += t;
                        else fr += t;
                        fp = fma(t, r, fp);
                    }
                    f = fl + fr;
                    fa = wsumf((float)(fr - fl)) + rf;
#pragma unroll
                    for (int s = 16; s > 0; s >>= 1) {
                        f += __shfl_xor_sync(0xffffffffu, f, s);
                        fp += __shfl_xor_sync(0xffffffffu, fp, s);
                    }
                    f += rinv;
                };
                int o = j;
                // the root lies within half of its origin; where FP32 rounding (a
                // term is good to 2^-20, a sum of K / 32 + 5 likewise) could have
                // the sign at the middle wrong, it is taken in FP64
                double half;
                if (j + 1 < K) {
                    half = 0.5 * (__ldcg(ds + j + 1) - dj);
                    float s = 0.f, sa = 0.f;
                    for (int i = lane; i < K; i += 32) {
                        const float t = __fdividef(pf[i].y, pf[i].x - (float)half);
                        s += t;
                        sa += fabsf(t);
                    }
                    s = wsumf(s) + rf;
                    sa = wsumf(sa) + rf;
                    bool beyond = s < 0.f;
                    if (!(fabsf(s) > (float)(K / 32 + 16) * 0x1p-22f * sa)) {
                        eval(dj, half);
                        beyond = f < 0.0;
                    }
                    if (beyond) {
                        o = j + 1;
                        const double d1 = __ldcg(ds + o);
                        __syncwarp();
                        for (int i = lane; i < K; i += 32) pf[i].x = (float)(__ldcg(ds + i) - d1);
                        __syncwarp();
                    }
                } else {
                    half = (double)(wsumf(sz) * 1.0001f) / rinv;
                }
                const double sg = o == j ? 1.0 : -1.0;
                const double dorg = o == j ? dj : __ldcg(ds + o);
                // FP32: bisection on the bits of |offset| to 2^-15
                unsigned bl = 0x00800000u, bh = __float_as_uint((float)half * 1.001f);
                for (int it = 0; it < 23 && bh > bl + 64u; ++it) {
                    const unsigned bm = bl + (bh - bl) / 2;
                    const float f = evalf((float)sg * __uint_as_float(bm));
                    if ((f < 0.f) == (sg > 0.0)) bl = bm;
                    else bh = bm;
                }
                // FP64: Newton on x f(x), which has no pole at the origin, inside
                // the bracket that the signs give
                double m = (double)__uint_as_float(bl + (bh - bl) / 2), ml = 0.0, mh = half * 1.001;
                m = fmin(m, half);
                double before = 1e300;
                for (int it = 0; it < 48; ++it) {
                    const double x = sg * m;
                    eval(dorg, x);
                    if ((f < 0.0) == (sg > 0.0)) ml = m;
                    else mh = m;
                    const double den = fma(x, fp, f);
                    const double mn = m - m * f * rcp(den);
                    const double st = fabs(mn - m);
                    const bool noise = fabs(f) <= (double)(fa * 0x1p-50f);  // rounding of the sum
                    if ((mn > ml && mn < mh && st <= 0.3 * m) || st <= 0x1p-20 * m) {
                        m = mn;
                        // converged, or as near as rounding of the sum allows
                        if (st <= 0x1p-50 * m || (st >= 0.25 * before && (noise || st <= 0x1p-36 * m))) break;
                        before = st;
                    } else if (noise) {  // the sign says nothing
                        break;
                    } else {  // halve the bracket's exponent
                        const ll a = __double_as_longlong(fmax(ml, m * 0x1p-16));
                        m = __longlong_as_double((a + __double_as_longlong(mh)) / 2);
                        before = 1e300;
                    }
                }
                if (lane == 0) {
                    double lam = fma(sg, m, dorg);
                    if (lam < dj) lam = dj;
                    if (j + 1 < K) lam = fmin(lam, __ldcg(ds + j + 1));
                    p.org[g] = o;
                    p.mu[g] = sg * m;
                    p.D[g] = lam;
                }
            }
        }
        if (!sync()) return;
        // ---- z from the roots ---------------------------------------------------
        for (int g = wid; g < n; g += W) {
            const int lo = g / K0 * K0, mid = lo + h, hi = min(lo + K0, n), K = hi - lo, i = g - lo;
            if (mid >= n) continue;
            const double di = __ldcg(p.ds + g);
            double pr = 1.0;
            for (int j = lane; j < K; j += 32) {
                const int oj = min(max(__ldcg(p.org + lo + j), 0), K - 1);
                const double t = (__ldcg(p.ds + lo + oj) - di) + __ldcg(p.mu + lo + j);  // root j - pole i
                pr *= j == i ? t : t * rcp(__ldcg(p.ds + lo + j) - di);
            }
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) pr *= __shfl_xor_sync(0xffffffffu, pr, s);
            if (lane == 0) p.zh[g] = copysign(sqrt(fabs(pr)), __ldcg(p.z + g));
        }
        if (!sync()) return;
        // ---- eigenvectors: Q blockdiag times the rank-one problem's ---------------
        // A unit is a column and one of wpc shares of its rows; every warp of a
        // column forms the column's coefficients itself.
        const int g0 = last ? n - p.want : 0, cols = n - g0;
        int wpc = 1;
        while (wpc < 16 && 2 * wpc * cols <= C * p.warps2 && 32 * wpc < K0) wpc *= 2;
        for (int unit = b + C * warp; unit < cols * wpc && warp < p.warps2; unit += C * p.warps2) {
            const int g = g0 + unit / wpc, part = unit % wpc;
            const int lo = g / K0 * K0, mid = lo + h, hi = min(lo + K0, n), K = hi - lo;
            double* out = last ? p.Z + (size_t)n * (n - 1 - g) : Qn + (size_t)n * g;
            if (last && part == 0 && lane == 0) p.lam_asc[g - g0] = __ldcg(p.D + g) * up;
            if (mid >= n) {  // unpaired
                for (int r = lo + 32 * part + lane; r < hi; r += 32 * wpc)
                    out[r] = __ldcg(Q + r + (size_t)n * g);
                continue;
            }
            double* u = reinterpret_cast<double*>(dsm) + (size_t)warp * K0;
            const int og = min(max(__ldcg(p.org + g), 0), K - 1);
            const double dorg = __ldcg(p.ds + lo + og), x = __ldcg(p.mu + g);
            double nrm = 0.0;
            __syncwarp();
            for (int i = lane; i < K; i += 32) {
                const double v = __ldcg(p.zh + lo + i) * rcp((__ldcg(p.ds + lo + i) - dorg) - x);
                nrm = fma(v, v, nrm);
                u[min(max(__ldcg(p.idx + lo + i), 0), K - 1)] = v;
            }
            nrm = wsum(nrm);
            const double inv = rsqrt(nrm);
            __syncwarp();
            for (int r = lo + 32 * part + lane; r < hi; r += 32 * wpc) {
                const bool top = r < mid;
                const int i0 = top ? 0 : h, i1 = top ? h : K;
                const double* q = Q + r + (size_t)n * lo;
                double s0 = 0.0, s1 = 0.0;
                int i = i0;
                for (; i + 7 < i1; i += 8) {  // eight loads in flight, two chains
                    double v[8];
#pragma unroll
                    for (int t = 0; t < 8; ++t) v[t] = __ldcg(q + (size_t)n * (i + t));
#pragma unroll
                    for (int t = 0; t < 8; t += 2) {
                        s0 = fma(v[t], u[i + t], s0);
                        s1 = fma(v[t + 1], u[i + t + 1], s1);
                    }
                }
                for (; i < i1; ++i) s0 = fma(__ldcg(q + (size_t)n * i), u[i], s0);
                out[r] = (s0 + s1) * inv;
            }
        }
        if (!last && !sync()) return;
        double* t = Q;
        Q = Qn;
        Qn = t;
    }
    if (!GRID) cluster_sync();
}

constexpr size_t DSMEM = 220 * 1024;
constexpr int DC_CLUSTER = 16;

}  // namespace

// Top `want` eigenpairs of the tridiagonal (d, e) of order n: lam_asc ascending,
// Z (n x want) descending columns.  No host synchronisation; a grid barrier that
// ran out leaves ctx->d_bar[2] nonzero.
void tridiag_top(Ctx* ctx, int64_t n, const double* d, const double* e, int64_t want,
                 double* lam_asc, double* Z) {
    auto r256 = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t n8 = r256(sizeof(double) * n), n4 = r256(sizeof(int) * n),
                 nn = r256(sizeof(double) * (size_t)n * n);
    char* base = static_cast<char*>(ctx->s_dc.get(ctx, 5 * n8 + 2 * n4 + 2 * nn));
    auto take = [&](size_t b) {
        char* q = base;
        base += b;
        return q;
    };
    DcArgs a{};
    a.n = (int)n;
    a.want = (int)want;
    a.d = d;
    a.e = e;
    a.D = reinterpret_cast<double*>(take(n8));
    a.ds = reinterpret_cast<double*>(take(n8));
    a.z = reinterpret_cast<double*>(take(n8));
    a.zh = reinterpret_cast<double*>(take(n8));
    a.mu = reinterpret_cast<double*>(take(n8));
    a.org = reinterpret_cast<int*>(take(n4));
    a.idx = reinterpret_cast<int*>(take(n4));
    a.Qa = reinterpret_cast<double*>(take(nn));
    a.Qb = reinterpret_cast<double*>(take(nn));
    a.Z = Z;
    a.lam_asc = lam_asc;
    a.bar = ctx->d_bar;
    a.err = reinterpret_cast<int*>(ctx->d_bar + 2);
    int64_t K0 = 1;
    while (K0 < n) K0 *= 2;
    // a warp's copy of the poles is 8 bytes an entry, so are its coefficients;
    // the block that sorts a merge needs 16 bytes an entry
    a.warps2 = (int)std::min<int64_t>(DW, (int64_t)(DSMEM / (8 * K0)));
    TN_REQUIRE(a.warps2 >= 2, "tridiag_top: order too large");
    const size_t dyn = (size_t)8 * K0 * a.warps2;
    // One cluster (barrier 0.2 us against 1.2) while its sixteen SMs hold the
    // FP64 work of a level, the whole grid above.
    const bool grid = n > 128 || ctx->trd_clusters == 0;
    if (grid) {
        TN_CHECK_CUDA(cudaMemsetAsync(a.bar, 0, sizeof(unsigned), ctx->stream));
        TN_CHECK_CUDA(cudaFuncSetAttribute(dc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)DSMEM));
        void* args[] = {&a};
        TN_CHECK_CUDA(cudaLaunchCooperativeKernel((void*)dc_kernel<true>, dim3((unsigned)ctx->sm_count),
                                                  dim3(DT), args, dyn, ctx->stream));
    } else {
        // blocks: a warp per root
        const int C = n <= 8 ? 1 : n <= 16 ? 2 : n <= 32 ? 4 : n <= 64 ? 8 : DC_CLUSTER;
        TN_CHECK_CUDA(cudaFuncSetAttribute(dc_kernel<false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = (unsigned)C;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)C);
        cfg.blockDim = dim3(DT);
        cfg.dynamicSmemBytes = dyn;
        cfg.stream = ctx->stream;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        TN_CHECK_CUDA(cudaLaunchKernelEx(&cfg, dc_kernel<false>, a));
    }
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

}  // namespace tn
