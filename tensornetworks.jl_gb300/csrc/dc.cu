// Eigen-decomposition of a real symmetric tridiagonal T by divide and conquer
// (J. J. M. Cuppen, Numer. Math. 36, 1981; eigenvectors by M. Gu and
// S. C. Eisenstat, SIAM J. Matrix Anal. Appl. 16, 1995), steps 2-4 of the
// eigensolver (eig.cu): top `want` eigenvalues and orthonormal eigenvectors.
//
// T is cut into 1 x 1 blocks, T = blockdiag(T1 - rho a^2 .., T2 - rho b^2 ..) +
// rho v v^T at every cut, v = (.., a, b, ..) with rho a b = |e| and b / a about the square
// root of the neighbouring diagonals' ratio, so that what is subtracted from either is
// no larger than it (Gram matrices are graded, and their small eigenvalues' vectors
// have to be right to that scale).  Neighbouring blocks merge level by level.  A merge of two
// eigensystems (D, Q) is the rank-one problem D + rho z z^T with
// z = Q^T v: its eigenvalues are the roots of 1 / rho + sum z_i^2 / (d_i - x),
// one between each two poles.
//
// Every merge runs the same steps without deflation, so that no step is serial
// in its size: equal poles are moved an ulp apart, entries of v^T Q get a floor of 2^-56
// of v's, off-diagonals one of 2^-58 of the neighbouring diagonals' mean (all backward
// errors of rounding size where they act; an absolute floor of 2^-58 mixed pairs of weight
// 1e-10 closer than 4e-8 of it, 2e-8 in the energy of a chain of 30 sites), after
// which all roots are simple.  Roots are kept as an offset from their nearest pole, to full relative
// accuracy, and z is recomputed from them (Loewner's formula), which makes the
// eigenvectors orthogonal to working precision however close the roots lie.
//
// What it replaced is serial in the order: a Sturm count is n steps of four FP64
// instructions of 64 clocks each, an inverse iteration six such sweeps, the QR
// of the vectors n grid barriers; at order 256, 128 vectors: bisection 1,071 us,
// inverse iteration 731, QR and its Q 1,114.  Here all of it takes 69 us at order
// 32, 92 at 64, 153 at 128, 195 at 256.
//
// A level is a chain of FP64 instructions that cost the same for one lane as for
// 32, so a warp finds several roots at once where merges are small (32 / K lanes),
// blocks of eight rows are merged by one warp without barriers, the FP32 start of a
// root is a search in up to 32 sections a round, and Newton stops when the next step
// would change nothing (two evaluations a root).  A warp per root throughout, with
// bisection and a confirming step, took 163 us at order 32, 207 at 64, 272 at 128
// and 313 at 256.
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
    double* rinv; // n: 1 / rho of the merge around a row
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
// Monotone map to integers whose unit step is an ulp, or 2^-112 below 2^-60 (FP32 holds
// its square root's reciprocal and more); in integers, as FP64 conversions cost 64
// clocks each.
constexpr int UEX = 1023 - 60;
constexpr ll UBITS = (ll)UEX << 52;
__device__ __forceinline__ ll to_grid(double v) {
    const ll bits = __double_as_longlong(v), a = bits & LLONG_MAX;
    const int s = UEX - (int)(a >> 52);  // below 2^-60 the mantissa moves down by s
    ll k;
    if (s <= 0) k = (1ll << 52) + a - UBITS;
    else if (s > 53) k = 0;
    else k = (((a & ((1ll << 52) - 1)) | (1ll << 52)) + (1ll << (s - 1))) >> s;
    return bits < 0 ? -k : k;
}
__device__ __forceinline__ double from_grid(ll k) {
    const ll a = k < 0 ? -k : k;
    ll bits;
    if (a >= (1ll << 52)) {
        bits = UBITS + a - (1ll << 52);
    } else if (a == 0) {
        bits = 0;
    } else {
        const int s = __clzll(a) - 11;  // mantissa's leading bit to bit 52
        bits = ((ll)(UEX - s) << 52) + ((a << s) - (1ll << 52));
    }
    return __longlong_as_double(k < 0 ? bits | LLONG_MIN : bits);
}
__device__ __forceinline__ ll shfl_up64(ll v, int o) {
    return __shfl_up_sync(0xffffffffu, v, o);
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

// floor(log2 |x|) of a normal x; zero counts as 2^-1023
__device__ __forceinline__ int expo(double x) { return ((__double2hiint(x) >> 20) & 0x7ff) - 1023; }

// T's off-diagonal e between diagonals d1 and d2 (all below 1) as rho a b
struct Cut {
    double rho, a, b;
};
__device__ __forceinline__ double pow2(int s) { return __hiloint2double((1023 + s) << 20, 0); }
__device__ __forceinline__ Cut cut(double d1, double d2, double e) {
    const int x1 = expo(d1), x2 = expo(d2), hi = max(x1, x2), lo = min(x1, x2);
    // the smaller side's factor 2^s: rho stays at the larger diagonal's size where |e|
    // does, and is |e| where |e| is the largest of the three
    const int s = max(min(max((lo - hi) / 2, expo(e) - hi), 0), -56);
    const double r = scale2(fabs(e), -s), f = pow2(max(hi - 58, -112));
    const double t = pow2(s);
    return Cut{__double_as_longlong(r) > __double_as_longlong(f) ? r : f, x1 < x2 ? t : 1.0, x1 < x2 ? 1.0 : t};
}

// sums over aligned groups of g lanes
__device__ __forceinline__ double gsum(double v, int g) {
    for (int o = g >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float gsumf(float v, int g) {
    for (int o = g >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// FP32 reciprocal, good to an ulp (denormals count as zero)
__device__ __forceinline__ float rcpf(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

constexpr int BASE = 8;  // rows of a base block

// base blocks are merged in shared memory by one warp, the rest through L2
template <bool LOC, class T>
__device__ __forceinline__ T ld(const T* p) {
    return LOC ? *p : __ldcg(p);
}

// A merge: K poles ds (ascending, distinct), z, 1 / rho.  The warp finds 32 / g roots,
// g lanes and K0 entries of pf to a root; this lane's is root j.  EPL elements a
// lane in registers (K0 <= EPL g), or 0: any number, read again for every sum.
// Out: origin pole o and offset of the root from it.
template <int EPL, bool LOC>
__device__ __forceinline__ void find_root(const double* ds, const double* zz, int K, int K0, int g, int j,
                                          double rinv, float2* pf, int& o_out, double& mu_out) {
    const int lane = threadIdx.x & 31, gl = lane & (g - 1);
    const float rf = (float)rinv;
    const double dj = ld<LOC>(ds + j);
    double dr[EPL ? EPL : 1], zr[EPL ? EPL : 1];  // poles, z^2
    if (EPL) {
#pragma unroll
        for (int t = 0; t < EPL; ++t) {
            const int i = gl + g * t;
            dr[t] = i < K ? ld<LOC>(ds + i) : 8.0;  // z = 0 there
            zr[t] = i < K ? ld<LOC>(zz + i) : 0.0;
            if (g * t < K0) zr[t] *= zr[t];
        }
    }
    auto each = [&](auto f) {  // f(i, pole, z^2)
        if (EPL) {
#pragma unroll
            for (int t = 0; t < EPL; ++t)
                if (g * t < K0) f(gl + g * t, dr[t], zr[t]);
        } else {
            for (int i = gl; i < K0; i += g) {
                const double z = i < K ? ld<LOC>(zz + i) : 0.0;
                f(i, i < K ? ld<LOC>(ds + i) : 8.0, z * z);
            }
        }
    };
    // the sum of the terms at org + x in FP64, its derivative and the terms' moduli
    double f, fp;
    float fa;
    auto eval = [&](double org, double x) {
        double fl = 0.0, fr = 0.0;  // poles up to j, above j
        fp = 0.0;
        each([&](int i, double d, double z2) {
            const double r = rcp((d - org) - x);
            const double t = z2 * r;
            if (i <= j) fl += t;
            else fr += t;
            fp = fma(t, r, fp);
        });
        f = fl + fr;
        fa = (float)(fr - fl);
        for (int s = g >> 1; s > 0; s >>= 1) {
            f += __shfl_xor_sync(0xffffffffu, f, s);
            fp += __shfl_xor_sync(0xffffffffu, fp, s);
            fa += __shfl_xor_sync(0xffffffffu, fa, s);
        }
        f += rinv;
        fa += rf;
    };
    auto fill = [&](double org) {
        __syncwarp();
        each([&](int i, double d, double z2) {  // entries from K on count zero
            pf[i] = make_float2((float)(d - org), (float)z2);
        });
        __syncwarp();
    };
    if (LOC)
        for (int i = K0 + gl; i < BASE; i += g) pf[i] = make_float2(8.f, 0.f);
    fill(dj);
    // the root lies within half of its origin; where FP32 rounding (a term is good
    // to 2^-20, a sum of K / g + 5 likewise) could have the sign at the middle
    // wrong, it is taken in FP64
    double half;
    float sz = 0.f, s = 0.f, sa = 0.f;
    const bool lastpole = j + 1 >= K;
    half = lastpole ? 0.0 : 0.5 * (ld<LOC>(ds + j + 1) - dj);
    {
        const float hf = (float)half;
#pragma unroll 4
        for (int i = gl; i < K0; i += g) {
            const float2 q = pf[i];
            const float t = __fdividef(q.y, q.x - hf);
            sz += q.y;
            s += t;
            sa += fabsf(t);
        }
    }
    sz = gsumf(sz, g);
    s = gsumf(s, g) + rf;
    sa = gsumf(sa, g) + rf;
    bool beyond = !lastpole && s < 0.f;
    const bool unsure = !lastpole && !(fabsf(s) > (float)(K / g + 16) * 0x1p-22f * sa);
    if (__any_sync(0xffffffffu, unsure)) {
        eval(dj, half);
        if (unsure) beyond = __double2hiint(f) < 0;
    }
    if (lastpole) half = (double)(sz * 1.0001f) * rcp(rinv);
    const int o = beyond ? j + 1 : j;
    const double sg = beyond ? -1.0 : 1.0;
    const double dorg = beyond ? ld<LOC>(ds + o) : dj;
    if (__any_sync(0xffffffffu, beyond)) fill(dorg);
    // FP32: the bits of |offset| to 2^-17 in sections; a base block's groups of four
    // lanes take four points a lane, larger merges one, by sp lanes where there are
    // many poles
    constexpr int PPL = LOC ? 4 : 1;
    const int lsp = K0 <= 32 ? 0 : K0 <= 64 ? 1 : K0 <= 128 ? 2 : K0 <= 256 ? 3 : 4, sp = 1 << lsp;
    const int ls = LOC ? 4 : 31 - __clz(g) - lsp;  // log2 of the sections
    const int pl = gl & (sp - 1), q0 = (gl >> lsp) * PPL;
    unsigned bl = 0x00800000u, bh = max(__float_as_uint((float)half * 1.001f), bl);
    const unsigned gmask = (g == 32 ? 0xffffffffu : (1u << g) - 1u) << (lane & ~(g - 1));
    for (int it = 0; it < 24; ++it) {
        const bool more = bh > bl + 64u;
        if (!__any_sync(0xffffffffu, more)) break;
        const unsigned step = (bh - bl) >> ls;
        float x[PPL], v[PPL];
#pragma unroll
        for (int r = 0; r < PPL; ++r) {
            x[r] = (float)sg * __uint_as_float(bl + step * (unsigned)(q0 + r));
            v[r] = rf;
        }
        if (LOC) {
#pragma unroll
            for (int i = 0; i < BASE; ++i) {
                const float2 q = pf[i];  // entries from K0 on have z = 0
#pragma unroll
                for (int r = 0; r < PPL; ++r) v[r] += q.y * rcpf(q.x - x[r]);
            }
        } else {
            float w = 0.f;
            v[0] = 0.f;
#pragma unroll 4
            for (int i = pl; i < K0; i += 2 * sp) {  // K0 / sp is even
                const float2 q = pf[i], q2 = pf[i + sp];
                v[0] += q.y * rcpf(q.x - x[0]);
                w += q2.y * rcpf(q2.x - x[0]);
            }
            v[0] += w;
            for (int t = sp >> 1; t > 0; t >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], t);
            v[0] += rf;
        }
        unsigned c = 0;  // points below the root, bl first
#pragma unroll
        for (int r = 0; r < PPL; ++r)
            c += (unsigned)__popc(__ballot_sync(0xffffffffu, q0 + r == 0 || (v[r] < 0.f) == (sg > 0.0)) & gmask);
        c >>= lsp;
        if (more) {
            if (c < (1u << ls)) bh = bl + step * c;
            bl += step * (c - 1);
        }
    }
    // FP64: Newton on x f(x), which has no pole at the origin, inside the bracket
    // that the signs give.  Steps are compared by their exponents relative to m.
    double m = fmin((double)__uint_as_float(bl + (bh - bl) / 2), half), ml = 0.0, mh = half * 1.001;
    int before = -20, jumps = 0;
    bool done = false;
    for (int it = 0; it < 48; ++it) {
        const double x = sg * m;
        eval(dorg, x);
        if (!done) {
            if ((__double2hiint(f) < 0) == (sg > 0.0)) ml = m;
            else mh = m;
            const double mn = fma(-m * f, rcp(fma(x, fp, f)), m);
            const int em = expo(m), st = expo(mn - m) - em;
            const bool noise = expo(f) <= ilogbf(fa) - 51;  // rounding of the sum
            const ll im = __double_as_longlong(mn);
            const bool inside = im > __double_as_longlong(ml) && im < __double_as_longlong(mh);
            // far below m, where FP32 could not follow the root to its pole, the function
            // is a line and one long step gets there
            const bool jump = inside && im < __double_as_longlong(m) && !noise && jumps < 3;
            if ((inside && st <= -3) || st <= -21 || jump) {
                jumps += st > -3;
                m = mn;
                // converged, or the next step would be (its error is the cube of
                // this over the square of the last), or as near as the sum allows
                done = st <= -51 || (before <= -8 && 3 * (st + 1) - 2 * before <= -56) ||
                       (st >= before - 2 && (noise || st <= -37));
                before = st;
            } else if (noise) {  // the sign says nothing
                done = true;
            } else {  // halve the bracket's exponent
                const ll a = __double_as_longlong(fmax(ml, m * 0x1p-16));
                m = __longlong_as_double((a + __double_as_longlong(mh)) / 2);
                before = 0;
            }
        }
        if (__all_sync(0xffffffffu, done)) break;
    }
    o_out = o;
    mu_out = sg * m;
}

// z_i from the roots (Loewner's formula), g lanes to an i
template <bool LOC>
__device__ __forceinline__ double new_z(const double* ds, const double* mu, const int* org, const double* z, int K,
                                        int g, int i) {
    const int gl = threadIdx.x & (g - 1);
    const double di = ld<LOC>(ds + i);
    double pr = 1.0;
    for (int j = gl; j < K; j += g) {
        const int oj = min(max(ld<LOC>(org + j), 0), K - 1);
        const double t = (ld<LOC>(ds + oj) - di) + ld<LOC>(mu + j);  // root j - pole i
        pr *= j == i ? t : t * rcp(ld<LOC>(ds + j) - di);
    }
    for (int s = g >> 1; s > 0; s >>= 1) pr *= __shfl_xor_sync(0xffffffffu, pr, s);
    return copysign(sqrt(fabs(pr)), ld<LOC>(z + i));
}

// Coefficients of an eigenvector in the merge's unsorted basis, to u; its norm's inverse.
template <bool LOC>
__device__ __forceinline__ double coefficients(const double* ds, const double* zh, const int* idx, double dorg,
                                               double x, int K, int g, double* u) {
    const int gl = threadIdx.x & (g - 1);
    double nrm = 0.0;
    for (int i = gl; i < K; i += g) {
        const double v = ld<LOC>(zh + i) * rcp((ld<LOC>(ds + i) - dorg) - x);
        nrm = fma(v, v, nrm);
        u[min(max(ld<LOC>(idx + i), 0), K - 1)] = v;
    }
    return rsqrt(gsum(nrm, g));
}

// a warp's shared memory while it merges a base block
struct BaseMem {
    double D[BASE], ds[BASE], z[BASE], zh[BASE], mu[BASE], Q[2][BASE * BASE];
    ll key[BASE], srt[BASE];
    int org[BASE], idx[BASE];
    double u[BASE][BASE];
    float2 pf[BASE][BASE];
};

template <bool GRID>
__global__ void __launch_bounds__(DT) dc_kernel(DcArgs p) {
    extern __shared__ __align__(16) unsigned char dsm[];
    __shared__ ll s_scan[DW];
    __shared__ unsigned s_max;
    const int n = p.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nt = (int)blockDim.x, nw = nt / 32;
    const int C = (int)gridDim.x, b = (int)blockIdx.x;  // a cluster launch is one cluster
    const int W = C * nw, wid = b + C * warp;
    unsigned arrivals = 0;
    auto sync = [&]() -> bool {
        if (GRID) {
            arrivals += (unsigned)C;
            return grid_sync(p.bar, p.err, arrivals);
        }
        __threadfence();  // results go through L2
        __syncwarp();
        cluster_sync();
        return true;
    };
    // power-of-two scale: |entries of T| < 1
    if (tid == 0) s_max = 0;
    __syncthreads();
    {
        unsigned m = 0;
        for (int i = tid; i < n; i += nt) {
            m = max(m, (unsigned)__double2hiint(p.d[i]) & 0x7fffffffu);
            if (i + 1 < n) m = max(m, (unsigned)__double2hiint(p.e[i]) & 0x7fffffffu);
        }
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) atomicMax(&s_max, m);
    }
    __syncthreads();
    const int ex = min(max((int)(s_max >> 20) - 1022, -900), 900);
    const double down = scalbn(1.0, -ex), up = s_max ? scalbn(1.0, ex) : 0.0;
    // the cut above row i
    auto cut_at = [&](int i) { return cut(p.d[i - 1] * down, p.d[i] * down, p.e[i - 1] * down); };
    double *Q = p.Qa, *Qn = p.Qb;
    // ---- base blocks: a warp each, levels 2, 4 and 8 in its shared memory ------------
    for (int B = wid; B * BASE < n; B += W) {
        BaseMem& s = *reinterpret_cast<BaseMem*>(dsm + (size_t)warp * sizeof(BaseMem));
        const int r0 = B * BASE, N = min(BASE, n - r0), i = lane & (BASE - 1);
        __syncwarp();
        if (lane < N) {
            double x = p.d[r0 + i] * down;
            if (r0 + i > 0) {
                const Cut c = cut_at(r0 + i);
                x = fma(-c.rho, c.b * c.b, x);
            }
            if (r0 + i + 1 < n) {
                const Cut c = cut_at(r0 + i + 1);
                x = fma(-c.rho, c.a * c.a, x);
            }
            s.D[i] = x;
        }
        for (int t = lane; t < BASE * BASE; t += 32) s.Q[0][t] = t % BASE == t / BASE ? 1.0 : 0.0;
        int cur = 0;
        for (int h = 1; h < N; h *= 2) {
            const int K0 = 2 * h;
            __syncwarp();
            const double *q = s.Q[cur];
            double* qn = s.Q[cur ^ 1];
            {  // poles: lanes 0..7
                const int lo = i / K0 * K0, mid = lo + h, hi = min(lo + K0, N);
                const bool on = lane < N && mid < N;
                if (lane < N) s.key[i] = okey(s.D[i]);
                __syncwarp();
                int rk = i - lo;
                if (on) {
                    const ll k = s.key[i];
                    rk = 0;
                    for (int t = lo; t < hi; ++t) rk += s.key[t] < k || (s.key[t] == k && t < i);
                    const Cut c = cut_at(r0 + mid);
                    double z = q[(i < mid ? mid - 1 : mid) + BASE * i];
                    if (expo(z) < -56) z = copysign(0x1p-56, z);
                    s.srt[lo + rk] = k;
                    s.z[lo + rk] = i < mid ? c.a * z : copysign(c.b, p.e[r0 + mid - 1]) * z;
                    s.idx[lo + rk] = i - lo;
                }
                __syncwarp();
                if (on) {  // i as a place in the order
                    const double v = unkey(s.srt[i]);
                    const int r = i - lo;
                    ll run = LLONG_MIN / 2;
                    for (int t = 0; t < r; ++t) run = max(run, to_grid(unkey(s.srt[lo + t])) - t);
                    s.ds[i] = to_grid(v) < run + r ? from_grid(run + r) : v;
                }
                __syncwarp();
            }
            // roots: groups of four lanes
            const int g = 4, jj = min(lane / g, N - 1);
            {
                const int lo = jj / K0 * K0, mid = lo + h;
                const bool on = lane / g < N && mid < N;
                // lanes without a root follow the first
                const int lo1 = on ? lo : 0, j = on ? jj - lo : 0, K = min(lo1 + K0, N) - lo1;
                const double rinv = rcp(cut_at(r0 + lo1 + h).rho);
                int o;
                double mu;
                find_root<2, true>(s.ds + lo1, s.z + lo1, K, K0, g, j, rinv, s.pf[lane / g], o, mu);
                __syncwarp();
                if (on && (lane & (g - 1)) == 0) {
                    double lam = s.ds[lo + o] + mu;
                    lam = fmax(lam, s.ds[jj]);
                    if (j + 1 < K) lam = fmin(lam, s.ds[jj + 1]);
                    s.org[jj] = o;
                    s.mu[jj] = mu;
                    s.D[jj] = lam;
                }
                __syncwarp();
                const double zh = new_z<true>(s.ds + lo1, s.mu + lo1, s.org + lo1, s.z + lo1, K, g, j);
                if (on && (lane & (g - 1)) == 0) s.zh[jj] = zh;
                __syncwarp();
                double* u = s.u[lane / g];
                const int jr = on ? jj : 0;
                const double inv = coefficients<true>(s.ds + lo1, s.zh + lo1, s.idx + lo1, s.ds[lo1 + s.org[jr]],
                                                      s.mu[jr], K, g, u);
                __syncwarp();
                if (lane / g < N)
                    for (int r = lane & (g - 1); r < K0 && lo + r < N; r += g) {
                        const int row = lo + r;
                        double v = 0.0;
                        if (on) {
                            const int i0 = row < mid ? 0 : h, i1 = row < mid ? h : K;
                            for (int t = i0; t < i1; ++t) v = fma(q[row + BASE * (lo + t)], u[t], v);
                            v *= inv;
                        } else {
                            v = q[row + BASE * jj];
                        }
                        qn[row + BASE * jj] = v;
                    }
            }
            cur ^= 1;
        }
        __syncwarp();
        if (lane < N) p.D[r0 + i] = s.D[i];
        if (n > BASE) {
            for (int t = lane; t < N * N; t += 32)
                Q[r0 + t % N + (size_t)n * (r0 + t / N)] = s.Q[cur][t % N + BASE * (t / N)];
        } else {
            for (int t = lane; t < N * p.want; t += 32)
                p.Z[t % N + N * (t / N)] = s.Q[cur][t % N + BASE * (N - 1 - t / N)];
            if (lane < p.want) p.lam_asc[lane] = s.D[N - p.want + lane] * up;
        }
    }
    if (!sync()) return;
    for (int h = BASE; h < n; h *= 2) {
        const int K0 = 2 * h, nm = (n + K0 - 1) / K0;
        const bool last = K0 >= n;
        // ---- poles of every merge: one block each -----------------------------
        for (int m = b; m < nm; m += C) {
            const int lo = m * K0, mid = lo + h, hi = min(lo + K0, n), K = hi - lo;
            if (mid >= n) continue;  // an unpaired block goes up as it is
            ll* key = reinterpret_cast<ll*>(dsm);
            ll* srt = key + K;
            const Cut cm = cut_at(mid);
            const double cb = copysign(cm.b, p.e[mid - 1]);
            if (tid == 0) p.rinv[mid] = rcp(cm.rho);
            for (int i = tid; i < K; i += nt) key[i] = okey(__ldcg(p.D + lo + i));
            __syncthreads();
            for (int i = tid; i < K; i += nt) {
                double z = __ldcg(Q + (i < h ? mid - 1 : mid) + (size_t)n * (lo + i));
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
                if (expo(z) < -56) z = copysign(0x1p-56, z);
                p.z[lo + rk] = z * (i < h ? cm.a : cb);
                p.idx[lo + rk] = i;
            }
            __syncthreads();
            // distinct: on a grid of ulps, 2^-82 below 2^-30, pole r at least one
            // step above pole r-1 (a prefix maximum); poles that are distinct
            // already stay
            const int per = (K + nt - 1) / nt, r0 = min(tid * per, K), r1 = min(r0 + per, K);
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
        // groups of g lanes, gw of them to a warp; unit u of the level at lane's group
        const int g = min(K0, 32), gw = 32 / g, gl = lane & (g - 1), sub = lane / g;
        // ---- roots ----------------------------------------------------------------
        if (warp < p.warps2) {
            for (int u0 = wid * gw; u0 < n; u0 += C * p.warps2 * gw) {
                const int r = u0 + sub;
                // an unpaired block or none: lanes follow the level's first root
                const bool on = r < n && r / K0 * K0 + h < n;
                if (!__any_sync(0xffffffffu, on)) continue;
                const int G = on ? r : 0, lo = G / K0 * K0, mid = lo + h, K = min(lo + K0, n) - lo, j = G - lo;
                float2* pf = reinterpret_cast<float2*>(dsm) + (size_t)warp * max(K0, 32) + sub * K0;
                const double rinv = __ldcg(p.rinv + mid);
                int o;
                double mu;
                if (K0 <= 128) find_root<4, false>(p.ds + lo, p.z + lo, K, K0, g, j, rinv, pf, o, mu);
                else find_root<0, false>(p.ds + lo, p.z + lo, K, K0, g, j, rinv, pf, o, mu);
                if (on && gl == 0) {
                    double lam = __ldcg(p.ds + lo + o) + mu;
                    lam = fmax(lam, __ldcg(p.ds + G));
                    if (j + 1 < K) lam = fmin(lam, __ldcg(p.ds + G + 1));
                    p.org[G] = o;
                    p.mu[G] = mu;
                    p.D[G] = lam;
                }
                __syncwarp();
            }
        }
        if (!sync()) return;
        // ---- z from the roots ---------------------------------------------------
        for (int u0 = wid * gw; u0 < n; u0 += W * gw) {
            const int r = u0 + sub;
            const bool on = r < n && r / K0 * K0 + h < n;
            if (!__any_sync(0xffffffffu, on)) continue;
            const int G = on ? r : 0, lo = G / K0 * K0, K = min(lo + K0, n) - lo;
            const double zh = new_z<false>(p.ds + lo, p.mu + lo, p.org + lo, p.z + lo, K, g, G - lo);
            if (on && gl == 0) p.zh[G] = zh;
        }
        if (!sync()) return;
        // ---- eigenvectors: Q blockdiag times the rank-one problem's ---------------
        // A unit is a column and one of wpc shares of its rows; every warp of a
        // column forms the column's coefficients itself.
        const int g0 = last ? n - p.want : 0, cols = n - g0;
        int wpc = 1;
        while (wpc < 16 && 2 * wpc * cols <= C * p.warps2 && 32 * wpc < K0) wpc *= 2;
        for (int u0 = wid * gw; u0 < cols * wpc && warp < p.warps2; u0 += C * p.warps2 * gw) {
            const int unit = u0 + sub;
            const bool have = unit < cols * wpc;
            const int c = g0 + (have ? unit : 0) / wpc, part = (have ? unit : 0) % wpc;
            const int lo = c / K0 * K0, mid = lo + h, hi = min(lo + K0, n);
            const bool on = mid < n;
            double* out = last ? p.Z + (size_t)n * (n - 1 - c) : Qn + (size_t)n * c;
            if (have && last && part == 0 && gl == 0) p.lam_asc[c - g0] = __ldcg(p.D + c) * up;
            double* u = reinterpret_cast<double*>(dsm) + (size_t)warp * max(K0, 32) + sub * K0;
            // lanes without a merged column form the first column's coefficients
            const int cc = on ? c : 0, lc = on ? lo : 0, K = min(lc + K0, n) - lc;
            const int og = min(max(__ldcg(p.org + cc), 0), K - 1);
            __syncwarp();
            const double inv = coefficients<false>(p.ds + lc, p.zh + lc, p.idx + lc, __ldcg(p.ds + lc + og),
                                                   __ldcg(p.mu + cc), K, g, u);
            __syncwarp();
            if (!have) continue;
            if (!on) {  // unpaired
                for (int r = lo + g * part + gl; r < hi; r += g * wpc) out[r] = __ldcg(Q + r + (size_t)n * c);
                continue;
            }
            for (int r = lo + g * part + gl; r < hi; r += g * wpc) {
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
    char* base = static_cast<char*>(ctx->s_dc.get(ctx, 6 * n8 + 2 * n4 + 2 * nn));
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
    a.rinv = reinterpret_cast<double*>(take(n8));
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
    const bool grid = n > 128 || ctx->trd_clusters == 0;
    const int nw = !grid && n <= 64 ? 4 : DW;  // warps of a block
    a.warps2 = (int)std::min<int64_t>(nw, (int64_t)(DSMEM / (8 * K0)));
    TN_REQUIRE(a.warps2 >= 2, "tridiag_top: order too large");
    const size_t dyn = std::max<size_t>((size_t)8 * std::max<int64_t>(K0, 32) * a.warps2, sizeof(BaseMem) * nw);
    // One cluster (barrier 0.2 us against 1.2) while its sixteen SMs hold the
    // FP64 work of a level, the whole grid above.
    if (grid) {
        TN_CHECK_CUDA(cudaMemsetAsync(a.bar, 0, sizeof(unsigned), ctx->stream));
        TN_CHECK_CUDA(cudaFuncSetAttribute(dc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)DSMEM));
        void* args[] = {&a};
        TN_CHECK_CUDA(cudaLaunchCooperativeKernel((void*)dc_kernel<true>, dim3((unsigned)ctx->sm_count),
                                                  dim3(DT), args, dyn, ctx->stream));
    } else {
        // blocks: a warp per root at the last level, up to order 64 one on each scheduler
        const int C = n <= 8 ? 1 : n <= 16 ? 2 : n <= 32 ? 8 : DC_CLUSTER;
        TN_CHECK_CUDA(cudaFuncSetAttribute(dc_kernel<false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = (unsigned)C;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)C);
        cfg.blockDim = dim3(32 * nw);
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
