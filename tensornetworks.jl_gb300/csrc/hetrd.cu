// Householder reduction of a Hermitian matrix to a real symmetric tridiagonal,
// G = Q T Q^H, in fixed point (fixp.cuh): step 1 of the eigensolver (eig.cu).
//
// One thread-block cluster holds the whole matrix in its shared memories up to
// order 208; above, the blocks of a cooperative grid do, and from about order 1100
// the rows stay in global memory (L2).  Row i belongs to block i mod C.  Step j:
//   A. a warp per row applies the pending rank-2 update of step j-1 to the
//      row and sums its product with v, in one pass, while a further warp forms
//      the reflector's scalars in FP64 (its only FP64 work: about thirty
//      instructions of 64 clocks); the row's product, its entry of column j+1
//      and its share of v^H A v go to every block;
//   B. after one barrier (cluster: 0.2 us, grid: 1.2 us) every block forms w,
//      column j+1 with this step's update and its exact squared norm itself.
// The FP64 version spent 8.7 us per step at order 256, 11 at 512: a 1.9 us grid
// barrier, five block sums of ten dependent 64-clock additions each and a serial
// square root and two divisions (2,000 clocks).
//
// In a cluster a step is a chain of dependent integer instructions (7,900 clocks at
// order 64: limbs of v 780, rows 2,200 with their sums, exchange 1,550, w 1,900,
// column and norm 1,150); the grid adds its barrier and vectors through L2, and at
// order 2048 the rows' integer multiplications and their traffic through L2 take
// 38,000 of 60,000 clocks.  Against the first version (8 row warps, one entry a lane
// at a time, w in two passes): rows two entries deep with the next two loaded ahead,
// 16 row warps and rows shared by warps in the grid forms, the products of w by
// 32-bit limbs, the new exponent of row j+1 from the last step's smallest exponent
// (so that w needs one pass) and work that nobody waits for behind the exchange took
// order 64 from 308 to 245 us, 128 from 699 to 571, 256 from 2,069 to 1,646, 512
// from 6,574 to 3,830, 1024 from 21.3 to 12.0 ms, 2048 from 98 to 58 ms.  With all bounds
// of the update vectors' scale (q_exponent) they take 262, 577, 1,826 and 4,198 us, 13.0
// and 59.6 ms.
//
// Reflector j is kept as V[j n + i] (i > j, the first entry explicit) and tau[j]:
// H_j = I - tau_j v_j v_j^H.  Results become FP64 while the exchange travels, or by
// the scalar warp while it waits: a launch of their own took 4.7 us.
#include <climits>
#include <cmath>

#include "common.cuh"
#include "fixp.cuh"
#include "grid_dev.cuh"

namespace tn {

namespace {

using namespace fixp;
using namespace griddev;

constexpr int HC = 16;   // blocks of a full cluster
constexpr int HROWS = 32;  // most rows of a block left in a step
constexpr int HPAD = 64;  // zeros after the vectors: rows run in steps of 64 entries

// A cluster with its rows in shared memory, a grid likewise, a grid with its rows in
// global memory.
enum Form { CLUSTER, GRID_SHARED, GRID_GLOBAL };

struct TrdOut {
    cplx* V;         // n x n, column j: reflector j
    cplx* tau;       // n
    double *d, *e;   // n: the tridiagonal
    int* perm;       // n: row of G that became row l, when psd
};

struct TrdIn {
    const cplx* G;  // n x n, lower triangle
    int n, psd;
    TrdOut o;
    zint* A;          // grid form: n x n rows in global memory
    zint* mp;         // grid form: mailbox, two buffers of n entries each
    zint* ma;
    ll* md;
    ull* mq;          // grid form: v^H A v, triple buffered by step
    int* mx;          // grid form: the products' largest number of bits, likewise
    zint* xr;         // rows in global memory: a block's copy of the column
    unsigned* part;   // grid form: per-block scale partials
    unsigned* bar;    // grid form: arrival counter (zero at launch)
    int* err;
};

__device__ __forceinline__ void bar_named(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// address in block `rank`'s shared memory of this block's address p
__device__ __forceinline__ uint32_t map_shared(const void* p, unsigned rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
// stores that report their bytes to the receiving block's mbarrier
__device__ __forceinline__ void st_async(uint32_t a, zint v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(a),
                 "l"(v.x), "l"(v.y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async(uint32_t a, ll v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
                 "l"(v), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t a, unsigned v) {
    asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// Waits for a phase of this block's mbarrier; false when the bound runs out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(bar);
    uint64_t t0 = 0;
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
        const uint64_t t = hclock();
        if (t0 == 0) t0 = t;
        else if (t - t0 > HWAIT_NS) return false;
    }
}

// sum modulo 2^64 by three 22-bit limbs (three REDUX; ten shuffles take 144 clocks)
__device__ __forceinline__ ll warp_sum64(ll v) {
    const unsigned a = __reduce_add_sync(0xffffffffu, (unsigned)v & 0x3fffffu);
    const unsigned b = __reduce_add_sync(0xffffffffu, (unsigned)(v >> 22) & 0x3fffffu);
    const unsigned c = __reduce_add_sync(0xffffffffu, (unsigned)((ull)v >> 44));
    return (ll)((ull)a + ((ull)b << 22) + ((ull)c << 44));
}

struct ShCtl {
    ull q;               // grid form: the block's share of v^H A v, its rows' largest product
    int pm;
    zint sum[HROWS];     // products of row segments with v
    zint first[HROWS];   // rows' entries of column j+1
    ll diag[HROWS];
    alignas(16) zint qt[2][8 * HC];  // cluster form: every warp's share and largest product, from every block
    uint64_t mbar[2];    // cluster form: a step's exchange has arrived
    int abort;
    unsigned S[3][NORM_LIMBS];  // squared norm, limbs, triple buffered by step
    int vm[3];           // largest entry of v 2^-e, log2, likewise
    int emin[3];         // smallest exponent of the rows left, likewise
    int shift[3];        // whether any exponent changed, likewise
    int em, c;           // smallest exponent of the rows left, the column's exponent
    zint alpha;          // first entry of the column before the shift
    ll beta;
    ll dint;  // diagonal entry just formed, in units of 2^(f - 61 - dexp)
    int dexp;
    zint v1, tau;
    ll c2;
    unsigned part[2 * HC];  // scale partials of the cluster's blocks
};

__device__ __forceinline__ zint ld_zint(const zint* p) {
    const longlong2 v = __ldcg(reinterpret_cast<const longlong2*>(p));
    return zint{v.x, v.y};
}

// x 2^s rounded to an integer (|x 2^s| < 2^62; denormal x counts as zero)
__device__ __forceinline__ ll to_fix(double x, int s) {
    const ll b = __double_as_longlong(x);
    const int ex = (int)((b >> 52) & 0x7ff);
    if (ex == 0) return 0;
    const ll m = (b & 0xfffffffffffffll) | 0x10000000000000ll;
    const ll r = sft(m, ex - 1075 + s);
    return b < 0 ? -r : r;
}

// x 2^-56 as FP64, |x| < 2^62
__device__ __forceinline__ double unit56(ll x) { return scale2(__ll2double_rn(x), -56); }

template <int FORM>
constexpr int ROW_WARPS = FORM == CLUSTER ? 8 : 16;  // of a block

template <int FORM>
__global__ void __launch_bounds__(32 * ROW_WARPS<FORM> + 32) hetrd_fix_kernel(TrdIn p) {
    constexpr bool GRID = FORM != CLUSTER;
    constexpr int RW = ROW_WARPS<FORM>;
    constexpr int HM = 32 * RW, HT = HM + 32;  // threads of the row warps; the scalar warp
    extern __shared__ __align__(16) unsigned char hsm[];
    __shared__ ShCtl sh;
    const int n = p.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int C = GRID ? (int)gridDim.x : (int)cluster_size();
    const int b = GRID ? (int)blockIdx.x : (int)cluster_rank();
    const int R = (n + C - 1) / C;
    // shared memory: v's limbs for products, v's and w's for the pending update,
    // exponents, their pending change and their bound; the column and the rows
    // unless they are in global memory; in the cluster form the mailbox
    int4* vD = reinterpret_cast<int4*>(hsm);
    int4* vU = vD + n + HPAD;
    int4* wU = vU + n + HPAD;
    zint* xs = reinterpret_cast<zint*>(wU + n + HPAD);
    zint* xr = FORM == GRID_GLOBAL ? p.xr + (size_t)b * n : xs;
    zint* A = FORM == GRID_GLOBAL ? p.A : xs + n;  // row i at A + row(i) n
    zint* mp = GRID ? p.mp : xs + n + (size_t)R * n;
    zint* ma = GRID ? p.ma : mp + 2 * n;
    ll* md = GRID ? p.md : reinterpret_cast<ll*>(ma + 2 * n);
    signed char* ee = FORM == GRID_GLOBAL   ? reinterpret_cast<signed char*>(xs)
                      : FORM == GRID_SHARED ? reinterpret_cast<signed char*>(A + (size_t)R * n)
                                            : reinterpret_cast<signed char*>(md + 2 * n);
    signed char* de = ee + n;
    signed char* cap = de + n;  // largest exponent a row may get
    auto row = [&](int i) { return FORM == GRID_GLOBAL ? i : i / C; };
    unsigned arrivals = 0;

    // ---- scale: a power of two above the Frobenius norm -------------------------
    if (tid < 3 * NORM_LIMBS) (&sh.S[0][0])[tid] = 0;
    if (tid == 0) {
        sh.abort = 0;
        sh.q = 0;
        sh.pm = 0;
        for (int k = 0; k < 3; ++k) {
            sh.emin[k] = INT_MAX;
            sh.vm[k] = INT_MIN;
            sh.shift[k] = 0;
            if (GRID && b == 0) p.mq[k] = 0, p.mx[k] = 0;
        }
        if (!GRID) {  // seen by the others after the cluster barrier below
            for (int k = 0; k < 2; ++k)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(
                    (uint32_t)__cvta_generic_to_shared(&sh.mbar[k])));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    // a block's shared memory takes others' stores from the time it runs, no earlier
    if (!GRID) cluster_sync();
    unsigned hmax = 0;
    for (int i = b + C * warp; i < n && warp < RW; i += RW * C)
        for (int l = lane; l <= i; l += 32) {
            const cplx v = p.G[i + (size_t)n * l];
            const double im = l == i ? 0.0 : v.y;
            hmax = max(hmax, max((unsigned)__double2hiint(v.x) & 0x7fffffffu,
                                 (unsigned)__double2hiint(im) & 0x7fffffffu));
        }
    hmax = __reduce_max_sync(0xffffffffu, hmax);
    __shared__ unsigned s_max;
    __shared__ float s_sum[RW];
    if (tid == 0) s_max = 0;
    __syncthreads();
    if (lane == 0 && warp < RW) atomicMax(&s_max, hmax);
    __syncthreads();
    auto share = [&](unsigned v, int slot) -> bool {  // this block's partial to all blocks
        if (GRID) {
            if (tid == 0) p.part[slot * C + b] = v;
            arrivals += (unsigned)C;
            return grid_sync(p.bar, p.err, arrivals);
        }
        if (tid < C) st_cluster(map_shared(&sh.part[slot * HC + b], tid), v);
        cluster_sync();
        return true;
    };
    auto shared_part = [&](int slot, int i) {
        return GRID ? __ldcg(p.part + slot * C + i) : sh.part[slot * HC + i];
    };
    if (!share(s_max, 0)) return;
    hmax = 0;
    for (int i = 0; i < C; ++i) hmax = max(hmax, shared_part(0, i));
    if (hmax >= 0x7ff00000u) {  // an infinity or NaN: no block goes on
        if (b == 0) {
            const double nan = __longlong_as_double(0x7ff8000000000000ll);
            for (int i = tid; i < n; i += HT) {
                p.o.d[i] = p.o.e[i] = nan;
                p.o.tau[i] = cmk(0, 0);
                if (p.psd) p.o.perm[i] = i;
            }
            for (int64_t i = tid; i < (int64_t)n * n; i += HT) p.o.V[i] = cmk(0, 0);
        }
        if (!GRID) cluster_sync();  // no block leaves while others read its memory
        return;
    }
    const int emax = max((int)(hmax >> 20), 1) - 1022;  // |entries| < 2^emax
    const double dn = scalbn(1.0, -max(emax, -1000));
    float sum = 0.f;
    for (int i = b + C * warp; i < n && warp < RW; i += RW * C)
        for (int l = lane; l <= i; l += 32) {
            const cplx v = p.G[i + (size_t)n * l];
            const float x = (float)(v.x * dn), y = l == i ? 0.f : (float)(v.y * dn);
            sum += (l == i ? 1.f : 2.f) * (x * x + y * y);
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0 && warp < RW) s_sum[warp] = sum;
    __syncthreads();
    sum = 0.f;
    for (int w = 0; w < RW; ++w) sum += s_sum[w];
    if (!share(__float_as_uint(sum), 1)) return;
    sum = 0.f;
    for (int i = 0; i < C; ++i) sum += __uint_as_float(shared_part(1, i));
    // F^2 < 2^(2 f): the FP32 sum is good to 1e-3
    int fe;
    frexpf(sum * 1.01f, &fe);
    const int f = max(emax, -1000) + (fe + 1) / 2;

    // ---- order, exponents, this block's rows as integers --------------------------
    // Rows of a graded matrix go by descending diagonal: eliminated in that order,
    // small eigenvalues keep their relative accuracy (in the opposite order they
    // lose it in FP64 too).
    int* perm = reinterpret_cast<int*>(wU);
    if (p.psd) {
        float* key = reinterpret_cast<float*>(vD);
        for (int l = tid; l < n; l += HT) key[l] = (float)scalbn(p.G[l + (size_t)n * l].x, -f);
        __syncthreads();
        for (int l = tid; l < n; l += HT) {
            const float k = key[l];
            int r = 0;
            for (int i = 0; i < n; ++i) r += key[i] > k || (key[i] == k && i < l);
            perm[r] = l;
            if (b == 0) p.o.perm[r] = l;
        }
    } else {
        for (int l = tid; l < n; l += HT) perm[l] = l;
    }
    __syncthreads();
    int em = INT_MAX;
    for (int l = tid; l < n; l += HT) {
        const int64_t pl = perm[l];
        const int e0 = p.psd ? next_exponent(0, EXP_MAX, (float)scalbn(p.G[pl + n * pl].x, -f), 0.f, 0.f, 0.f) : 0;
        ee[l] = (signed char)e0;
        de[l] = 0;
        cap[l] = (signed char)min(EXP_MAX, e0 + EXP_GAIN);
        em = min(em, e0);
    }
    em = __reduce_min_sync(0xffffffffu, em);
    if (lane == 0) atomicMin(&sh.emin[0], em);
    __syncthreads();
    em = sh.emin[0];  // over all rows: at most the smallest below row 0
    int c = max(0, em - 6);
    if (tid == 0) {
        sh.em = em;
        sh.c = c;
    }
    auto entry = [&](int i, int l) {  // (i, l) of the reordered matrix
        const int64_t pi = perm[i], pl = perm[l];
        cplx v = pl <= pi ? p.G[pi + n * pl] : p.G[pl + n * pi];
        if (pl > pi) v.y = -v.y;
        if (pl == pi) v.y = 0.0;
        return v;
    };
    for (int i = b + C * warp; i < n && warp < RW; i += RW * C)
        for (int l = lane; l < n; l += 32) {
            const cplx v = entry(i, l);
            const int s = 61 - f + ee[i] + ee[l];
            A[(size_t)row(i) * n + l] = zint{to_fix(v.x, s), to_fix(v.y, s)};
        }

    // One entry of the next column (rows left from l1 on): kept, its square added.
    auto emit = [&](int l, int l1, zint x, int el, int emn, Norm2& S) {
        xr[l] = x;
        if (l == l1) sh.alpha = x;
        norm_add(S, x, el - emn);
    };
    auto add_norm = [&](const Norm2& S, int buf) {  // exact: limbs through warp adds
        unsigned mine = 0;
#pragma unroll
        for (int k = 0; k < NORM_LIMBS; ++k) {
            const unsigned t = __reduce_add_sync(0xffffffffu, norm_limb(S, k));
            if (lane == k) mine = t;
        }
        if (lane < NORM_LIMBS && mine) atomicAdd(&sh.S[buf][lane], mine);
    };
    if (warp < RW) {  // column 0
        Norm2 S{0, 0};
        for (int l = tid; l < n; l += HM) {
            const cplx v = entry(l, 0);
            if (l == 0) {
                sh.dint = to_fix(v.x, 61 - f + 2 * c);
                sh.dexp = 2 * c;
                continue;
            }
            const int s = 61 - f + ee[l] + c;
            emit(l, 1, zint{to_fix(v.x, s), to_fix(v.y, s)}, ee[l], em, S);
        }
        add_norm(S, 0);
    }
    // an integer of unit 2^(f - 61 - s) as FP64
    auto unfix = [&](ll x, int s) { return scalbn(__ll2double_rn(x), f - 61 - s); };
    __syncthreads();
    for (int l = tid; l < 3 * (n + HPAD); l += HT) vD[l] = make_int4(0, 0, 0, 0);  // vU and wU too
    // block `lane`'s mailbox
    uint32_t rmp = 0, rma = 0, rmd = 0, rqt = 0, rbar = 0;
    if (!GRID && lane < C) {
        rmp = map_shared(mp, lane);
        rma = map_shared(ma, lane);
        rmd = map_shared(md, lane);
        rqt = map_shared(sh.qt, lane);
        rbar = map_shared(sh.mbar, lane);
    }
    int i0 = b, nrows = b < n ? (n - 1 - b) / C + 1 : 0;  // the first own row above j, own rows left
    for (int j = 0; j + 1 < n; ++j) {
        __syncthreads();  // squared norm of the column, its entries and alpha
        // its bit length, by lanes
        const unsigned nl = lane < NORM_LIMBS ? sh.S[j % 3][lane] : 0;
        unsigned below = __shfl_up_sync(0xffffffffu, nl, 1);
        if (lane == 0) below = 0;
        const unsigned nc = norm_carry(nl, below);
        const unsigned some = __ballot_sync(0xffffffffu, nc != 0);
        const int kt = 31 - __clz(some | 1);
        const int bl = 22 * kt + 32 - __clz(__shfl_sync(0xffffffffu, nc, kt));  // zero: no column
        const int shf = bl ? norm_shift(bl) : 0;
        em = sh.em;
        c = sh.c;
        const int l0 = j + 1, s0 = ee[l0] - em;  // first row left
        const int gb = p.psd ? min(em, guard_bits(n - j)) : 0;
        const int cn = max(0, em - 6);  // its new exponent: its diagonal is at most the trace, n 2^(-2 em)
        const int buf = j & 1, nb = (j + 1) % 3;
        if (warp == RW) {
            // beta and v's first entry for the row warps, then tau and c2 while
            // the rows' results travel
            double ar = 0.0, ai = 0.0, be = 0.0, sq = 0.0, tr = 0.0, ti = 0.0;
            const ll dint = sh.dint;
            const int dexp = sh.dexp;
            if (lane == 0) {
                ll beta = 0;
                zint al{0, 0};
                if (bl) {
                    // squared norm in v's unit: S 2^(2 shf - 112 - 56), in [1/4, 1)
                    const NormTop S = norm_top(sh.S[j % 3]);
                    sq = scale2(__ull2double_rn(S.top), S.bl + 2 * shf - 232);
                    al = zsft(sh.alpha, shf - s0);
                    be = sq * rsqrt(sq);
                    be = al.x < 0 ? be : -be;
                    beta = __double2ll_rn(scale2(be, 56));
                }
                sh.beta = beta;
                sh.v1 = zint{al.x - beta, al.y};
                if (!GRID)
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                                     (uint32_t)__cvta_generic_to_shared(&sh.mbar[buf])),
                                 "r"(40 * (n - j - 1) + 16 * RW * C)
                                 : "memory");
                ar = scale2(__ll2double_rn(al.x), -56);
                ai = scale2(__ll2double_rn(al.y), -56);
            }
            __syncwarp();
            bar_named(2, HT);
            if (lane == 0) {
                zint tau{0, 0};
                ll c2 = 0;
                if (bl) {
                    // |beta - alpha|^2 = s + |alpha|^2 + 2 |beta alpha_r| (no cancellation)
                    const double D = fma(ar, ar, fma(ai, ai, fma(-(be + be), ar, sq)));
                    const double ri = recip(be * D);
                    tr = (be - ar) * ri;
                    ti = -ai * ri;
                    tau = zint{__double2ll_rn(scale2(tr, 59)), __double2ll_rn(scale2(ti, 59))};
                    c2 = __double2ll_rn(scale2(D * ri * ri, 58));  // |tau|^2 = D / (beta D)^2
                }
                sh.tau = tau;
                sh.c2 = c2;
            }
            __syncwarp();
            bar_named(3, HT);  // the exchange; tau and c2
            if (lane == 0) {
                if (b == 0) {
                    p.o.tau[j] = cmk(tr, ti);
                    p.o.d[j] = unfix(dint, dexp);
                    p.o.e[j] = unfix(sh.beta, shf + em + c);
                }
                if (b == l0 % C)
                    p.o.V[(size_t)j * n + l0] = cmk(unit56(sh.v1.x), unit56(sh.v1.y));
            }
            if (sh.abort) break;
        } else {
            // column -> v's limbs for the products (the first entry still alpha)
            for (int l = l0 + tid; l < n; l += HM) vD[l] = limbs29(zsft(xr[l], shf - 2 * (ee[l] - em) - gb));
            __syncwarp();
            bar_named(1, HM);
            // ---- A. rows: pending update, product with v ------------------------
            const bool moved = sh.shift[j % 3] != 0;
            // row i from its entry l on, every dl-th 64 of them: its lane's share of
            // the product; the entry of column j+1 and the diagonal one as they pass
            auto row_part = [&](int i, int l, int dl, zint& first, ll& dg) -> zint {
                zint* a = A + (size_t)row(i) * n;
                Dot s{0, 0, 0, 0, 0, 0};
                const int4 wi = wU[i], vi = vU[i];
                const int di = de[i];
                auto one = [&](zint x, int l) {  // entries from n on count zero
                    if (moved) x = zsft(x, di + de[min(l, n - 1)]);
                    update(x, wi, vi, wU[l], vU[l]);
                    if (l < n) a[l] = x;
                    if (l == l0) first = x;
                    if (l == i) dg = x.x;
                    dot_add(s, x, vD[l]);
                };
                zint x0 = a[min(l, n - 1)], x1 = a[min(l + 32, n - 1)];
                for (int t = 0; l - lane < n; l += dl, ++t) {
                    if (FORM == GRID_GLOBAL && (t & 15) == 15) dot_carry(s);  // others: up to 36 entries in all
                    const zint y0 = a[min(l + dl, n - 1)], y1 = a[min(l + dl + 32, n - 1)];
                    one(x0, l);
                    one(x1, l + 32);
                    x0 = y0;
                    x1 = y1;
                }
                return dot_value(s);
            };
            if (!GRID) {
                // a warp to a row; lane k keeps and finishes the warp's k-th row
                zint P{0, 0}, Aj{0, 0};
                ll Dg = 0;
                int k = 0;
                int i = b + C * warp;
                if (i <= j) i += (j - i + RW * C) / (RW * C) * (RW * C);  // first own row above j
                const int w0 = i;
                for (; i < n; i += RW * C, ++k) {
                    zint first{0, 0};
                    ll dg = 0;
                    const zint t = row_part(i, l0 + lane, 64, first, dg);
                    const ll px = warp_sum64(t.x), py = warp_sum64(t.y);
                    const ll fx = __shfl_sync(0xffffffffu, first.x, 0), fy = __shfl_sync(0xffffffffu, first.y, 0);
                    dg = __shfl_sync(0xffffffffu, dg, (i - l0) & 31);
                    if (lane == k) {
                        P = zint{px, py};
                        Aj = zint{fx, fy};
                        Dg = dg;
                    }
                }
                bar_named(2, HT);  // beta and the first entry of v
                const int io = w0 + RW * C * lane;
                ll q = 0;
                int pm = 0;
                if (lane < k) {
                    P = minus_real(P, Aj, sh.beta, s0 + gb);
                    pm = max(bits64(P.x), bits64(P.y));
                    q = re_dot(io == l0 ? zsft(sh.v1, -s0 - gb) : value29(vD[io]), P);
                }
                // every warp sends its share of q, rows or not: a block that has
                // everybody's share knows that nobody reads the buffer it will
                // write two steps on
                ll qs = 0;
                for (int r = 0; r < k; ++r) {
                    const zint pr{__shfl_sync(0xffffffffu, P.x, r), __shfl_sync(0xffffffffu, P.y, r)};
                    const zint ar{__shfl_sync(0xffffffffu, Aj.x, r), __shfl_sync(0xffffffffu, Aj.y, r)};
                    const ll dr = __shfl_sync(0xffffffffu, Dg, r);
                    qs += __shfl_sync(0xffffffffu, q, r);
                    if (lane < C) {
                        const int ir = buf * n + w0 + RW * C * r;
                        st_async(rmp + 16 * ir, pr, rbar + 8 * buf);
                        st_async(rma + 16 * ir, ar, rbar + 8 * buf);
                        st_async(rmd + 8 * ir, dr, rbar + 8 * buf);
                    }
                }
                pm = __reduce_max_sync(0xffffffffu, pm);
                if (lane < C) st_async(rqt + 16 * (8 * HC * buf + RW * b + warp), zint{qs, pm}, rbar + 8 * buf);
            } else {
                // Local row r is matrix row i0 + C r; 2^ls warps share a row while there
                // are more warps than rows (a warp alone on its scheduler takes 1,900
                // clocks for 64 entries: order 512 4,427 us without sharing, 3,794 with)
                if (i0 <= j) {
                    i0 += C;
                    --nrows;
                }
                int ls = 0;
                if (nrows > 0) {
                    ls = nrows > RW ? 0 : 31 - __clz(RW) - (nrows > 1 ? 32 - __clz(nrows - 1) : 0);
                    ls = min(ls, 31 - __clz((n - l0 + 63) >> 6));
                }
                for (int r = warp >> ls; r < nrows; r += RW >> ls) {
                    const int i = i0 + C * r, seg = warp & ((1 << ls) - 1);
                    zint first{0, 0};
                    ll dg = 0;
                    const zint t = row_part(i, l0 + 64 * seg + lane, 64 << ls, first, dg);
                    if (seg == 0 && lane == 0) sh.first[r] = first;
                    if (((i - l0) >> 6 & ((1 << ls) - 1)) == seg && ((i - l0) & 31) == lane) sh.diag[r] = dg;
                    const ll px = warp_sum64(t.x), py = warp_sum64(t.y);
                    if (lane == 0) sh.sum[(r << ls) + seg] = zint{px, py};
                }
                bar_named(2, HT);  // the rows' sums; beta and the first entry of v
                ll qs = 0;
                int pm = 0;
                for (int r = warp; r < nrows; r += RW) {  // a warp finishes a row
                    const int i = i0 + C * r, ir = buf * n + i;
                    zint P{0, 0};
                    for (int t = 0; t < 1 << ls; ++t) {
                        const zint u = sh.sum[(r << ls) + t];
                        P = zint{P.x + u.x, P.y + u.y};
                    }
                    const zint Aj = sh.first[r];
                    P = minus_real(P, Aj, sh.beta, s0 + gb);
                    if (lane == 0) {
                        mp[ir] = P;
                        ma[ir] = Aj;
                        md[ir] = sh.diag[r];
                    }
                    pm = max(pm, max(bits64(P.x), bits64(P.y)));
                    qs += re_dot(i == l0 ? zsft(sh.v1, -s0 - gb) : value29(vD[i]), P);
                }
                if (lane == 0) {
                    if (qs) atomicAdd(&sh.q, (ull)qs);
                    if (pm) atomicMax(&sh.pm, pm);
                }
                __syncwarp();
                bar_named(1, HM);
                arrivals += (unsigned)C;
                if (tid == 0) {
                    atomicAdd(p.mq + j % 3, sh.q);
                    if (sh.pm) atomicMax(p.mx + j % 3, sh.pm);
                    sh.q = 0;
                    sh.pm = 0;
                    grid_arrive(p.bar);
                }
            }
            // while the results travel: v for the back-transformation, the largest
            // entry of v 2^-e
            int vm = -s0 - gb;
            for (int l = l0 + tid; l < n; l += HM) {
                const int d = ee[l] - em;
                const zint x = xr[l];
                if (l > l0 && l % C == b) {
                    const zint v = zsft(x, shf - d);
                    p.o.V[(size_t)j * n + l] = cmk(unit56(v.x), unit56(v.y));
                }
                const int bits = max(bits64(x.x), bits64(x.y));
                if (bits) vm = max(vm, bits + shf - 2 * d - gb - 56);  // zeros have no size, whatever the shift
            }
            vm = __reduce_max_sync(0xffffffffu, vm);
            if (lane == 0) atomicMax(&sh.vm[j % 3], vm);
            if (tid < NORM_LIMBS) sh.S[nb][tid] = 0;
            if (GRID) {
                if (tid == 0) {
                    if (!grid_wait(p.bar, p.err, arrivals)) sh.abort = 1;
                    if (b == 0) p.mq[(j + 2) % 3] = 0, p.mx[(j + 2) % 3] = 0;  // every block has read step j - 1's
                }
            } else if (!mbar_wait(&sh.mbar[buf], (uint32_t)(j >> 1) & 1u)) {
                sh.abort = 1;
            }
            __syncwarp();
            bar_named(3, HT);  // the exchange; tau and c2
            if (sh.abort) {
                if (tid == 0) atomicExch(p.err, 1);
                break;
            }
        }
        // ---- B. w, column j+1, its norm ----------------------------------------
        if (warp < RW) {
            const int off = buf * n;
            // the first entry's loads travel while h is found
            zint pf{0, 0}, af{0, 0};
            ll df = 0;
            if (l0 + tid < n) {
                const int o = off + l0 + tid;
                pf = GRID ? ld_zint(mp + o) : mp[o];
                af = GRID ? ld_zint(ma + o) : ma[o];
                df = GRID ? __ldcg(md + o) : md[o];
            }
            ll q = 0;
            int pm = 0;
            if (GRID) {
                q = (ll)__ldcg(p.mq + j % 3);
                pm = __ldcg(p.mx + j % 3);
            } else {  // every warp adds all shares itself
#pragma unroll
                for (int t = 0; t < RW * HC; t += 32)
                    if (t + lane < RW * C) {
                        const zint s = sh.qt[buf][t + lane];
                        q += s.x;
                        pm = max(pm, (int)s.y);
                    }
                q = warp_sum64(q);
                pm = __reduce_max_sync(0xffffffffu, pm);
            }
            // h = log2 sqrt(v^H A v): w and v scaled by its powers stay bounded
            const int h = p.psd ? q_exponent(q, sh.vm[j % 3], pm, n - j) : 0;
            const ll al2 = q_scaled(sh.c2, q, h);
            const zint tau = sh.tau;
            // float copies for the exponents' estimate
            const float tx = (float)(int)(tau.x >> 32) * 0x1p-27f, ty = (float)(int)(tau.y >> 32) * 0x1p-27f;
            const float fp = __int_as_float((127 - 61 - h) << 23), fv = __int_as_float((127 + shf + h + gb - 56) << 23);
            const float fa = (float)(int)(al2 >> 32) * 0x1p-25f, ft = fabsf(tx) + fabsf(ty);
            int emn = INT_MAX, any = 0;
            for (int l = l0 + tid; l < n; l += HM) {
                const bool top = l == l0;
                const zint pl = l == l0 + tid ? pf : GRID ? ld_zint(mp + off + l) : mp[off + l];
                const zint x = xr[l];
                const int el = ee[l];
                int en = el;
                if (p.psd) {
                    const float px = __ll2float_rn(pl.x) * fp, py = __ll2float_rn(pl.y) * fp;
                    const float vx = __ll2float_rn(x.x) * fv, vy = __ll2float_rn(x.y) * fv;
                    const float wx = tx * px - ty * py - fa * vx, wy = tx * py + ty * px - fa * vy;
                    const float av = fabsf(vx) + fabsf(vy);
                    const float a = __ll2float_rn(l == l0 + tid ? df : GRID ? __ldcg(md + off + l) : md[off + l]) * 0x1p-61f;
                    en = next_exponent(el, cap[l], a, 2.f * (wx * vx + wy * vy),
                                       2.f * av * (ft * (fabsf(px) + fabsf(py)) + fa * av), fmaxf(vx * vx + vy * vy, 2.f * (wx * wx + wy * wy)));
                    if (top) en = cn;  // its row becomes column j+1
                }
                const int d = en - el;
                const zint vt = zsft(top ? sh.v1 : x, (top ? cn + h - em : shf + h + d) + gb);
                wU[l] = limbs31(make_w(tau, zsft(pl, d - h), al2, vt));
                vU[l] = limbs29(vt);
                ee[l] = (signed char)en;
                de[l] = (signed char)d;
                if (!top) {
                    emn = min(emn, en);
                    any |= d;
                }
            }
            emn = __reduce_min_sync(0xffffffffu, emn);
            any = __reduce_or_sync(0xffffffffu, (unsigned)any);
            if (lane == 0) {
                atomicMin(&sh.emin[nb], emn);
                if (any) sh.shift[nb] = 1;
            }
            __syncwarp();
            bar_named(1, HM);
            emn = l0 + 1 < n ? sh.emin[nb] : em;
            const int4 w1 = wU[l0], v1 = vU[l0];
            const int d0 = de[l0];
            Norm2 S2{0, 0};
            for (int l = l0 + tid; l < n; l += HM) {
                zint x = zsft(l == l0 + tid ? af : GRID ? ld_zint(ma + off + l) : ma[off + l], de[l] + d0);
                update(x, wU[l], vU[l], w1, v1);
                if (l > l0) {
                    emit(l, l0 + 1, x, ee[l], emn, S2);
                } else {
                    sh.dint = x.x;
                    sh.dexp = 2 * cn;
                }
            }
            if (l0 + 32 * warp < n) add_norm(S2, nb);
            if (tid == 0) {
                sh.em = emn;
                sh.c = cn;
                // buffers of the step after next
                sh.emin[(j + 2) % 3] = INT_MAX;
                sh.vm[(j + 2) % 3] = INT_MIN;
                sh.shift[(j + 2) % 3] = 0;
            }
        }
    }
    __syncthreads();
    if (b == 0 && tid == 0) {
        p.o.d[n - 1] = unfix(sh.dint, sh.dexp);
        p.o.tau[n - 1] = cmk(0, 0);
    }
    if (!GRID) cluster_sync();  // no block leaves while its shared memory is written
}

size_t hetrd_smem(Form form, int64_t n, int64_t C) {
    const size_t R = (size_t)((n + C - 1) / C);
    return 48 * (size_t)(n + HPAD) + 3 * (size_t)n + (form == GRID_GLOBAL ? 0 : 16 * (R + 1) * n) +
           (form == CLUSTER ? 80 * (size_t)n : 0);
}

constexpr size_t HSMEM = 220 * 1024;  // dynamic shared memory a block can have beside ShCtl

template <int FORM>
void launch(Ctx* ctx, const TrdIn& a, int64_t C, size_t smem) {
    auto k = hetrd_fix_kernel<FORM>;
    // the limit for the largest order, the same from every thread
    TN_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HSMEM));
    TN_REQUIRE(smem <= HSMEM && (a.n + C - 1) / C <= HROWS, "hetrd: matrix order too large");
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at;
    cfg.gridDim = dim3((unsigned)C);
    cfg.blockDim = dim3(32 * ROW_WARPS<FORM> + 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (FORM == CLUSTER) {
        TN_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = (unsigned)C;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
    } else {
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
    }
    TN_CHECK_CUDA(cudaLaunchKernelEx(&cfg, k, a));
}

// whether this GPU can hold the widest cluster at all
int clusters_fit() {
    auto k = hetrd_fix_kernel<CLUSTER>;
    TN_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HSMEM));
    TN_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = HC;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3(HC);
    cfg.blockDim = dim3(32 * ROW_WARPS<CLUSTER> + 32);
    cfg.dynamicSmemBytes = HSMEM;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int fit = 0;
    TN_CHECK_CUDA(cudaOccupancyMaxActiveClusters(&fit, k, &cfg));
    return fit;
}

}  // namespace

// G (n x n Hermitian, lower triangle read) -> T (d, e) and the reflectors: column
// j of V is v_j in rows j+1.. (rows above are not written), tau[j] its scalar.  psd: G
// is positive semidefinite and keeps graded accuracy, its row perm[l] as row l of Q.
// No host synchronisation; a grid barrier that ran out leaves ctx->d_bar[2] nonzero.
void hetrd(Ctx* ctx, const cplx* G, int64_t n, double* d, double* e, cplx* tau, cplx* V, bool psd, int* perm) {
    if (ctx->trd_clusters < 0) ctx->trd_clusters = clusters_fit();
    // Blocks of the cluster: the row work of a step (n^2 / 3 entries on average at
    // 180 clocks per 32) against the exchange with more blocks.  The grid's barrier
    // and vectors through L2 cost 4 us a step more, its rows next to nothing: order
    // 160 took 837 us in a cluster and 1,069 on the grid, 200 1,179 and 1,329, 256
    // 1,900 and 1,646 when the line was drawn (now 200 takes 1,210 in its cluster, 256
    // 1,826 on the grid).
    int64_t C = n <= 16 ? 1 : n <= 32 ? 4 : n <= 64 ? 8 : HC;
    const bool grid = n > 208 || ctx->trd_clusters == 0;
    if (grid) C = ctx->sm_count;
    const bool rows_global = grid && hetrd_smem(GRID_SHARED, n, C) > HSMEM;
    auto r256 = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t nn = r256(sizeof(zint) * (size_t)n * n), n8 = r256(sizeof(ll) * n),
                 nz = r256(sizeof(zint) * 2 * n);
    const size_t nx = r256(sizeof(zint) * (size_t)n * C);
    const size_t total = (rows_global ? nn + nx : 0) + (grid ? 256 + 2 * nz + 2 * n8 + r256(2 * 4 * C) : 0);
    char* base = total ? static_cast<char*>(ctx->s_trd.get(ctx, total)) : nullptr;
    auto take = [&](size_t b) {
        char* q = base;
        base += b;
        return q;
    };
    TrdIn a{};
    a.G = G;
    a.n = (int)n;
    a.psd = psd ? 1 : 0;
    a.o.V = V;
    a.o.d = d;
    a.o.e = e;
    a.o.tau = tau;
    a.o.perm = perm;
    a.err = reinterpret_cast<int*>(ctx->d_bar + 2);
    a.bar = ctx->d_bar;
    if (grid) {
        a.mq = reinterpret_cast<ull*>(take(256));
        a.mx = reinterpret_cast<int*>(a.mq + 4);
        a.mp = reinterpret_cast<zint*>(take(nz));
        a.ma = reinterpret_cast<zint*>(take(nz));
        a.md = reinterpret_cast<ll*>(take(2 * n8));
        a.part = reinterpret_cast<unsigned*>(take(r256(2 * 4 * C)));
    }
    if (rows_global) {
        a.A = reinterpret_cast<zint*>(take(nn));
        a.xr = reinterpret_cast<zint*>(take(nx));
        launch<GRID_GLOBAL>(ctx, a, C, hetrd_smem(GRID_GLOBAL, n, C));
    } else if (grid) {
        launch<GRID_SHARED>(ctx, a, C, hetrd_smem(GRID_SHARED, n, C));
    } else {
        launch<CLUSTER>(ctx, a, C, hetrd_smem(CLUSTER, n, C));
    }
    ctx->count();
    TN_CHECK_CUDA(cudaGetLastError());
}

}  // namespace tn
