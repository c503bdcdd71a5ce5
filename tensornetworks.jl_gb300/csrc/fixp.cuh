// Fixed-point arithmetic of the Householder tridiagonalisation (hetrd.cu).
//
// A warp's FP64 instruction occupies its GB300 scheduler for 64 clocks (measured,
// whatever the number of active lanes: DFMA and DADD 64, division 670, square
// root 684, a five-step shuffle sum 622), a 32 x 32 + 64 bit integer
// multiply-add for 2.7 to 4.  So the reduction runs on 62-bit integers, whose
// products are 32-bit multiply-adds of two limbs per factor.
//
// A Gram matrix is graded: |A_il| <= sqrt(A_ii A_ll), and eigenvectors of small
// eigenvalues need every entry to that scale's precision, as FP64 keeps it.  Row l
// therefore has an exponent e_l >= 0 that keeps its scaled diagonal at 1/2 or
// below; all quantities below are bounded by that (Cauchy-Schwarz), and with
// F >= |A|_F a power of two their units are (m = min e less guard_bits)
//   entries             A_il 2^(e_i + e_l)                     2^-61 F
//   column              x_l 2^(e_l + c)                        2^-61 F
//   reflector v, |column| scaled to [1/2, 1)                   2^-56
//   product             p_l 2^(e_l + m), p = A v               2^-61 F
//   v^H p               2^(2 m)                                2^-60 F
//   update vectors      v_l 2^(e_l + h - m), h = log2 sqrt(v^H p)   2^-56
//                       w_l 2^(e_l - h + m)                    2^-57 F
// All exponents are zero for a matrix that is not positive semidefinite.
#pragma once

#include "common.cuh"

namespace tn {
namespace fixp {

typedef long long ll;
typedef unsigned long long ull;
typedef __int128 i128;
typedef unsigned __int128 u128;

struct zint {
    ll x, y;
};

#define TN_HD __host__ __device__ __forceinline__

// re = x.hi 2^29 + x.lo with a signed low limb, both parts: (re hi, re lo, im hi, im lo)
TN_HD int4 limbs29(zint v) {
    int4 r;
    const ll hx = (v.x + (1ll << 28)) >> 29, hy = (v.y + (1ll << 28)) >> 29;
    r.x = (int)hx;
    r.y = (int)(v.x - (hx << 29));
    r.z = (int)hy;
    r.w = (int)(v.y - (hy << 29));
    return r;
}
TN_HD zint value29(int4 l) { return zint{((ll)l.x << 29) + l.y, ((ll)l.z << 29) + l.w}; }

TN_HD int4 limbs31(zint v) {
    int4 r;
    const ll hx = (v.x + (1ll << 30)) >> 31, hy = (v.y + (1ll << 30)) >> 31;
    r.x = (int)hx;
    r.y = (int)(v.x - (hx << 31));
    r.z = (int)hy;
    r.w = (int)(v.y - (hy << 31));
    return r;
}

TN_HD ll mw(int a, int b, ll c) { return (ll)a * b + c; }

// a -= w_i conj(v_l) + v_i conj(w_l), rounded to nearest: w limbs 31, v limbs 29,
// product unit 2^-113 F.  High products (2^60) shift by +8 into the entries' unit,
// the two kinds of cross products (2^31, 2^29) by -21 and -23, low ones by -52;
// without the low products an entry is 2^-56 F off in every step.
TN_HD void update(zint& a, int4 wi, int4 vi, int4 wl, int4 vl) {
    ll m = mw(wi.x, vl.x, 0), c1 = mw(wi.x, vl.y, 1ll << 20), c2 = mw(wi.y, vl.x, 0), c3 = mw(wi.y, vl.y, 0);
    m = mw(wi.z, vl.z, m), c1 = mw(wi.z, vl.w, c1), c2 = mw(wi.w, vl.z, c2), c3 = mw(wi.w, vl.w, c3);
    m = mw(vi.x, wl.x, m), c1 = mw(vi.y, wl.x, c1), c2 = mw(vi.x, wl.y, c2), c3 = mw(vi.y, wl.y, c3);
    m = mw(vi.z, wl.z, m), c1 = mw(vi.w, wl.z, c1), c2 = mw(vi.z, wl.w, c2), c3 = mw(vi.w, wl.w, c3);
    a.x -= (ll)((ull)m << 8) + ((c1 + ((c2 + (c3 >> 29)) >> 2)) >> 21);
    m = mw(wi.z, vl.x, 0), c1 = mw(wi.z, vl.y, 1ll << 20), c2 = mw(wi.w, vl.x, 0), c3 = mw(wi.w, vl.y, 0);
    m = mw(-wi.x, vl.z, m), c1 = mw(-wi.x, vl.w, c1), c2 = mw(-wi.y, vl.z, c2), c3 = mw(-wi.y, vl.w, c3);
    m = mw(vi.z, wl.x, m), c1 = mw(vi.w, wl.x, c1), c2 = mw(vi.z, wl.y, c2), c3 = mw(vi.w, wl.y, c3);
    m = mw(-vi.x, wl.z, m), c1 = mw(-vi.y, wl.z, c1), c2 = mw(-vi.x, wl.w, c2), c3 = mw(-vi.y, wl.w, c3);
    a.y -= (ll)((ull)m << 8) + ((c1 + ((c2 + (c3 >> 29)) >> 2)) >> 21);
}

// Running sum of a v over a row: high products (which may wrap: only the final
// sum has to fit), cross products (bounded by Cauchy-Schwarz below 2^63 for
// a 32nd of any row up to 4096 entries) and low products (2^57 an entry whatever the
// row: dot_carry moves their upper part on after at most 32 entries).
struct Dot {
    ll mx, my, cx, cy, lx, ly;
};
TN_HD void dot_add(Dot& s, zint a, int4 v) {
    const int4 l = limbs29(zint{(a.x + 4) >> 3, (a.y + 4) >> 3});  // unit 2^-58 F
    s.mx = mw(l.x, v.x, s.mx), s.cx = mw(l.x, v.y, s.cx), s.cx = mw(l.y, v.x, s.cx), s.lx = mw(l.y, v.y, s.lx);
    s.mx = mw(-l.z, v.z, s.mx), s.cx = mw(-l.z, v.w, s.cx), s.cx = mw(-l.w, v.z, s.cx), s.lx = mw(-l.w, v.w, s.lx);
    s.my = mw(l.x, v.z, s.my), s.cy = mw(l.x, v.w, s.cy), s.cy = mw(l.y, v.z, s.cy), s.ly = mw(l.y, v.w, s.ly);
    s.my = mw(l.z, v.x, s.my), s.cy = mw(l.z, v.y, s.cy), s.cy = mw(l.w, v.x, s.cy), s.ly = mw(l.w, v.y, s.ly);
}
TN_HD void dot_carry(Dot& s) {
    s.cx += s.lx >> 29;
    s.lx &= (1ll << 29) - 1;
    s.cy += s.ly >> 29;
    s.ly &= (1ll << 29) - 1;
}
TN_HD zint dot_value(const Dot& s) {  // unit 2^-61 F
    return zint{(ll)((ull)s.mx << 5) + ((s.cx + (s.lx >> 29) + (1ll << 23)) >> 24),
                (ll)((ull)s.my << 5) + ((s.cy + (s.ly >> 29) + (1ll << 23)) >> 24)};
}

// Limbs of 32 bits: v = hi 2^32 + lo with a signed low limb (|v| < 2^63 - 2^31).
struct limb32 {
    int h, l;
};
TN_HD limb32 split32(ll v) { return limb32{(int)((v + (1ll << 31)) >> 32), (int)v}; }

// Running sum of products a b = m 2^64 + x 2^32 + l; the cross products of a call's
// two terms stay below 2^63 for |a| < 2^61, |b| < 2^62.
struct Prod {
    ll m, x, l;
};
TN_HD Prod mul32(limb32 a, limb32 b) {
    return Prod{mw(a.h, b.h, 0), mw(a.l, b.h, mw(a.h, b.l, 0)), mw(a.l, b.l, 0)};
}
TN_HD Prod mul32(limb32 a, limb32 b, Prod c) {
    return Prod{mw(a.h, b.h, c.m), mw(a.l, b.h, mw(a.h, b.l, c.x)), (mw(a.l, b.l, 0) >> 1) + (c.l >> 1)};
}
// the sum of one product / 2^s, of two / 2^s; 32 < s < 64, rounded
TN_HD ll prod1(const Prod& p, int s) {
    return (ll)((ull)p.m << (64 - s)) + ((p.x + (p.l >> 32) + (1ll << (s - 33))) >> (s - 32));
}
TN_HD ll prod2(const Prod& p, int s) {
    return (ll)((ull)p.m << (64 - s)) + ((p.x + (p.l >> 31) + (1ll << (s - 33))) >> (s - 32));
}

// x 2^s (s negative: rounded), componentwise; zero beyond |s| = 62 (upwards only a
// zero gets there)
struct Shift {
    int l, r;
    ll half;
};
TN_HD Shift shift_by(int s) {
    Shift h;
    h.l = s > 0 ? (s < 63 ? s : 63) : 0;
    h.r = s < 0 ? (s > -63 ? -s : 63) : 0;
    h.half = (1ll << h.r) >> 1 & 0x7fffffffffffffffll;
    return h;
}
TN_HD ll sft(ll x, Shift h) { return (ll)(((ull)x << h.l) + (ull)h.half) >> h.r; }
TN_HD ll sft(ll x, int s) { return sft(x, shift_by(s)); }
TN_HD zint zsft(zint v, int s) {
    const Shift h = shift_by(s);
    return zint{sft(v.x, h), sft(v.y, h)};
}

// p - a b 2^-s for b real (unit 2^-56), s >= 0
TN_HD zint minus_real(zint p, zint a, ll b, int s) {
    const limb32 lb = split32(b);
    const zint t{prod1(mul32(split32(a.x), lb), 56), prod1(mul32(split32(a.y), lb), 56)};
    const zint u = zsft(t, -s);
    return zint{p.x - u.x, p.y - u.y};
}
// Re(conj(v) p), unit 2^-60 F
TN_HD ll re_dot(zint v, zint p) {
    return prod2(mul32(split32(v.x), split32(p.x), mul32(split32(v.y), split32(p.y))), 57);
}

// w = tau p - al v: tau in units of 2^-59, al 2^-57, p 2^-61 F, v 2^-56; w 2^-57 F
TN_HD zint make_w(zint tau, zint p, ll al, zint v) {
    const limb32 tx = split32(tau.x), ty = split32(tau.y), px = split32(p.x), py = split32(p.y), la = split32(al);
    const limb32 ny = split32(-tau.y);  // not ty's limbs negated: the lower one may be -2^31
    return zint{prod2(mul32(tx, px, mul32(ny, py)), 63) - prod1(mul32(split32(v.x), la), 56),
                prod2(mul32(tx, py, mul32(ty, px)), 63) - prod1(mul32(split32(v.y), la), 56)};
}

TN_HD u128 abs2(zint x) {
    const ull a = (ull)(x.x < 0 ? -x.x : x.x), b = (ull)(x.y < 0 ? -x.y : x.y);
    return (u128)a * a + (u128)b * b;
}

TN_HD int bits128(u128 s) {
    const ull h = (ull)(s >> 64), l = (ull)s;
#ifdef __CUDA_ARCH__
    return h ? 128 - __clzll(h) : 64 - __clzll(l);
#else
    return h ? 128 - __builtin_clzll(h) : (l ? 64 - __builtin_clzll(l) : 0);
#endif
}

// Sum of |x_l|^2 2^(56 - 2 d_l), exact: 192 bits, summed across up to 1024 threads as
// nine 22-bit limbs.
struct Norm2 {
    u128 lo;
    ull hi;
};
TN_HD void norm_add(Norm2& s, zint x, int d) {
    const u128 a = abs2(x);
    const int sl = 56 - 2 * d;  // d <= EXP_MAX
    const u128 t = s.lo + (a << sl);
    s.hi += (sl ? (ull)(a >> (128 - sl)) : 0) + (t < s.lo ? 1 : 0);
    s.lo = t;
}
constexpr int NORM_LIMBS = 9;
TN_HD unsigned norm_limb(const Norm2& s, int k) {
    const unsigned m = 0x3fffff;
    if (k < 5) return (unsigned)(s.lo >> (22 * k)) & m;
    if (k == 5) return ((unsigned)(s.lo >> 110) | (unsigned)(s.hi << 18)) & m;
    return (unsigned)(s.hi >> (22 * k - 128)) & m;
}
// From the summed limbs (32 bits each): the sum as top 2^(bl - 64), bl = 0 for zero.
struct NormTop {
    int bl;
    ull top;
};
TN_HD NormTop norm_top(const unsigned* l) {
    u128 L = 0, H = l[8];
#pragma unroll
    for (int k = 3; k >= 0; --k) {
        L = (L << 22) + l[k];
        H = (H << 22) + l[k + 4];
    }
    H += L >> 88;
    L &= (((u128)1) << 88) - 1;
    NormTop r{0, 0};
    const int h = bits128(H);
    if (h >= 64) {
        r.bl = 88 + h;
        r.top = (ull)(H >> (h - 64));
    } else if (h > 0) {
        r.bl = 88 + h;
        r.top = (ull)((H << (64 - h)) | (L >> (24 + h)));
    } else {
        const int b = bits128(L);
        r.bl = b;
        if (b) r.top = (ull)(b >= 64 ? L >> (b - 64) : L << (64 - b));
    }
    return r;
}
// The sum's bit length from limbs k and k - 1 alone: 22 k + that of this, k the
// highest for which it is nonzero (one short where a carry from further below
// reaches a power of two)
TN_HD unsigned norm_carry(unsigned l, unsigned below) { return l + (below >> 22); }

// Shift that takes the column to a norm in [1/2, 1) in the unit 2^-56.  The
// reflector is H = I - tau v v^H with v = column - beta e_1, H^H (column) =
// beta e_1, beta real of the sign opposite to the first entry's real part (LAPACK
// zlarfg's choice), tau = 1 / (beta conj(beta - alpha)).
TN_HD int norm_shift(int bl) { return 56 - ((bl - 56 + 401) / 2 - 200); }

// The new exponent of a row from its scaled diagonal a before the update and the
// float estimates d of 2 Re(w conj v), b of 2 |w||v| and v2 of the larger of |v|^2 and
// 2 |w|^2 in the same scale: unchanged while the larger of the diagonals before and after
// and v2 / 32 lies in [2^-14, 1/2], else such that it is at most 1/4, and never above cap.
// v2 matters where q is below its floor or the row holds rounding errors only.
constexpr int EXP_MAX = 28;   // 2^-56 F on the diagonal
constexpr int EXP_GAIN = 18;  // a row's rounding errors stay 2^-20 of its scale
TN_HD int next_exponent(int e, int cap, float a, float d, float b, float v2) {
    const float est = fmaxf(fmaxf(fabsf(a), fabsf(a - d)), v2 * 0x1p-5f) + 1e-5f * (fabsf(a) + b) + 1e-30f;
    if (est <= 0.5f && est >= 0x1p-14f) return e;
#ifdef __CUDA_ARCH__
    const int l = (int)((__float_as_uint(est) >> 23) & 0xff) - 126;  // est < 2^l
#else
    int l;
    frexpf(est, &l);
#endif
    // a 2^(2 k) <= 1/4: 2 k <= -2 - l
    const int k = (-2 - l) >= 0 ? (-2 - l) / 2 : -((l + 3) / 2);
    const int r = e + k;
    return r < 0 ? 0 : r > cap ? cap : r;
}

TN_HD int bits64(ll x) {  // of |x|
    const ull a = (ull)(x < 0 ? -x : x);
#ifdef __CUDA_ARCH__
    return 64 - __clzll((ll)a);
#else
    return a ? 64 - __builtin_clzll(a) : 0;
#endif
}

// h = log2 sqrt(q) of the largest that v^H A v can be, q in units of 2^-60 and off by
// two of them a row at most (a q that rounds to zero says nothing of p, which is
// bounded by sqrt of the true one), with the floor that rounding errors of the
// product need, from the largest entry 2^vm of v 2^-e.
// Rows' exponents bound the scaled matrix' diagonal, not its norm, which can be the sum of
// n of them; v^H A v 2^(2 m) and the product stay in range with m this much below the
// smallest exponent (4^g >= n / 2, and none where that is zero: |A| is below F).
TN_HD int guard_bits(int n) { return bits64(n - 1) / 2; }
constexpr int Q_FLOOR = 12;
// Where rows hold nothing but rounding errors the matrix is not positive, and p, of at most
// pm bits, has to bound h itself.
TN_HD int q_exponent(ll q, int vm, int pm, int n) {
    const int lo = vm - Q_FLOOR, h = (bits64((q > 0 ? q : 0) + 4ll * n) - 61) >> 1, hp = pm - 62;
    return h > lo ? (h > hp ? h : hp) : lo > hp ? lo : hp;
}
// al = |tau|^2 / 2 q 2^(-2 h), unit 2^-57, from |tau|^2 / 2 in units of 2^-59
TN_HD ll q_scaled(ll c2, ll q, int h) { return prod1(mul32(split32(c2), split32(sft(q, -2 * h))), 62); }

}  // namespace fixp
}  // namespace tn
