// The steps of hetrd_fix_kernel (csrc/hetrd.cu) on the CPU with its arithmetic
// (csrc/fixp.cuh), and their backward error on random positive semidefinite matrices
// of the kinds that truncated splits meet.
//   reduction <order>: n beside s in every other place, s = 10^-2 .. 10^-8, likewise
//   reduction file <path>: a matrix, its order and lower triangle by rows
//   reduction <seed> <matrices> <largest order> <flat>: prints how many are off by more
//   than 64 n 2^-53 of the norm or leave the numbers' range, and the largest error
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "fixp.cuh"

using namespace tn::fixp;
typedef std::complex<double> C;
typedef std::complex<long double> CL;

struct Reduced {
    std::vector<double> d, e;
    std::vector<C> tau, V;  // reflector j in V[j n + j + 1 ..]
    double wmax = 0, pmax = 0, qmax = 0;  // in units whose ranges are 32, 4 and 8
};

static ll fix(double x, int s) { return llrint(std::ldexp(x, s)); }
static double unfix(ll x, int s) { return std::ldexp((double)x, s); }
static zint fix(C x, int s) { return zint{fix(x.real(), s), fix(x.imag(), s)}; }

// G by rows in the order of descending diagonal
static Reduced reduce(const std::vector<C>& G, int n) {
    Reduced r;
    r.d.assign(n, 0);
    r.e.assign(n, 0);
    r.tau.assign(n, 0);
    r.V.assign((size_t)n * n, 0);
    double F2 = 0;
    for (const C& g : G) F2 += std::norm(g);
    int f;
    std::frexp(std::sqrt(F2), &f);
    std::vector<int> e(n), en(n), cap(n), dl(n, 0);
    for (int l = 0; l < n; ++l) {
        e[l] = next_exponent(0, EXP_MAX, (float)std::ldexp(G[l + (size_t)n * l].real(), -f), 0, 0, 0);
        cap[l] = std::min(EXP_MAX, e[l] + EXP_GAIN);
    }
    int em = *std::min_element(e.begin(), e.end()), c = std::max(0, em - 6);
    std::vector<zint> A((size_t)n * n), x(n), p(n), ac(n), vd(n);
    std::vector<int4> w4(n), v4(n);
    std::vector<ll> dg(n);
    for (int i = 0; i < n; ++i)
        for (int l = 0; l < n; ++l) A[(size_t)i * n + l] = fix(G[i + (size_t)n * l], 61 - f + e[i] + e[l]);
    for (int l = 0; l < n; ++l) x[l] = fix(G[l], 61 - f + e[l] + c);
    r.d[0] = unfix(fix(G[0].real(), 61 - f + 2 * c), f - 61 - 2 * c);
    bool pending = false;
    for (int j = 0; j + 1 < n; ++j) {
        const int l0 = j + 1, s0 = e[l0] - em, cn = std::max(0, em - 6), g = std::min(em, guard_bits(n - j));
        Norm2 S{0, 0};
        for (int l = l0; l < n; ++l) norm_add(S, x[l], e[l] - em);
        unsigned limb[NORM_LIMBS];
        for (int k = 0; k < NORM_LIMBS; ++k) limb[k] = norm_limb(S, k);
        int bl = 0;
        for (int k = 0; k < NORM_LIMBS; ++k) {
            const unsigned t = norm_carry(limb[k], k ? limb[k - 1] : 0);
            if (t) bl = 22 * k + 32 - __builtin_clz(t);
        }
        const int sh = bl ? norm_shift(bl) : 0;
        ll beta = 0, c2 = 0;
        zint tau{0, 0}, v1{0, 0};
        if (bl) {
            const NormTop T = norm_top(limb);
            const double s = std::ldexp((double)T.top, T.bl - 64 - 56 + 2 * sh - 112);
            const zint al = zsft(x[l0], sh - s0);
            const double ar = unfix(al.x, -56), ai = unfix(al.y, -56), b = al.x < 0 ? std::sqrt(s) : -std::sqrt(s);
            beta = fix(b, 56);
            v1 = zint{al.x - beta, al.y};
            const double D = s + ar * ar + ai * ai - 2 * b * ar, ri = 1 / (b * D), tr = (b - ar) * ri, ti = -ai * ri;
            tau = zint{fix(tr, 59), fix(ti, 59)};
            c2 = fix(D * ri * ri, 58);
            r.tau[j] = C(tr, ti);
        }
        r.e[j] = unfix(beta, -sh + f - 61 - em - c);
        std::vector<int4> vl(n);
        int vm = -s0 - g;
        for (int l = l0; l < n; ++l) {
            vd[l] = zsft(x[l], sh - 2 * (e[l] - em) - g);
            vl[l] = limbs29(vd[l]);
            const zint v = l == l0 ? v1 : zsft(x[l], sh - (e[l] - em));
            r.V[(size_t)j * n + l] = C(unfix(v.x, -56), unfix(v.y, -56));
            const int bits = std::max(bits64(x[l].x), bits64(x[l].y));
            if (bits) vm = std::max(vm, bits + sh - 2 * (e[l] - em) - g - 56);
        }
        ll q = 0;
        int pm = 0;
        double qd = 0;
        for (int i = l0; i < n; ++i) {
            Dot D{0, 0, 0, 0, 0, 0};
            for (int l = l0; l < n; ++l) {
                zint& a = A[(size_t)i * n + l];
                if (pending) {
                    a = zsft(a, dl[i] + dl[l]);
                    update(a, w4[i], v4[i], w4[l], v4[l]);
                }
                dot_add(D, a, vl[l]);
                if ((l - l0) % 32 == 31) dot_carry(D);
            }
            ac[i] = A[(size_t)i * n + l0];
            p[i] = minus_real(dot_value(D), ac[i], beta, s0 + g);
            dg[i] = A[(size_t)i * n + i].x;
            pm = std::max(pm, std::max(bits64(p[i].x), bits64(p[i].y)));
            const ll t = re_dot(i == l0 ? zsft(v1, -s0 - g) : vd[i], p[i]);
            q += t;
            qd += unfix(t, -60);
            r.pmax = std::max(r.pmax, std::max(std::fabs(unfix(p[i].x, -61)), std::fabs(unfix(p[i].y, -61))));
        }
        r.qmax = std::max(r.qmax, std::fabs(qd));
        const int h = q_exponent(q, vm, pm, n - j);
        const ll al2 = q_scaled(c2, q, h);
        const float tx = (float)unfix(tau.x, -59), ty = (float)unfix(tau.y, -59), fa = (float)unfix(al2, -57),
                    ft = std::fabs(tx) + std::fabs(ty);
        int emn = INT_MAX;
        for (int l = l0; l < n; ++l) {
            const float px = (float)unfix(p[l].x, -61 - h), py = (float)unfix(p[l].y, -61 - h),
                        vx = (float)unfix(x[l].x, sh + h + g - 56), vy = (float)unfix(x[l].y, sh + h + g - 56);
            const float wx = tx * px - ty * py - fa * vx, wy = tx * py + ty * px - fa * vy, av = std::fabs(vx) + std::fabs(vy);
            en[l] = l == l0 ? cn
                            : next_exponent(e[l], cap[l], (float)unfix(dg[l], -61), 2.f * (wx * vx + wy * vy),
                                            2.f * av * (ft * (std::fabs(px) + std::fabs(py)) + fa * av), std::max(vx * vx + vy * vy, 2.f * (wx * wx + wy * wy)));
            dl[l] = en[l] - e[l];
            const zint vt = zsft(l == l0 ? v1 : x[l], (l == l0 ? cn + h - em : sh + h + dl[l]) + g);
            const zint w = make_w(tau, zsft(p[l], dl[l] - h), al2, vt);
            const double lift = std::ldexp(1.0, dl[l] - h - 61);
            r.pmax = std::max(r.pmax, lift * std::max(std::fabs((double)p[l].x), std::fabs((double)p[l].y)));
            r.wmax = std::max(r.wmax, std::max(std::fabs(unfix(w.x, -57)), std::fabs(unfix(w.y, -57))));
            w4[l] = limbs31(w);
            v4[l] = limbs29(vt);
            if (l > l0) emn = std::min(emn, en[l]);
        }
        pending = true;
        for (int l = l0; l < n; ++l) {
            x[l] = zsft(ac[l], dl[l] + dl[l0]);
            update(x[l], w4[l], v4[l], w4[l0], v4[l0]);
        }
        for (int l = l0; l < n; ++l) e[l] = en[l];
        if (emn != INT_MAX) em = emn;
        c = cn;
        r.d[l0] = unfix(x[l0].x, f - 61 - 2 * c);
    }
    return r;
}

// |Q T Q^H - G| over |G|
static double backward(const std::vector<C>& G, int n, const Reduced& r) {
    std::vector<CL> B((size_t)n * n);
    for (size_t t = 0; t < B.size(); ++t) B[t] = CL(G[t].real(), G[t].imag());
    long double nrm = 0, err = 0;
    for (const CL& b : B) nrm += std::norm(b);
    for (int j = 0; j + 1 < n; ++j) {  // H^H B H
        const CL tau(r.tau[j].real(), r.tau[j].imag());
        std::vector<CL> v(n), y(n, 0);
        for (int l = j + 1; l < n; ++l) v[l] = CL(r.V[(size_t)j * n + l].real(), r.V[(size_t)j * n + l].imag());
        for (int l = 0; l < n; ++l)
            for (int i = j + 1; i < n; ++i) y[l] += std::conj(v[i]) * B[i + (size_t)n * l];
        for (int l = 0; l < n; ++l)
            for (int i = j + 1; i < n; ++i) B[i + (size_t)n * l] -= std::conj(tau) * v[i] * y[l];
        std::fill(y.begin(), y.end(), CL(0));
        for (int l = j + 1; l < n; ++l)
            for (int i = 0; i < n; ++i) y[i] += B[i + (size_t)n * l] * v[l];
        for (int l = j + 1; l < n; ++l)
            for (int i = 0; i < n; ++i) B[i + (size_t)n * l] -= tau * y[i] * std::conj(v[l]);
    }
    for (int i = 0; i < n; ++i)
        for (int l = 0; l < n; ++l) {
            const double t = i == l ? r.d[i] : std::abs(i - l) == 1 ? r.e[std::min(i, l)] : 0.0;
            err = std::max(err, std::abs(B[i + (size_t)n * l] - CL(t)));
        }
    return (double)(err / std::sqrt(nrm));
}

static bool off(const Reduced& r, double err, int n) {
    return !(err <= 64 * n * 0x1p-53) || r.wmax > 31 || r.pmax > 3.9 || r.qmax > 7.9;
}

int main(int argc, char** argv) {
    if (argc == 3) {  // a matrix from a file: its order and lower triangle by rows
        FILE* f = std::fopen(argv[2], "r");
        int n = 0;
        if (!f || std::fscanf(f, "%d", &n) != 1) return 1;
        std::vector<C> P((size_t)n * n);
        for (int i = 0; i < n; ++i)
            for (int l = 0; l <= i; ++l) {
                double x, y;
                if (std::fscanf(f, "%la %la", &x, &y) != 2) return 1;
                P[i + (size_t)n * l] = C(x, y);
                P[l + (size_t)n * i] = C(x, -y);
            }
        std::fclose(f);
        const Reduced r = reduce(P, n);
        printf("%d of 1, p %.2f\n", (int)off(r, backward(P, n, r), n), r.pmax);
        return 0;
    }
    if (argc == 2) {
        const int n = std::atoi(argv[1]);
        int bad = 0;
        for (int k = 2; k <= 8; ++k) {
            std::vector<C> P((size_t)n * n, std::pow(10.0, -k));
            for (int i = 1; i < n; ++i) P[i] = P[(size_t)n * i] = 0;
            P[0] = n;
            const Reduced r = reduce(P, n);
            bad += off(r, backward(P, n, r), n);
        }
        printf("%d of 7\n", bad);
        return 0;
    }
    std::mt19937_64 gen(std::atoi(argv[1]));
    const int count = std::atoi(argv[2]), most = std::atoi(argv[3]), flat = argc > 4 ? std::atoi(argv[4]) : 0;
    std::uniform_real_distribution<double> U(0, 1);
    std::normal_distribution<double> N(0, 1);
    auto cn = [&] { return C(N(gen), N(gen)); };
    int bad = 0, done = 0;
    double worst = 0, wmax = 0, pmax = 0, qmax = 0;
    for (int it = 0; it < count; ++it) {
        const int m = 2 + (int)(U(gen) * (most - 1)), n = 1 + (int)(U(gen) * most), kind = (int)(U(gen) * (flat ? 9 : 7));
        std::vector<C> T((size_t)m * n);
        for (C& t : T) t = cn();
        std::vector<int> a(m), b(n);
        for (int& s : a) s = (int)(U(gen) * 3);
        for (int& s : b) s = (int)(U(gen) * 3);
        std::vector<double> rows(m, 1.0), cols(n, 1.0);
        const double dr = 20 * U(gen), dc = 15 * U(gen), fill = U(gen);
        const bool noisy = U(gen) < 0.6;
        const double level = std::pow(10.0, -22 + 7 * U(gen));
        if (kind == 1 || kind == 2 || kind == 4) for (double& s : rows) s = std::pow(10.0, -dr * U(gen));
        if (kind == 2 || kind == 3) for (double& s : cols) s = std::pow(10.0, -dc * U(gen));
        // a large row before many of equal size that are nearly parallel, or graded columns under equal rows
        if (kind == 7) {
            const double low = std::pow(10.0, -1 - 6 * U(gen));
            for (int i = 1; i < m; ++i) rows[i] = low;
        }
        if (kind == 8) for (int k = 0; k < n; ++k) cols[k] = std::pow(10.0, -0.3 * k);
        for (int i = 0; i < m; ++i)
            for (int k = 0; k < n; ++k) {
                C& t = T[i + (size_t)m * k];
                if (kind == 6 && k) t = T[i] * cn();
                if (kind == 7 && i > 1) t = T[1 + (size_t)m * k] / rows[1] + 1e-3 * t;
                t *= rows[i] * cols[k];
                if (kind % 2 == 0 && kind < 6 && a[i] != b[k]) t = 0;
                if (kind == 5 && U(gen) > 0.3) t = 0;
                if (noisy && U(gen) < fill) t += level * std::pow(10.0, -6 * U(gen)) * cn();
            }
        std::vector<C> G((size_t)m * m);
        for (int i = 0; i < m; ++i)
            for (int l = 0; l <= i; ++l) {
                C s = 0;
                for (int k = 0; k < n; ++k) s += T[i + (size_t)m * k] * std::conj(T[l + (size_t)m * k]);
                G[i + (size_t)m * l] = i == l ? C(s.real()) : s;
                G[l + (size_t)m * i] = std::conj(G[i + (size_t)m * l]);
            }
        std::vector<int> perm(m);
        for (int i = 0; i < m; ++i) perm[i] = i;
        std::stable_sort(perm.begin(), perm.end(), [&](int i, int l) { return G[i + (size_t)m * i].real() > G[l + (size_t)m * l].real(); });
        std::vector<C> P((size_t)m * m);
        double top = 0;
        for (int i = 0; i < m; ++i)
            for (int l = 0; l < m; ++l) top = std::max(top, std::abs(P[i + (size_t)m * l] = G[perm[i] + (size_t)m * perm[l]]));
        if (!(top > 1e-280)) continue;
        const Reduced r = reduce(P, m);
        const double err = backward(P, m, r);
        ++done;
        worst = std::max(worst, err / (64 * m * 0x1p-53));
        wmax = std::max(wmax, r.wmax);
        pmax = std::max(pmax, r.pmax);
        qmax = std::max(qmax, r.qmax);
        bad += off(r, err, m);
    }
    printf("%d of %d, worst %.1e of the bound, w %.2f p %.2f q %.2f\n", bad, done, worst, wmax, pmax, qmax);
    return 0;
}
