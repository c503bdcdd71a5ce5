// Gauge moves, two-site splits, environment blocks, the two-site effective
// Hamiltonian product and expectation values on device-resident MPS.
#include <algorithm>
#include <map>
#include <string>
#include "mps.cuh"
#include "mixed.cuh"

namespace tn {

static const cplx ONE = {1.0, 0.0};
static const cplx ZERO = {0.0, 0.0};

// ---- gauge moves (gmps.jl:60-112) -----------------------------------------
// moveright!: SVD with the right bond as columns, M[(Dl,s),Dr]; the isometry
// stays, S*Vt is absorbed into the next site.
void moveright(tn_mps* psi, int idx, const Trunc& t) {
    if (!(0 < idx && idx < psi->N)) return;
    Ctx* ctx = psi->ctx;
    const int d = psi->d;
    const int64_t Dl = psi->dl(idx), Dr = psi->dr(idx), Dr2 = psi->dr(idx + 1);
    DBuf X, Y;
    SplitResult r = trunc_split(ctx, psi->site(idx), Dl * d, Dr, t.cutoff, t.maxdim, t.mindim,
                                true, X, Y, nullptr);
    const int64_t k = r.k;
    DBuf next(ctx, sizeof(cplx) * k * d * Dr2);
    zgemm(ctx, OP_N, OP_N, k, d * Dr2, Dr, ONE, Y.c(), k, 0, psi->site(idx + 1), Dr, 0, ZERO,
          next.c(), k, 0);
    psi->A[idx - 1] = std::move(X);
    psi->A[idx] = std::move(next);
    psi->dims[idx] = k;
}

// moveleft!: SVD with the left bond as columns; the co-isometry stays, U*S is
// absorbed into the previous site.
void moveleft(tn_mps* psi, int idx, const Trunc& t) {
    if (!(1 < idx && idx <= psi->N)) return;
    Ctx* ctx = psi->ctx;
    const int d = psi->d;
    const int64_t Dl = psi->dl(idx), Dr = psi->dr(idx), Dl0 = psi->dl(idx - 1);
    DBuf X, Y;
    SplitResult r = trunc_split(ctx, psi->site(idx), Dl, d * Dr, t.cutoff, t.maxdim, t.mindim,
                                false, X, Y, nullptr);
    const int64_t k = r.k;
    DBuf prev(ctx, sizeof(cplx) * Dl0 * d * k);
    zgemm(ctx, OP_N, OP_N, Dl0 * d, k, Dl, ONE, psi->site(idx - 1), Dl0 * d, 0, X.c(), Dl, 0,
          ZERO, prev.c(), Dl0 * d, 0);
    psi->A[idx - 1] = std::move(Y);
    psi->A[idx - 2] = std::move(prev);
    psi->dims[idx - 1] = k;
}

void movecenter(tn_mps* psi, int idx, const Trunc& t) {
    const int N = psi->N;
    TN_REQUIRE(idx >= 1 && idx <= N, "The index is out of range.");
    if (psi->center == 0) {
        for (int i = 1; i <= idx - 1; ++i) moveright(psi, i, t);
        for (int i = 1; i <= N - idx; ++i) moveleft(psi, N + 1 - i, t);
    } else if (idx > psi->center) {
        for (int i = psi->center; i <= idx - 1; ++i) moveright(psi, i, t);
    } else if (idx < psi->center) {
        const int c = psi->center;
        for (int i = 1; i <= c - idx; ++i) moveleft(psi, c + 1 - i, t);
    }
    psi->center = idx;
}

cplx mps_norm(tn_mps* psi) {
    if (psi->center == 0) movecenter(psi, 1, no_trunc());
    const int c = psi->center;
    const double n2 = znorm2(psi->ctx, psi->site(c), psi->size(c));
    return cmk(sqrt(n2), 0.0);
}

void mps_normalize(tn_mps* psi) {
    if (psi->center == 0) movecenter(psi, 1, no_trunc());
    const cplx n = mps_norm(psi);
    const int c = psi->center;
    zscale(psi->ctx, psi->site(c), psi->size(c), cmk(1.0 / n.x, 0.0));
}

void two_site(tn_mps* psi, int site, DBuf& buf) {
    Ctx* ctx = psi->ctx;
    const int d = psi->d;
    const int64_t Dl = psi->dl(site), Dm = psi->dr(site), Dr = psi->dr(site + 1);
    const size_t need = sizeof(cplx) * Dl * d * d * Dr;
    if (buf.bytes < need) buf = DBuf(ctx, need);
    if (ctx->mixed && Dm >= 64) {
        // mixed-precision sweep: the two-site tensor only seeds the Lanczos
        // solve, so the 3xTF32 tensor-core product is enough
        mixed_gemm(ctx, Dl * d, d * Dr, Dm, psi->site(site), false, psi->site(site + 1), buf.c());
        return;
    }
    zgemm(ctx, OP_N, OP_N, Dl * d, d * Dr, Dm, ONE, psi->site(site), Dl * d, 0,
          psi->site(site + 1), Dm, 0, ZERO, buf.c(), Dl * d, 0);
}

SplitResult replacesites2(tn_mps* psi, const cplx* theta, int site, bool direction, bool normalize,
                          const Trunc& t, std::vector<double>* S) {
    const int d = psi->d;
    const int64_t Dl = psi->dl(site), Dr = psi->dr(site + 1);
    DBuf X, Y;
    SplitResult r = trunc_split(psi->ctx, theta, Dl * d, d * Dr, t.cutoff, t.maxdim, t.mindim,
                                !direction, X, Y, S);
    psi->A[site - 1] = std::move(X);
    psi->A[site] = std::move(Y);
    psi->dims[site] = r.k;
    psi->center = direction ? site : site + 1;
    if (normalize) mps_normalize(psi);
    return r;
}

void replacesite1(tn_mps* psi, DBuf&& A, int site, bool direction, bool normalize) {
    psi->A[site - 1] = std::move(A);
    const int nxt = site + 1 - 2 * (direction ? 1 : 0);
    if (0 < nxt && nxt <= psi->N) movecenter(psi, nxt, no_trunc());
    if (normalize) mps_normalize(psi);
}

std::vector<double> singular_values(tn_mps* psi, int site) {
    movecenter(psi, site, no_trunc());
    Ctx* ctx = psi->ctx;
    const int64_t m = psi->dl(site) * psi->d, n = psi->dr(site);
    DBuf X, Y;
    std::vector<double> S;
    trunc_split(ctx, psi->site(site), m, n, 0.0, 0, 1, m <= n, X, Y, &S);
    return S;
}

// ---- environment blocks (projmps.jl:50-95) ---------------------------------
void env_left(Ctx* ctx, const cplx* L, int64_t ca, int64_t wl, int64_t cb, const cplx* A,
              int64_t ca2, const tn_mpo* H, int site, const cplx* B, int64_t cb2, int d, cplx* out) {
    if (!H) {
        cplx* X = ctx->s_t1.c(ctx, (size_t)ca * d * cb2);
        zgemm(ctx, OP_N, OP_N, ca, d * cb2, cb, ONE, L, ca, 0, B, cb, 0, ZERO, X, ca, 0);
        zgemm(ctx, OP_C, OP_N, ca2, cb2, ca * d, ONE, A, ca * d, 0, X, ca * d, 0, ZERO, out, ca2, 0);
        return;
    }
    const int64_t wr = H->w[site];
    cplx* X = ctx->s_t1.c(ctx, (size_t)ca * wl * d * cb2);
    cplx* Y = ctx->s_t2.c(ctx, (size_t)ca * d * wr * cb2);
    zgemm(ctx, OP_N, OP_N, ca * wl, d * cb2, cb, ONE, L, ca * wl, 0, B, cb, 0, ZERO, X, ca * wl, 0);
    small_apply(ctx, X, Y, H->Ml[site - 1].c(), (int)(wl * d), (int)(d * wr), ca, cb2, ca,
                ca * wl * d, ca, ca * d * wr);
    zgemm(ctx, OP_C, OP_N, ca2, wr * cb2, ca * d, ONE, A, ca * d, 0, Y, ca * d, 0, ZERO, out, ca2, 0);
}

void env_right(Ctx* ctx, const cplx* R, int64_t ca2, int64_t wr, int64_t cb2, const cplx* A,
               int64_t ca, const tn_mpo* H, int site, const cplx* B, int64_t cb, int d, cplx* out) {
    if (!H) {
        cplx* Z = ctx->s_t1.c(ctx, (size_t)ca * d * cb2);
        zgemm(ctx, OP_R, OP_N, ca * d, cb2, ca2, ONE, A, ca * d, 0, R, ca2, 0, ZERO, Z, ca * d, 0);
        zgemm(ctx, OP_N, OP_T, ca, cb, d * cb2, ONE, Z, ca, 0, B, cb, 0, ZERO, out, ca, 0);
        return;
    }
    const int64_t wl = H->w[site - 1];
    cplx* Z = ctx->s_t1.c(ctx, (size_t)ca * d * wr * cb2);
    cplx* Z2 = ctx->s_t2.c(ctx, (size_t)ca * wl * d * cb2);
    zgemm(ctx, OP_R, OP_N, ca * d, wr * cb2, ca2, ONE, A, ca * d, 0, R, ca2, 0, ZERO, Z, ca * d, 0);
    small_apply(ctx, Z, Z2, H->Mr[site - 1].c(), (int)(d * wr), (int)(wl * d), ca, cb2, ca,
                ca * d * wr, ca, ca * wl * d);
    zgemm(ctx, OP_N, OP_T, ca * wl, cb, d * cb2, ONE, Z2, ca * wl, 0, B, cb, 0, ZERO, out, ca * wl, 0);
}

// out[a,s1',s2',c'] = sum L[a,w,b] W12[(w,s1,s2),(s1',s2',w'')] th[b,s1,s2,c] R[c',w'',c]
// as L*theta (GEMM), the W12 leg (small_apply), then *R^T (GEMM).
void heff2_fp64(Ctx* ctx, const cplx* L, const cplx* W12, const cplx* R, int64_t cl, int64_t cr,
                int d, int64_t wl, int64_t wr, const cplx* theta, cplx* out) {
    const int64_t d2 = (int64_t)d * d;
    cplx* T1 = ctx->s_t1.c(ctx, (size_t)cl * wl * d2 * cr);
    cplx* T2 = ctx->s_t2.c(ctx, (size_t)cl * d2 * wr * cr);
    zgemm(ctx, OP_N, OP_N, cl * wl, d2 * cr, cl, ONE, L, cl * wl, 0, theta, cl, 0, ZERO, T1,
          cl * wl, 0);
    small_apply(ctx, T1, T2, W12, (int)(wl * d2), (int)(d2 * wr), cl, cr, cl, cl * wl * d2, cl,
                cl * d2 * wr);
    zgemm(ctx, OP_N, OP_T, cl * d2, cr, wr * cr, ONE, T2, cl * d2, 0, R, cr, 0, ZERO, out, cl * d2, 0);
}

// ---- operators on the physical leg ------------------------------------------
std::vector<const cplx*> upload_op_matrices(Ctx* ctx, const double* ops, size_t n, int d, DBuf& out) {
    // small_apply form M[I=i, J=o] = op[o, i]; equal operators share one
    const size_t dd = (size_t)d * d;
    std::vector<cplx> M;
    std::vector<size_t> at(n);
    std::map<std::string, size_t> seen;  // by their bytes
    for (size_t t = 0; t < n; ++t) {
        const double* op = ops + 2 * dd * t;
        const auto f = seen.emplace(std::string(reinterpret_cast<const char*>(op), sizeof(cplx) * dd), M.size());
        at[t] = f.first->second;
        if (!f.second) continue;
        for (int o = 0; o < d; ++o)
            for (int i = 0; i < d; ++i) {
                const double* e = op + 2 * (o + (size_t)d * i);
                M.resize(M.size() + 1);
                M.back() = cmk(e[0], e[1]);
            }
    }
    std::vector<const cplx*> p(n);
    if (n == 0) return p;
    out = DBuf(ctx, sizeof(cplx) * M.size());
    TN_CHECK_CUDA(cudaMemcpyAsync(out.p, M.data(), sizeof(cplx) * M.size(), cudaMemcpyHostToDevice,
                                  ctx->stream));
    ctx->sync();
    for (size_t t = 0; t < n; ++t) p[t] = out.c() + at[t];
    return p;
}

void upload_op_matrix(Ctx* ctx, const double* op, int d, DBuf& out) { upload_op_matrices(ctx, op, 1, d, out); }

void apply_site_op(tn_mps* psi, int site, const cplx* M) {
    Ctx* ctx = psi->ctx;
    const int d = psi->d;
    const int64_t Dl = psi->dl(site), Dr = psi->dr(site);
    DBuf out(ctx, sizeof(cplx) * Dl * d * Dr);
    small_apply(ctx, psi->site(site), out.c(), M, d, d, Dl, Dr, Dl, Dl * d, Dl, Dl * d);
    psi->A[site - 1] = std::move(out);
}

// ---- expectation values (mps.jl:87-134) ------------------------------------
// A term is <bra| op_1 .. op_len |ket>: the left block of its first site with op_1,
// against the right block of its last site with op_len (or that of the next site,
// for one operator).  All blocks of a site come from one pair of products: the
// left block's second factor is the site's bra tensor beside copies with each
// operator applied, the right block's the ket tensor likewise.  A launch makes the
// copies of all sites, another all terms' sums.  Per term and site it took an
// operator, two products and a dot; 10 sites of bond dimension 8 with 47 terms: 309
// launches, 42 now, 2.22 ms -> 0.39; 64 sites of 128 with 317: 41.3 -> 7.6 ms.

struct StackTask {  // one operator's copy of one tensor
    const cplx* T;   // [l, d, r]
    const cplx* M;   // M[I + d J] = op[J, I], null: the tensor itself
    cplx* out;
    int64_t l, r, ldl;  // rows a block of the output is apart: l d, or the stack's height
    int adjoint;        // sum_J conj(op[J, s]) T[., J, .] (bra), else sum_I op[s, I] T[., I, .]
};

__global__ void __launch_bounds__(128) stack_ops_kernel(const StackTask* __restrict__ tasks, int d) {
    const StackTask k = tasks[blockIdx.y];
    const int64_t total = k.l * d * k.r;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = i % k.l, c = i / k.l / d;
        const int s = (int)(i / k.l % d);
        const cplx* t = k.T + a + k.l * d * c;
        cplx v;
        if (!k.M) {
            v = t[k.l * s];
        } else {
            v = cmk(0, 0);
            for (int q = 0; q < d; ++q)
                v = cfma(t[k.l * q], k.adjoint ? cconj(k.M[s + d * q]) : k.M[q + d * s], v);
        }
        k.out[a + k.ldl * (s + d * c)] = v;
    }
}

struct DotTask {  // sum of x[i + ldx j] y[i + rows j]
    const cplx *x, *y;
    int64_t ldx, rows, n;
};

__global__ void __launch_bounds__(128) term_dots_kernel(const DotTask* __restrict__ tasks, cplx* __restrict__ part) {
    const DotTask k = tasks[blockIdx.y];
    cplx s = cmk(0, 0);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < k.n; i += (int64_t)gridDim.x * blockDim.x)
        s = cfma(k.x[i % k.rows + k.ldx * (i / k.rows)], k.y[i], s);
    __shared__ cplx red[4];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s.x += __shfl_down_sync(0xffffffffu, s.x, o);
        s.y += __shfl_down_sync(0xffffffffu, s.y, o);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0)
        part[blockIdx.x + (int64_t)gridDim.x * blockIdx.y] = cadd(cadd(red[0], red[1]), cadd(red[2], red[3]));
}

// Term by term, for blocks too large to keep all of them.
static std::vector<cplx> inner_terms_serial(Ctx* ctx, const tn_mps* bra, const tn_mps* ket,
                                            const std::vector<Term>& terms) {
    const int N = ket->N, d = ket->d;
    // right overlap blocks: R[i] is the block from site i (i = N+1 is the edge)
    std::vector<DBuf> R(N + 2);
    std::vector<int64_t> ra(N + 2, 1), rb(N + 2, 1);
    R[N + 1] = DBuf(ctx, sizeof(cplx));
    zfill(ctx, R[N + 1].c(), 1, ONE);
    for (int i = N; i >= 2; --i) {
        ra[i] = bra->dl(i);
        rb[i] = ket->dl(i);
        R[i] = DBuf(ctx, sizeof(cplx) * ra[i] * rb[i]);
        env_right(ctx, R[i + 1].c(), ra[i + 1], 1, rb[i + 1], bra->site(i), ra[i], nullptr, i,
                  ket->site(i), rb[i], d, R[i].c());
    }
    DBuf out(ctx, sizeof(cplx) * std::max<size_t>(terms.size(), 1));
    DBuf L(ctx, sizeof(cplx)), Lt1, Lt2, B;
    zfill(ctx, L.c(), 1, ONE);
    int64_t la = 1, lb = 1;
    std::vector<std::vector<size_t>> by_site(N + 1);
    for (size_t t = 0; t < terms.size(); ++t) {
        by_site[terms[t].first].push_back(t);
    }
    for (int site = 1; site <= N; ++site) {
        for (size_t t : by_site[site]) {
            const Term& T = terms[t];
            int64_t ta = la, tb = lb;
            const cplx* cur = L.c();
            for (int j = 0; j < T.len; ++j) {
                const int s = site + j;
                const int64_t Dl = ket->dl(s), Dr = ket->dr(s);
                const size_t nb = sizeof(cplx) * Dl * d * Dr;
                if (B.bytes < nb) B = DBuf(ctx, nb);
                small_apply(ctx, ket->site(s), B.c(), T.dops[j], d, d, Dl, Dr, Dl, Dl * d, Dl, Dl * d);
                DBuf& dst = (j % 2 == 0) ? Lt1 : Lt2;
                const size_t nl = sizeof(cplx) * bra->dr(s) * Dr;
                if (dst.bytes < nl) dst = DBuf(ctx, nl);
                env_left(ctx, cur, ta, 1, tb, bra->site(s), bra->dr(s), nullptr, s, B.c(), Dr, d,
                         dst.c());
                cur = dst.c();
                ta = bra->dr(s);
                tb = Dr;
            }
            const int rs = site + T.len;
            bilinear_dot(ctx, cur, R[rs].c(), ta * tb, out.c() + t);
        }
        DBuf Ln(ctx, sizeof(cplx) * bra->dr(site) * ket->dr(site));
        env_left(ctx, L.c(), la, 1, lb, bra->site(site), bra->dr(site), nullptr, site,
                 ket->site(site), ket->dr(site), d, Ln.c());
        L = std::move(Ln);
        la = bra->dr(site);
        lb = ket->dr(site);
    }
    std::vector<cplx> res(terms.size());
    if (!terms.empty()) {
        TN_CHECK_CUDA(cudaMemcpyAsync(res.data(), out.p, sizeof(cplx) * res.size(),
                                      cudaMemcpyDeviceToHost, ctx->stream));
    }
    ctx->sync();
    for (size_t t = 0; t < terms.size(); ++t) res[t] = cmul(terms[t].coeff, res[t]);
    return res;
}

static std::vector<cplx> inner_terms_blocks(Ctx* ctx, const tn_mps* bra, const tn_mps* ket,
                                            const std::vector<Term>& terms) {
    const int N = ket->N, d = ket->d;
    // the operators that a term starts or, from two on, ends with, by site
    std::vector<std::vector<const cplx*>> lops(N + 2), rops(N + 2);
    auto index = [](std::vector<const cplx*>& v, const cplx* op) {
        const auto it = std::find(v.begin(), v.end(), op);
        if (it != v.end()) return (int64_t)(it - v.begin()) + 1;
        v.push_back(op);
        return (int64_t)v.size();
    };
    std::vector<int64_t> li(terms.size()), ri(terms.size(), 0);
    int first_last = N + 1, last_first = 0;
    for (size_t t = 0; t < terms.size(); ++t) {
        const Term& T = terms[t];
        TN_REQUIRE(T.first >= 1 && T.first + T.len - 1 <= N && T.len >= 1, "term sites out of range");
        li[t] = index(lops[T.first], T.dops[0]);
        if (T.len > 1) ri[t] = index(rops[T.first + T.len - 1], T.dops[T.len - 1]);
        first_last = std::min(first_last, T.len > 1 ? T.first + T.len - 1 : T.first + 1);
        last_first = std::max(last_first, T.first);
    }
    std::vector<cplx> res(terms.size());
    if (terms.empty()) return res;
    // left blocks are ca2 (1 + operators) x cb2, right blocks ca x cb (1 + operators)
    auto nl = [&](int i) { return (int64_t)lops[i].size() + 1; };
    auto nr = [&](int i) { return (int64_t)rops[i].size() + 1; };
    auto lbytes = [&](int i) { return sizeof(cplx) * nl(i) * bra->dr(i) * ket->dr(i); };
    auto rbytes = [&](int i) { return sizeof(cplx) * nr(i) * bra->dl(i) * ket->dl(i); };
    size_t bytes = 0;
    for (int i = 1; i <= N; ++i)
        bytes += lbytes(i) + rbytes(i) + sizeof(cplx) * (nl(i) * bra->size(i) + nr(i) * ket->size(i));
    if (bytes > ((size_t)1 << 30)) return inner_terms_serial(ctx, bra, ket, terms);

    // tensors with their operators
    std::vector<DBuf> WL(N + 1), WR(N + 1), L(N + 1), R(N + 2);
    std::vector<StackTask> st;
    int64_t most = 1;
    for (int i = 1; i <= N; ++i) {
        if (nl(i) > 1) {
            WL[i] = DBuf(ctx, sizeof(cplx) * nl(i) * bra->size(i));
            for (int64_t k = 0; k < nl(i); ++k)
                st.push_back({bra->site(i), k ? lops[i][k - 1] : nullptr, WL[i].c() + k * bra->size(i), bra->dl(i),
                              bra->dr(i), bra->dl(i), 1});
            most = std::max(most, bra->size(i));
        }
        if (nr(i) > 1) {
            WR[i] = DBuf(ctx, sizeof(cplx) * nr(i) * ket->size(i));
            for (int64_t k = 0; k < nr(i); ++k)
                st.push_back({ket->site(i), k ? rops[i][k - 1] : nullptr, WR[i].c() + k * ket->dl(i), ket->dl(i),
                              ket->dr(i), nr(i) * ket->dl(i), 0});
            most = std::max(most, ket->size(i));
        }
    }
    // The kernels' tasks go up by copies on the stream, the sums come back by the
    // kernel's stores.
    int64_t parts = 1;
    for (int i = 1; i <= N; ++i)
        parts = std::max(parts, std::min<int64_t>((bra->dr(i) * ket->dr(i) + 1023) / 1024, 16));
    const size_t nsum = 2 * (size_t)parts * terms.size();  // first: its stores need 16 bytes' alignment
    double* h = ctx->pinned(nsum + (sizeof(StackTask) * st.size() + sizeof(DotTask) * terms.size()) / sizeof(double));
    const cplx* sums = reinterpret_cast<const cplx*>(h);
    StackTask* hst = reinterpret_cast<StackTask*>(h + nsum);
    DotTask* hdt = reinterpret_cast<DotTask*>(hst + st.size());
    std::copy(st.begin(), st.end(), hst);
    unset(h, nsum);
    DBuf dst(ctx, sizeof(StackTask) * st.size()), ddt(ctx, sizeof(DotTask) * terms.size());
    TN_CHECK_CUDA(cudaMemcpyAsync(dst.p, hst, dst.bytes, cudaMemcpyHostToDevice, ctx->stream));
    for (size_t t = 0; t < st.size(); t += 65535) {
        const dim3 g((unsigned)std::min<int64_t>((most + 127) / 128, 64), (unsigned)std::min<size_t>(st.size() - t, 65535));
        stack_ops_kernel<<<g, 128, 0, ctx->stream>>>(dst.as<const StackTask>() + t, d);
        ctx->count();
    }
    TN_CHECK_CUDA(cudaGetLastError());

    // right blocks, from the last site to the first that a term needs
    R[N + 1] = DBuf(ctx, sizeof(cplx));
    zfill(ctx, R[N + 1].c(), 1, ONE);
    for (int i = N; i >= std::max(first_last, 2); --i) {
        const int64_t ca = bra->dl(i), cb = ket->dl(i), ca2 = bra->dr(i), cb2 = ket->dr(i), q = nr(i);
        cplx* Z = ctx->s_t1.c(ctx, (size_t)ca * d * cb2);
        zgemm(ctx, OP_R, OP_N, ca * d, cb2, ca2, ONE, bra->site(i), ca * d, 0, R[i + 1].c(), ca2, 0, ZERO, Z, ca * d, 0);
        R[i] = DBuf(ctx, rbytes(i));
        zgemm(ctx, OP_N, OP_T, ca, q * cb, d * cb2, ONE, Z, ca, 0, q > 1 ? WR[i].c() : ket->site(i), q * cb, 0, ZERO,
              R[i].c(), ca, 0);
    }
    // left blocks
    DBuf edge(ctx, sizeof(cplx));
    zfill(ctx, edge.c(), 1, ONE);
    for (int i = 1; i <= last_first; ++i) {
        const int64_t ca = bra->dl(i), cb = ket->dl(i), ca2 = bra->dr(i), cb2 = ket->dr(i), q = nl(i);
        const cplx* P = i > 1 ? L[i - 1].c() : edge.c();
        cplx* X = ctx->s_t1.c(ctx, (size_t)ca * d * cb2);
        zgemm(ctx, OP_N, OP_N, ca, d * cb2, cb, ONE, P, i > 1 ? nl(i - 1) * ca : 1, 0, ket->site(i), cb, 0, ZERO, X, ca, 0);
        L[i] = DBuf(ctx, lbytes(i));
        zgemm(ctx, OP_C, OP_N, q * ca2, cb2, ca * d, ONE, q > 1 ? WL[i].c() : bra->site(i), ca * d, 0, X, ca * d, 0,
              ZERO, L[i].c(), q * ca2, 0);
    }
    // sums; terms of three operators and more go on from their left block first
    std::vector<DBuf> mid;
    DBuf B;
    for (size_t t = 0; t < terms.size(); ++t) {
        const Term& T = terms[t];
        const int s = T.first, e = s + T.len - 1;
        int64_t ta = bra->dr(s), tb = ket->dr(s);
        DotTask k;
        k.x = L[s].c() + li[t] * ta;
        k.ldx = nl(s) * ta;
        if (T.len > 2) {
            DBuf cur(ctx, sizeof(cplx) * ta * tb);
            TN_CHECK_CUDA(cudaMemcpy2DAsync(cur.p, sizeof(cplx) * ta, k.x, sizeof(cplx) * k.ldx, sizeof(cplx) * ta, tb,
                                            cudaMemcpyDeviceToDevice, ctx->stream));
            for (int j = s + 1; j < e; ++j) {
                const int64_t Dl = ket->dl(j), Dr = ket->dr(j);
                if (B.bytes < sizeof(cplx) * Dl * d * Dr) B = DBuf(ctx, sizeof(cplx) * Dl * d * Dr);
                small_apply(ctx, ket->site(j), B.c(), T.dops[j - s], d, d, Dl, Dr, Dl, Dl * d, Dl, Dl * d);
                DBuf nx(ctx, sizeof(cplx) * bra->dr(j) * Dr);
                env_left(ctx, cur.c(), ta, 1, tb, bra->site(j), bra->dr(j), nullptr, j, B.c(), Dr, d, nx.c());
                cur = std::move(nx);
                ta = bra->dr(j);
                tb = Dr;
            }
            k.x = cur.c();
            k.ldx = ta;
            mid.push_back(std::move(cur));
        }
        k.y = T.len == 1 ? R[s + 1].c() : R[e].c() + ri[t] * ta * tb;
        k.rows = ta;
        k.n = ta * tb;
        hdt[t] = k;
    }
    TN_CHECK_CUDA(cudaMemcpyAsync(ddt.p, hdt, ddt.bytes, cudaMemcpyHostToDevice, ctx->stream));
    for (size_t t = 0; t < terms.size(); t += 65535) {
        term_dots_kernel<<<dim3((unsigned)parts, (unsigned)std::min<size_t>(terms.size() - t, 65535)), 128, 0, ctx->stream>>>(
            ddt.as<const DotTask>() + t, reinterpret_cast<cplx*>(h) + parts * t);
        ctx->count();
    }
    TN_CHECK_CUDA(cudaGetLastError());
    ctx->sync();
    check_set(h, nsum);
    for (size_t t = 0; t < terms.size(); ++t) {
        cplx v = sums[parts * t];
        for (int64_t k = 1; k < parts; ++k) v = cadd(v, sums[parts * t + k]);
        res[t] = cmul(terms[t].coeff, v);
    }
    return res;
}

std::vector<cplx> inner_terms(Ctx* ctx, const tn_mps* bra, const tn_mps* ket,
                              const std::vector<Term>& terms) {
    TN_REQUIRE(bra->N == ket->N && bra->d == ket->d, "GMPS must share the same properties.");
    try {
        return inner_terms_blocks(ctx, bra, ket, terms);
    } catch (const Error& e) {
        if (e.code != TN_ERR_OOM) throw;
    }
    return inner_terms_serial(ctx, bra, ket, terms);  // no room for all blocks at once
}

}  // namespace tn
