// Adjoint entry points: parameter gradients of E0 and of the Green functions.
//
// E0: Hellmann-Feynman, dE0/dtheta = <psi|dH/dtheta|psi>.
// G:  G_c(z) = b1^2 [ (z - ph (T - E0))^-1 ]_11 with T the Lanczos tridiagonal
//     of the start vector phi = C|psi> (compute_dynamic_cpu,
//     green_class_compute_dynamic.f90:191-334; b1 = |phi|).  The gradient is
//     taken exactly for the K-step recurrence (one_step_Lanczos_fast,
//     Lanczos_plain.f90:247-302):
//       w_k = H v_k - b_k v_{k-1},  a_k = <w_k, v_k>,  r_k = w_k - a_k v_k,
//       b_{k+1} = |r_k|,  v_{k+1} = r_k / b_{k+1}.
//     The continued fraction's vector-Jacobian product gives abar_k, bbar_k
//     and E0bar; the recurrence is then reversed step by step
//     (one H*w product and one bilinear <wbar_k|dH|v_k> per step), with the
//     Lanczos vectors recomputed from checkpoints every m steps (m ~ sqrt(2K)).
//     The start-vector cotangent goes back through C^T (the same c/c+ map with
//     dagger flipped) to psibar.
// psi: psi is the normalised lowest eigenvector; its cotangent psibar adds
//     -<lambda|dH/dtheta|psi> with (H - E0) lambda = (1 - |psi><psi|) psibar,
//     solved by conjugate gradients on the complement of psi.
// All vectors and arithmetic are FP64.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <vector>

#include "edk_grad.h"
#include "edk_internal.h"

extern "C" {
cudaStream_t edk_internal_stream(edk_ctx *ctx);
int edk_internal_fail(edk_ctx *ctx, int code, const char *msg);
void edk_internal_count(edk_ctx *ctx, int64_t h2d, int64_t d2h);
edk_ctx *edk_internal_h_ctx(edk_h *h);
void edk_internal_h_info(const edk_h *h, int *nc, int *nb, int *nup, int *ndn);
void edk_internal_add_launches(edk_ctx *ctx, int64_t n);
int edk_internal_h_sibling(edk_h *h, int nup, int ndn, edk_h **out);
const uint64_t *edk_internal_h_states(const edk_h *h, int spin);
int edk_internal_h_is_sz(const edk_h *h);
const int32_t *edk_internal_h_rank(const edk_h *h);
cudaMemPool_t edk_internal_pool(edk_ctx *ctx);
int edk_internal_pinned(edk_ctx *ctx, size_t doubles, double **buf, cudaEvent_t *ev);
}

using namespace edk;

namespace {

// Device memory from the context's stream-ordered pool (plain memory without one).
struct DBuf {
    void *p = nullptr;
    cudaStream_t st = nullptr;
    bool pooled = false;
    DBuf() = default;
    DBuf(size_t bytes, edk_ctx *ctx) : st(edk_internal_stream(ctx))
    {
        if (!bytes) bytes = 16;
        const cudaMemPool_t pool = edk_internal_pool(ctx);
        pooled = pool != nullptr;
        const cudaError_t e = pooled ? cudaMallocFromPoolAsync(&p, bytes, pool, st) : cudaMalloc(&p, bytes);
        if (e != cudaSuccess) {
            (void)cudaGetLastError();
            p = nullptr;
        }
    }
    DBuf(DBuf &&o) noexcept : p(o.p), st(o.st), pooled(o.pooled) { o.p = nullptr; }
    DBuf &operator=(DBuf &&o) noexcept
    {
        std::swap(p, o.p);
        std::swap(st, o.st);
        std::swap(pooled, o.pooled);
        return *this;
    }
    DBuf(const DBuf &) = delete;
    ~DBuf()
    {
        if (p && pooled) cudaFreeAsync(p, st);
        else if (p) cudaFree(p);
    }
    double *d() const { return static_cast<double *>(p); }
};

// After a call: the pool keeps what it held before it, or up to 1 GB.
struct PoolGuard {
    edk_ctx *ctx;
    cudaMemPool_t pool;
    uint64_t before = 0;
    explicit PoolGuard(edk_ctx *c) : ctx(c), pool(edk_internal_pool(c))
    {
        if (pool) cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &before);
    }
    ~PoolGuard()
    {
        uint64_t now = 0;
        if (!pool || cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &now) != cudaSuccess) return;
        const uint64_t keep = std::max<uint64_t>(before, (uint64_t)1 << 30);
        if (now > keep && cudaStreamSynchronize(edk_internal_stream(ctx)) == cudaSuccess)
            cudaMemPoolTrimTo(pool, (size_t)keep);
    }
};

struct HDel {
    void operator()(edk_h *h) const { if (h) edk_h_destroy(h); }
};
using HPtr = std::unique_ptr<edk_h, HDel>;

// Jordan-Wigner sign of moving one electron between orbitals a and b of the
// same spin: parity of the occupied orbitals strictly between them.
int hop_sign(uint64_t s, int a, int b)
{
    const int lo = a < b ? a : b, hi = a < b ? b : a;
    if (hi - lo < 2) return 1;
    const uint64_t mask = ((1ull << hi) - 1ull) & ~((1ull << (lo + 1)) - 1ull);
    return (__builtin_popcountll(s & mask) & 1) ? -1 : 1;
}

// Per-sector device data of the parameter operators and the reduction scratch.
struct Ops {
    edk_ctx *ctx = nullptr;
    cudaStream_t st = nullptr;
    int64_t dup = 0, ddn = 0, dim = 0;
    int np = 0, grid = 0;
    DBuf tables, scratch;       // parameters, spin states and hop maps in one upload
    const uint32_t *st_up = nullptr, *st_dn = nullptr;
    const ParamDev *params = nullptr;
    double *partials = nullptr, *out = nullptr;
    unsigned *counter = nullptr;
    int fail(int code, const char *msg) { return edk_internal_fail(ctx, code, msg); }
    int cuda(cudaError_t e, const char *where)
    {
        if (e == cudaSuccess) return EDK_OK;
        char buf[256];
        snprintf(buf, sizeof buf, "%s: %s", where, cudaGetErrorString(e));
        return fail(e == cudaErrorMemoryAllocation ? EDK_ERR_NOMEM : EDK_ERR_CUDA, buf);
    }
};

// Map of the symmetric hop c+_p c_q + c+_q c_p on one spin's basis:
// (rank of the target + 1) * sign, 0 where the hop does not apply.
void hop_map(const uint64_t *states, const int32_t *rank, int64_t n, int p, int q, int32_t *map)
{
    const uint64_t bp = 1ull << p, bq = 1ull << q;
    for (int64_t i = 0; i < n; ++i) {
        const uint64_t s = states[i];
        const bool hp = (s & bp) != 0, hq = (s & bq) != 0;
        map[i] = hp == hq ? 0 : (rank[s ^ bp ^ bq] + 1) * hop_sign(s, p, q);
    }
}

int ops_setup(edk_h *h, int np, const edk_param *prm, Ops &o)
{
    o.ctx = edk_internal_h_ctx(h);
    o.st = edk_internal_stream(o.ctx);
    if (np < 1 || np > kMaxGradParams || !prm) return o.fail(EDK_ERR_INVALID, "1..64 parameters");
    if (edk_internal_h_is_sz(h)) return o.fail(EDK_ERR_UNSUPPORTED, "parameter gradients of a Nambu sector");
    int nc, nb, nup, ndn;
    edk_internal_h_info(h, &nc, &nb, &nup, &ndn);
    edk_h_dims(h, &o.dim, &o.dup, &o.ddn);
    o.np = np;
    const int ns = nc + nb;
    if (ns > 32) return o.fail(EDK_ERR_UNSUPPORTED, "gradients need at most 32 orbitals per spin");
    const uint64_t *su = edk_internal_h_states(h, 0), *sd = edk_internal_h_states(h, 1);
    const int32_t *rank = edk_internal_h_rank(h);
    int rc;
    // words of the upload: the parameters, the spin states, then the maps
    const size_t pw = sizeof(ParamDev) / 4 * (size_t)np;
    std::vector<uint32_t> up(pw);
    up.insert(up.end(), su, su + o.dup);
    up.insert(up.end(), sd, sd + o.ddn);
    std::vector<ParamDev> pd(np);
    std::vector<size_t> at[2] = {std::vector<size_t>(np, 0), std::vector<size_t>(np, 0)};
    for (int q = 0; q < np; ++q) {
        const edk_param &p = prm[q];
        ParamDev &d = pd[q];
        d.mapu = d.mapd = nullptr;
        d.bq = 0;
        int a = -1, b = -1;
        if (p.kind == EDK_PARAM_EC) {
            if (p.i < 0 || p.i >= nc || p.j < 0 || p.j >= nc) return o.fail(EDK_ERR_INVALID, "Ec index");
            a = nb + p.i; b = nb + p.j;
        } else if (p.kind == EDK_PARAM_EB) {
            if (p.i < 0 || p.i >= nb || p.j < 0 || p.j >= nb) return o.fail(EDK_ERR_INVALID, "Eb index");
            a = p.i; b = p.j;
        } else if (p.kind == EDK_PARAM_VBC) {
            if (p.i < 0 || p.i >= nb || p.j < 0 || p.j >= nc) return o.fail(EDK_ERR_INVALID, "Vbc index");
            a = p.i; b = nb + p.j;
        } else if (p.kind == EDK_PARAM_U) {
            if (p.i < 0 || p.i >= nc || p.j < 0 || p.j >= nc) return o.fail(EDK_ERR_INVALID, "U index");
            a = nb + std::min(p.i, p.j); b = nb + std::max(p.i, p.j);
        } else {
            return o.fail(EDK_ERR_INVALID, "parameter kind");
        }
        if (p.kind != EDK_PARAM_U && (p.spin < 0 || p.spin > 2)) return o.fail(EDK_ERR_INVALID, "parameter spin");
        d.spin_mask = p.kind == EDK_PARAM_U ? 3 : (p.spin == 2 ? 3 : 1 << p.spin);
        d.bp = 1u << a;
        d.bq = 1u << b;
        if (p.kind == EDK_PARAM_U) {
            d.kind = a == b ? kParamDouble : kParamPair;
        } else if (a == b) {
            d.kind = kParamNumber;
        } else {
            d.kind = kParamHop;
            for (int s = 0; s < 2; ++s) {
                if (!((d.spin_mask >> s) & 1)) continue;
                const int64_t n = s == 0 ? o.dup : o.ddn;
                at[s][q] = up.size();
                up.resize(up.size() + (size_t)n);
                hop_map(s == 0 ? su : sd, rank, n, a, b, reinterpret_cast<int32_t *>(up.data() + at[s][q]));
            }
        }
    }
    o.tables = DBuf(sizeof(uint32_t) * up.size(), o.ctx);
    if (!o.tables.p) return o.fail(EDK_ERR_NOMEM, "gradient tables");
    const uint32_t *dev_up = static_cast<const uint32_t *>(o.tables.p);
    for (int q = 0; q < np; ++q) {
        if (at[0][q]) pd[q].mapu = reinterpret_cast<const int32_t *>(dev_up + at[0][q]);
        if (at[1][q]) pd[q].mapd = reinterpret_cast<const int32_t *>(dev_up + at[1][q]);
    }
    std::memcpy(up.data(), pd.data(), sizeof(ParamDev) * np);
    o.params = static_cast<const ParamDev *>(o.tables.p);
    o.st_up = dev_up + pw;
    o.st_dn = dev_up + pw + o.dup;
    if ((rc = o.cuda(cudaMemcpyAsync(o.tables.p, up.data(), sizeof(uint32_t) * up.size(), cudaMemcpyHostToDevice, o.st),
                     "h2d")))
        return rc;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    o.grid = sms * 4;
    const size_t nq = std::max(np, 4);
    o.scratch = DBuf(sizeof(double) * ((size_t)o.grid * nq + nq + 4) + 64, o.ctx);
    if (!o.scratch.p) return o.fail(EDK_ERR_NOMEM, "gradient scratch");
    o.partials = o.scratch.d();
    o.out = o.partials + (size_t)o.grid * nq;
    o.counter = reinterpret_cast<unsigned *>(o.out + nq + 2);
    if ((rc = o.cuda(cudaMemsetAsync(o.counter, 0, 16, o.st), "memset"))) return rc;
    // the upload reads the host vector before it goes out of scope
    if ((rc = o.cuda(cudaStreamSynchronize(o.st), "sync"))) return rc;
    edk_internal_count(o.ctx, (int64_t)(sizeof(uint32_t) * (o.dup + o.ddn) + sizeof(ParamDev) * np), 0);
    return EDK_OK;
}

// <a|dH_q|b> for every parameter, into `out` on the device (added to it when acc).
int ops_bilinear_dev(Ops &o, const double *a, const double *b, double *out, bool acc)
{
    edk_internal_add_launches(o.ctx, 1);
    return o.cuda(launch_bilinear(o.dup, o.ddn, a, b, o.st_up, o.st_dn, o.np, o.params, o.partials, o.counter, out,
                                  o.grid, acc, o.st),
                  "bilinear kernel");
}

// The same to the host.
int ops_bilinear(Ops &o, const double *a, const double *b, double *out_host)
{
    int rc = ops_bilinear_dev(o, a, b, o.out, false);
    if (rc) return rc;
    if ((rc = o.cuda(cudaMemcpyAsync(out_host, o.out, sizeof(double) * o.np, cudaMemcpyDeviceToHost, o.st), "d2h")))
        return rc;
    return o.cuda(cudaStreamSynchronize(o.st), "sync");
}

// Vector helpers on the sector of `o` (length o.dim).
struct Vec {
    Ops &o;
    int lincomb(double *out, bool acc, const double *x0, double c0, const double *x1 = nullptr, double c1 = 0,
                const double *x2 = nullptr, double c2 = 0, const double *x3 = nullptr, double c3 = 0)
    {
        edk_internal_add_launches(o.ctx, 1);
        return o.cuda(launch_lincomb(o.dim, out, acc, x0, c0, x1, c1, x2, c2, x3, c3, o.grid, o.st), "lincomb");
    }
    // up to 4 dot products in one pass, to the host
    int dots(double *res, const double *x0, const double *y0, const double *x1 = nullptr, const double *y1 = nullptr,
             const double *x2 = nullptr, const double *y2 = nullptr, const double *x3 = nullptr,
             const double *y3 = nullptr)
    {
        edk_internal_add_launches(o.ctx, 1);
        int rc = o.cuda(launch_dots(o.dim, x0, y0, x1, y1, x2, y2, x3, y3, o.partials, o.counter, o.out, o.grid, o.st),
                        "dots");
        if (rc) return rc;
        double t[4];
        if ((rc = o.cuda(cudaMemcpyAsync(t, o.out, sizeof t, cudaMemcpyDeviceToHost, o.st), "d2h"))) return rc;
        if ((rc = o.cuda(cudaStreamSynchronize(o.st), "sync"))) return rc;
        const int n = x3 ? 4 : x2 ? 3 : x1 ? 2 : 1;
        for (int i = 0; i < n; ++i) res[i] = t[i];
        return EDK_OK;
    }
};

// Elements of one array of the continued fraction (64 MB): with the frequencies all
// at once a call's memory would grow with steps times frequencies.
constexpr int kCfElements = 1 << 22;

// Forward Lanczos of phi (K steps or until breakdown) keeping checkpoints, the
// continued fraction with its vector-Jacobian product, then the reverse sweep, all
// queued on the stream: every coefficient stays on the device (GradScalars), and
// the host reads only b_k, to learn where the chain ends.  Adds to theta_bar
// (target-sector parameters), writes phibar (target sector) and returns the e0bar
// of this chain.
//   G(z) = b_1^2 u_1 with (z - ph (T - e0)) u = e1.
int chain_vjp(edk_h *ht, Ops &o, const double *phi, int K, double e0, double ph, int nw, const double *wn,
              const double *gbar, double *theta_bar, double *phibar, double &e0bar_out, double *G_out,
              edk_grad_stats *stats)
{
    Vec v{o};
    const int64_t n = o.dim;
    const size_t vb = sizeof(double) * (size_t)n;
    int rc;
    double nrm2 = 0.0;
    if ((rc = v.dots(&nrm2, phi, phi))) return rc;
    const double b1 = std::sqrt(nrm2);
    if (!(b1 > 1e-300)) return o.fail(EDK_ERR_ZERO_START, "gradient: zero start vector");
    K = (int)std::min<int64_t>(K, n);
    const int m = std::max(2, (int)std::ceil(std::sqrt(2.0 * K)));
    const int nseg = (K + m - 1) / m;
    // scalars (K + 2 each), theta, and the continued fraction's buffers
    // the latter for at most kCfElements / K frequencies at a time
    const int nwc = std::min(nw, std::max(32, kCfElements / K));
    const size_t ks = (size_t)K + 2, nsc = 4 * ks + 8 + o.np;
    DBuf sc(sizeof(double) * nsc, o.ctx), cf(sizeof(double) * ((size_t)nwc * (4 * (size_t)K + 9)), o.ctx);
    if (!sc.p || !cf.p) return o.fail(EDK_ERR_NOMEM, "gradient scalars");
    const GradScalars S{sc.d(), sc.d() + ks, sc.d() + 2 * ks, sc.d() + 3 * ks, sc.d() + 4 * ks};
    double *theta = sc.d() + 4 * ks + 8;
    double2 *cf_cp = reinterpret_cast<double2 *>(cf.p), *cf_u = cf_cp + (size_t)K * nwc, *cf_gs = cf_u + (size_t)K * nwc;
    double *cf_in = reinterpret_cast<double *>(cf_gs + nwc), *cf_G = cf_in + 3 * (size_t)nwc,
           *cf_parts = cf_G + 2 * (size_t)nwc;
    if ((rc = o.cuda(cudaMemsetAsync(sc.p, 0, sizeof(double) * nsc, o.st), "memset"))) return rc;
    if ((rc = o.cuda(cudaMemcpyAsync(S.be + 1, &b1, sizeof b1, cudaMemcpyHostToDevice, o.st), "h2d"))) return rc;
    const GradPass ps{n, o.grid, o.partials, o.counter, o.st};
    auto count = [&](cudaError_t e, const char *where, int launches = 1) {
        edk_internal_add_launches(o.ctx, launches);
        return o.cuda(e, where);
    };
    // ---- forward ----
    std::vector<DBuf> ck(2 * nseg);       // (v_{s-1}, v_s) at segment starts s = 1 + j m
    std::vector<double> be(K + 2, 0.0);
    {
        DBuf va(vb, o.ctx), vbuf(vb, o.ctx), vc(vb, o.ctx), hv(vb, o.ctx);
        if (!va.p || !vbuf.p || !vc.p || !hv.p) return o.fail(EDK_ERR_NOMEM, "gradient vectors");
        double *vkm1 = va.d(), *vk = vbuf.d(), *vnext = vc.d();
        if ((rc = o.cuda(cudaMemsetAsync(vkm1, 0, vb, o.st), "memset"))) return rc;
        if ((rc = v.lincomb(vk, false, phi, 1.0 / b1))) return rc;
        // The host reads the b_k at each segment's start, one segment late, so that a
        // chain that broke down is left soon and steps stay queued meanwhile.
        double *seen = nullptr;
        cudaEvent_t seen_ev = nullptr;
        if (nseg > 2 && (rc = edk_internal_pinned(o.ctx, (size_t)K + 2, &seen, &seen_ev))) return rc;
        for (int k = 1; k <= K; ++k) {
            if ((k - 1) % m == 0) {
                const int j = (k - 1) / m;
                if (seen && j >= 2) {
                    if ((rc = o.cuda(cudaEventSynchronize(seen_ev), "sync"))) return rc;
                    bool broke = false;
                    for (int q = 2; q <= k - m; ++q) broke = broke || !(seen[q] > 1e-25);
                    if (broke) break;
                }
                if (seen && j >= 1 && k + m <= K) {
                    if ((rc = o.cuda(cudaMemcpyAsync(seen, S.be, sizeof(double) * (k + 1), cudaMemcpyDeviceToHost, o.st),
                                     "d2h")))
                        return rc;
                    if ((rc = o.cuda(cudaEventRecord(seen_ev, o.st), "event"))) return rc;
                }
                ck[2 * j] = DBuf(vb, o.ctx);
                ck[2 * j + 1] = DBuf(vb, o.ctx);
                if (!ck[2 * j].p || !ck[2 * j + 1].p) return o.fail(EDK_ERR_NOMEM, "gradient checkpoints");
                if ((rc = o.cuda(cudaMemcpyAsync(ck[2 * j].p, vkm1, vb, cudaMemcpyDeviceToDevice, o.st), "copy")))
                    return rc;
                if ((rc = o.cuda(cudaMemcpyAsync(ck[2 * j + 1].p, vk, vb, cudaMemcpyDeviceToDevice, o.st), "copy")))
                    return rc;
            }
            if ((rc = edk_hmult(ht, EDK_F64, n, vk, hv.p))) return rc;
            if ((rc = count(pass_fwd_w(ps, hv.d(), vkm1, vk, k, S), "gradient forward"))) return rc;
            if ((rc = count(pass_fwd_r(ps, vnext, hv.d(), vk, k, S), "gradient forward"))) return rc;
            if (k == K) break;
            if ((rc = count(pass_fwd_scale(ps, vnext, k, S), "gradient forward"))) return rc;
            std::swap(vkm1, vk);
            std::swap(vk, vnext);
        }
        if ((rc = o.cuda(cudaMemcpyAsync(be.data(), S.be, sizeof(double) * (K + 2), cudaMemcpyDeviceToHost, o.st), "d2h")))
            return rc;
        if ((rc = o.cuda(cudaStreamSynchronize(o.st), "sync"))) return rc;
    }   // the forward vectors are not needed any more
    int Keff = 1;
    while (Keff < K && be[Keff + 1] > 1e-25) ++Keff;
    if (stats) stats->forward_steps += Keff;
    const bool has_next = be[Keff + 1] > 1e-25;
    // ---- continued fraction and its VJP ----
    for (int w0 = 0; w0 < nw; w0 += nwc) {
        const int nq = std::min(nwc, nw - w0);
        std::vector<double> in(wn + w0, wn + w0 + nq);
        in.insert(in.end(), gbar + 2 * (size_t)w0, gbar + 2 * (size_t)(w0 + nq));
        if ((rc = o.cuda(cudaMemcpyAsync(cf_in, in.data(), sizeof(double) * in.size(), cudaMemcpyHostToDevice, o.st),
                         "h2d")))
            return rc;
        if ((rc = count(pass_cf(Keff, e0, ph, nq, cf_in, cf_in + nq, S, cf_cp, cf_u, cf_gs, cf_G, cf_parts, o.st),
                        "gradient continued fraction", 2)))
            return rc;
        if (G_out && nwc < nw &&
            (rc = o.cuda(cudaMemcpyAsync(G_out + 2 * (size_t)w0, cf_G, sizeof(double) * 2 * nq, cudaMemcpyDeviceToHost,
                                         o.st), "d2h")))
            return rc;
    }
    // ---- reverse sweep over segments, last first ----
    const int mseg = m + 2;
    std::vector<DBuf> seg(mseg);
    for (auto &sg : seg) {
        sg = DBuf(vb, o.ctx);
        if (!sg.p) return o.fail(EDK_ERR_NOMEM, "gradient segment");
    }
    if (stats) stats->stored_vectors = std::max<int32_t>(stats->stored_vectors, 2 * nseg + mseg + 4);
    DBuf vbn_b(vb, o.ctx), vbc_b(vb, o.ctx), wbar_b(vb, o.ctx), hw_b(vb, o.ctx);
    if (!vbn_b.p || !vbc_b.p || !wbar_b.p || !hw_b.p) return o.fail(EDK_ERR_NOMEM, "gradient adjoints");
    double *vbn = vbn_b.d(), *vbc = vbc_b.d(), *wbar = wbar_b.d();
    if ((rc = o.cuda(cudaMemsetAsync(vbn, 0, vb, o.st), "memset"))) return rc;   // vbar_{Keff+1} = 0
    if ((rc = o.cuda(cudaMemsetAsync(vbc, 0, vb, o.st), "memset"))) return rc;   // vbar_{Keff} (partial)
    const int jlast = (Keff - 1) / m;
    for (int j = jlast; j >= 0; --j) {
        const int s0 = 1 + j * m, e1 = std::min(s0 + m - 1, Keff);
        // replay: seg[i] = v_{s0-1+i}
        if ((rc = o.cuda(cudaMemcpyAsync(seg[0].p, ck[2 * j].p, vb, cudaMemcpyDeviceToDevice, o.st), "copy")))
            return rc;
        if ((rc = o.cuda(cudaMemcpyAsync(seg[1].p, ck[2 * j + 1].p, vb, cudaMemcpyDeviceToDevice, o.st), "copy")))
            return rc;
        for (int k = s0; k <= e1; ++k) {
            const int i = k - (s0 - 1);
            if (k == Keff && !has_next) {
                if ((rc = o.cuda(cudaMemsetAsync(seg[i + 1].p, 0, vb, o.st), "memset"))) return rc;
                continue;
            }
            if ((rc = edk_hmult(ht, EDK_F64, n, seg[i].p, seg[i + 1].p))) return rc;
            if ((rc = count(pass_replay(ps, seg[i + 1].d(), seg[i - 1].d(), seg[i].d(), k, S), "gradient replay")))
                return rc;
            if (stats) stats->replay_steps++;
        }
        for (int k = e1; k >= s0; --k) {
            const int i = k - (s0 - 1);
            const double *vkp = seg[i + 1].d(), *vkk = seg[i].d(), *vkm = seg[i - 1].d();
            if ((rc = count(pass_rev_wbar(ps, k < Keff, vbn, vbc, wbar, vkp, vkk, vkm, k, S), "gradient reverse")))
                return rc;
            if ((rc = edk_hmult(ht, EDK_F64, n, wbar, hw_b.p))) return rc;
            // theta_bar += <wbar| dH |v_k>
            if ((rc = ops_bilinear_dev(o, wbar, vkk, theta, true))) return rc;
            if ((rc = count(pass_rev_next(ps, vbn, vbc, hw_b.d(), wbar, vkk, vkm, k, S), "gradient reverse"))) return rc;
            std::swap(vbn, vbc);
            if (stats) stats->reverse_steps++;
        }
    }
    // vbn = vbar_1; seg[1] = v_1 (replay of the first segment)
    if ((rc = count(pass_rev_start(ps, phibar, vbn, seg[1].d(), S), "gradient reverse"))) return rc;
    std::vector<double> th(o.np);
    if ((rc = o.cuda(cudaMemcpyAsync(th.data(), theta, sizeof(double) * o.np, cudaMemcpyDeviceToHost, o.st), "d2h")))
        return rc;
    if ((rc = o.cuda(cudaMemcpyAsync(&e0bar_out, S.dot + 4, sizeof(double), cudaMemcpyDeviceToHost, o.st), "d2h")))
        return rc;
    if (G_out && nwc == nw && (rc = o.cuda(cudaMemcpyAsync(G_out, cf_G, sizeof(double) * 2 * nw, cudaMemcpyDeviceToHost, o.st), "d2h")))
        return rc;
    if ((rc = o.cuda(cudaStreamSynchronize(o.st), "sync"))) return rc;
    for (int q = 0; q < o.np; ++q) theta_bar[q] += th[q];
    return EDK_OK;
}

}  // namespace

extern "C" {

int edk_dh_bilinear(edk_h *h, const void *a_dev, const void *b_dev, int32_t np, const edk_param *params,
                    double *out_host)
{
    if (!h || !a_dev || !b_dev || !out_host) return EDK_ERR_INVALID;
    Ops o;
    int rc = ops_setup(h, np, params, o);
    if (rc) return rc;
    return ops_bilinear(o, static_cast<const double *>(a_dev), static_cast<const double *>(b_dev), out_host);
}

int edk_grad_e0(edk_h *h, const void *psi_dev, int32_t np, const edk_param *params, double *grad_host)
{
    if (!h || !psi_dev || !grad_host) return EDK_ERR_INVALID;
    Ops o;
    int rc = ops_setup(h, np, params, o);
    if (rc) return rc;
    const double *psi = static_cast<const double *>(psi_dev);
    double n2 = 0.0;
    Vec v{o};
    if ((rc = v.dots(&n2, psi, psi))) return rc;
    if (!(n2 > 0.0)) return o.fail(EDK_ERR_ZERO_START, "zero state vector");
    if ((rc = ops_bilinear(o, psi, psi, grad_host))) return rc;
    for (int q = 0; q < np; ++q) grad_host[q] /= n2;
    return EDK_OK;
}

int edk_grad_green(edk_h *h, const void *psi_dev, double e0, int32_t nchain, const edk_green_spec *chains,
                   int32_t nitergreen, int32_t nw, const double *wn_host, const double *gbar_host, double e0bar,
                   int32_t np, const edk_param *params, double cg_tol, double *grad_host, double *G_host,
                   edk_grad_stats *stats)
{
    if (!h || !psi_dev || !grad_host || nchain < 0 || (nchain > 0 && (!chains || !wn_host || !gbar_host)) ||
        (nchain > 0 && (nw < 1 || nitergreen < 1)))
        return EDK_ERR_INVALID;
    if (stats) std::memset(stats, 0, sizeof *stats);
    PoolGuard guard(edk_internal_h_ctx(h));
    Ops o;
    int rc = ops_setup(h, np, params, o);
    if (rc) return rc;
    Vec v{o};
    const int64_t n = o.dim;
    const size_t vb = sizeof(double) * (size_t)n;
    int nc, nb, nup, ndn;
    edk_internal_h_info(h, &nc, &nb, &nup, &ndn);
    const int ns = nc + nb;
    // normalised psi
    DBuf psi_b(vb, o.ctx), psibar_b(vb, o.ctx);
    if (!psi_b.p || !psibar_b.p) return o.fail(EDK_ERR_NOMEM, "gradient vectors");
    double n2 = 0.0;
    if ((rc = v.dots(&n2, static_cast<const double *>(psi_dev), static_cast<const double *>(psi_dev)))) return rc;
    if (!(n2 > 0.0)) return o.fail(EDK_ERR_ZERO_START, "zero state vector");
    const double *psi = psi_b.d();
    if ((rc = v.lincomb(psi_b.d(), false, static_cast<const double *>(psi_dev), 1.0 / std::sqrt(n2)))) return rc;
    if ((rc = o.cuda(cudaMemsetAsync(psibar_b.p, 0, vb, o.st), "memset"))) return rc;
    std::vector<double> grad(np, 0.0), tb(np);
    double e0bar_total = e0bar;
    // ---- chains ----
    for (int c = 0; c < nchain; ++c) {
        const edk_green_spec &g = chains[c];
        if (g.spin < 0 || g.spin > 1 || g.site < 0 || g.site >= nc) return o.fail(EDK_ERR_INVALID, "chain spec");
        const int d = g.dagger ? 1 : -1;
        const int tnu = nup + (g.spin == 0 ? d : 0), tnd = ndn + (g.spin == 1 ? d : 0);
        if (tnu < 0 || tnu > ns || tnd < 0 || tnd > ns) {
            if (G_host) std::memset(G_host + (size_t)c * 2 * nw, 0, sizeof(double) * 2 * nw);
            continue;
        }
        edk_h *ht_raw = nullptr;
        if ((rc = edk_internal_h_sibling(h, tnu, tnd, &ht_raw))) return rc;
        HPtr ht(ht_raw);
        Ops ot;
        if ((rc = ops_setup(ht.get(), np, params, ot))) return rc;
        const size_t tvb = sizeof(double) * (size_t)ot.dim;
        DBuf phi(tvb, o.ctx), phibar(tvb, o.ctx);
        if (!phi.p || !phibar.p) return o.fail(EDK_ERR_NOMEM, "gradient vectors");
        int64_t od = 0;
        if ((rc = edk_apply_c(h, EDK_F64, g.site, g.spin, g.dagger ? 1 : 0, g.site2, g.sign2, psi, phi.p, &od)))
            return rc;
        double e0b = 0.0;
        std::vector<double> tg(np, 0.0);
        if ((rc = chain_vjp(ht.get(), ot, phi.d(), nitergreen, e0, g.dagger ? 1.0 : -1.0, nw, wn_host,
                            gbar_host + (size_t)c * 2 * nw, tg.data(), phibar.d(), e0b,
                            G_host ? G_host + (size_t)c * 2 * nw : nullptr, stats)))
            return rc;
        for (int q = 0; q < np; ++q) grad[q] += tg[q];
        e0bar_total += e0b;
        // psibar += C^T phibar (the map with dagger flipped, from the target sector back)
        DBuf back(vb, o.ctx);
        if (!back.p) return o.fail(EDK_ERR_NOMEM, "gradient vectors");
        if ((rc = edk_apply_c(ht.get(), EDK_F64, g.site, g.spin, g.dagger ? 0 : 1, g.site2, g.sign2, phibar.p, back.p,
                              &od)))
            return rc;
        if ((rc = v.lincomb(psibar_b.d(), true, back.d(), 1.0))) return rc;
    }
    // ---- E0 (Hellmann-Feynman) ----
    if ((rc = ops_bilinear(o, psi, psi, tb.data()))) return rc;
    for (int q = 0; q < np; ++q) grad[q] += e0bar_total * tb[q];
    // ---- eigenvector: (H - E0) lambda = P psibar, lambda orthogonal to psi ----
    if (nchain > 0) {
        double pp[2];
        if ((rc = v.dots(pp, psibar_b.d(), psi, psibar_b.d(), psibar_b.d()))) return rc;
        if (pp[1] > 0.0) {
            DBuf x_b(vb, o.ctx), r_b(vb, o.ctx), p_b(vb, o.ctx), ap_b(vb, o.ctx), cg_b(sizeof(CgScalars), o.ctx);
            if (!x_b.p || !r_b.p || !p_b.p || !ap_b.p || !cg_b.p) return o.fail(EDK_ERR_NOMEM, "gradient CG vectors");
            double *x = x_b.d(), *r = r_b.d(), *p = p_b.d(), *ap = ap_b.d();
            if ((rc = o.cuda(cudaMemsetAsync(x, 0, vb, o.st), "memset"))) return rc;
            if ((rc = v.lincomb(r, false, psibar_b.d(), 1.0, psi, -pp[0]))) return rc;
            if ((rc = v.lincomb(p, false, r, 1.0))) return rc;
            double rr = 0.0;
            if ((rc = v.dots(&rr, r, r))) return rc;
            const double tol = cg_tol > 0.0 ? cg_tol : 1e-10;
            const int maxit = 20000;
            CgScalars cg{rr, rr, {0.0, 0.0}, 0.0, 0.0, 0, rr > tol * tol * rr ? 0 : 1};
            CgScalars *cgd = static_cast<CgScalars *>(cg_b.p);
            if ((rc = o.cuda(cudaMemcpyAsync(cgd, &cg, sizeof cg, cudaMemcpyHostToDevice, o.st), "h2d"))) return rc;
            const GradPass ps{n, o.grid, o.partials, o.counter, o.st};
            // sixteen iterations are queued between looks at the device's stop flag, which
            // turns the passes behind the last iteration into no-ops
            while (!cg.done) {
                for (int q = 0; q < 16; ++q) {
                    if ((rc = edk_hmult(h, EDK_F64, n, p, ap))) return rc;
                    edk_internal_add_launches(o.ctx, 4);
                    if ((rc = o.cuda(pass_cg(ps, x, r, p, ap, psi, e0, tol * tol, maxit, cgd), "gradient CG"))) return rc;
                }
                if ((rc = o.cuda(cudaMemcpyAsync(&cg, cgd, sizeof cg, cudaMemcpyDeviceToHost, o.st), "d2h"))) return rc;
                if ((rc = o.cuda(cudaStreamSynchronize(o.st), "sync"))) return rc;
            }
            if (stats) {
                stats->cg_iterations = cg.it;
                stats->cg_residual = cg.it > 0 ? std::sqrt(cg.rr / cg.rr0) : 0.0;   // rr0 may be 0
            }
            if ((rc = ops_bilinear(o, x, psi, tb.data()))) return rc;
            for (int q = 0; q < np; ++q) grad[q] -= tb[q];
        }
    }
    std::memcpy(grad_host, grad.data(), sizeof(double) * np);
    return EDK_OK;
}

}  // extern "C"
