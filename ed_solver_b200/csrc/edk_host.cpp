// C-ABI of the Krylov engine: contexts, sector Hamiltonians and the host-side
// drivers that sequence the device kernels (Lanczos passes 1 and 2, Green
// chains, c/c+ maps, continued fractions).
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "edk_internal.h"
#include "edk_tables.h"
#include "edk_tridiag.h"

using namespace edk;

// ---------------------------------------------------------------------------
// device buffer helper
// ---------------------------------------------------------------------------
namespace {

struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    ~DevBuf() { release(); }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    cudaError_t ensure(size_t n) {
        if (n <= bytes && p) return cudaSuccess;
        release();
        cudaError_t e = cudaMalloc(&p, n > 0 ? n : 16);
        if (e == cudaSuccess) bytes = n;
        return e;
    }
    template <typename T> T *as() const { return static_cast<T *>(p); }
};

template <typename T>
cudaError_t upload(DevBuf &b, const std::vector<T> &v, cudaStream_t st)
{
    cudaError_t e = b.ensure(sizeof(T) * (v.empty() ? 1 : v.size()));
    if (e != cudaSuccess || v.empty()) return e;
    e = cudaMemcpyAsync(b.p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(st);   // host vectors may go out of scope
}

std::vector<double> default_ran_tab()
{
    // splitmix64 seeded with 1234567, mapped to [0,1) and rounded to 3
    // decimals half away from zero (the reference's ANINT, random.f90:80-91).
    std::vector<double> t(10001);
    uint64_t x = 1234567ull;
    for (int i = 0; i < 10001; ++i) {
        x += 0x9E3779B97F4A7C15ull;
        uint64_t z = x;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z = z ^ (z >> 31);
        const double u = (double)(z >> 11) * (1.0 / 9007199254740992.0);
        t[i] = std::floor(u * 1000.0 + 0.5) / 1000.0;
    }
    return t;
}

}  // namespace

// ---------------------------------------------------------------------------
// context
// ---------------------------------------------------------------------------
struct edk_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    int num_sms = 148;
    std::string last_error;
    int64_t launches = 0;
    // reduction scratch (partials, counter, sums, flags) and Lanczos coefficients
    DevBuf partials, counter, sums, flags, tri_diag, tri_sub, coef, ran_tab, ran_tab_user;
    DevBuf cf_n, cf_diag, cf_sub, cf_e, cf_ph, cf_scale, cf_wn, cf_G, cf_flag;
    // Krylov workspace shared by all sector Hamiltonians of this context:
    // v_{k-1}, v_k, s, s', scratch (per element type), grown on demand
    DevBuf work[2][5];
    size_t work_limit = 0;   // > 0: the largest Krylov workspace a pass may allocate (bytes)
    size_t tri_cap = 0;
    int reduce_grid = 0;
    // Replay pairs of fused Lanczos steps as a CUDA graph.  Off: programmatic
    // launches overlap one step's end with the next one's tables, which two-step
    // graphs cut at every replay (us per step of a 160-step chain, graph / plain:
    // 400 states 9.0 / 6.5, 63,504 10.1 / 9.2, 853,776 23.5 / 21.8, 11.8 million
    // equal; graphs of 4 to 32 steps gain less than 0.7 us on pairs).  A graph's
    // host time is the smaller one (about 1 us a step against 3.5 us).
    bool graphs = false;
    cudaStream_t capture_stream = nullptr;   // private stream the graphs are captured on
    // pinned host copies of alpha, beta and the flags for the overlapped
    // convergence checks of Lanczos pass 1
    double *pin_tri = nullptr;
    size_t pin_cap = 0;
    cudaEvent_t pin_ev = nullptr;
    int fp32_sums = 0;       // FP32 vectors: sum the hop terms in FP32 (edk_ctx_set_fp32_sums)
    int64_t fp32_sums_min_dim = (int64_t)1 << 20;
    int kernel_path = 0;     // 0 = fastest applicable row kernel, 1 = generic row kernel only,
                             // 2/3 = the fast kernel where applicable
    // optional event timing of row-kernel launches: (class, start, stop)
    bool timing = false;
    struct Timed { int cls; cudaEvent_t a, b; double elems; int n; };
    bool capturing = false;  // a graph capture is in progress: launches are not timed
    std::vector<Timed> timed;
    std::vector<cudaEvent_t> event_pool;
    int64_t t_count[8] = {0};
    double t_ms[8] = {0};
    double t_elems[8] = {0};
    // host<->device bytes moved by the library (explicit copies)
    int64_t h2d_bytes = 0, d2h_bytes = 0;
    // sector Hamiltonians kept by edk_solve between calls (key: model hash, nup, ndn)
    std::vector<std::pair<std::string, edk_h *>> hcache;
    // batched chains: device copies of the item list, Hamiltonians, coefficients,
    // per-block workspace, and the autotuned launch shape per problem class
    DevBuf b_hams, b_items, b_queue, b_alpha, b_beta, b_done, b_work;
    DevBuf tile_scratch;      // partial sums of the two-pass row step (kind 5)
    // buffers of the other drivers (edk_internal_scratch), at most 256 MB each
    // between calls; edk_ctx_trim gives them back
    DevBuf scratch[3];
    struct BatchShape { int block, cluster, clusters; };   // clusters: resident at a time
    std::vector<std::pair<std::string, BatchShape>> batch_tuned;
    // fast-kernel launch shape timed per sector shape (element type, dim_up,
    // dim_dn, table widths, impurity sites): a rebuilt Hamiltonian of the same
    // shape (a new bath, a cleared cache) reuses it instead of timing again
    std::vector<std::pair<std::string, FastShape>> fast_by_shape;
    // stream-ordered pool of the Krylov vectors kept between the Lanczos passes
    // (keep_basis); it keeps freed chunks, up to 5/8 of the device, so later
    // passes reuse them without mapping new device memory
    cudaMemPool_t basis_pool = nullptr;
    cudaMemPool_t get_basis_pool() {
        if (basis_pool) return basis_pool;
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        if (cudaMemPoolCreate(&basis_pool, &props) != cudaSuccess) {
            (void)cudaGetLastError();
            basis_pool = nullptr;
            return nullptr;
        }
        size_t free_b = 0, total_b = 0;
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) { (void)cudaGetLastError(); total_b = 0; }
        uint64_t keep = (uint64_t)(total_b / 8 * 5);
        cudaMemPoolSetAttribute(basis_pool, cudaMemPoolAttrReleaseThreshold, &keep);
        return basis_pool;
    }
    // bytes the basis pool holds but no basis uses
    size_t basis_pool_idle() const {
        if (!basis_pool) return 0;
        uint64_t reserved = 0, used = 0;
        if (cudaMemPoolGetAttribute(basis_pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
            cudaMemPoolGetAttribute(basis_pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess)
            return 0;
        return reserved > used ? (size_t)(reserved - used) : 0;
    }
    cudaEvent_t get_event() {
        if (!event_pool.empty()) { cudaEvent_t e = event_pool.back(); event_pool.pop_back(); return e; }
        cudaEvent_t e = nullptr;
        cudaEventCreate(&e);
        return e;
    }
    void drain_timing() {
        for (auto &t : timed) {
            float ms = 0.f;
            if (cudaEventSynchronize(t.b) == cudaSuccess && cudaEventElapsedTime(&ms, t.a, t.b) == cudaSuccess) {
                t_ms[t.cls] += ms;
                t_count[t.cls] += t.n;
                t_elems[t.cls] += t.elems;
            }
            event_pool.push_back(t.a);
            event_pool.push_back(t.b);
        }
        timed.clear();
    }
    ~edk_ctx() {
        drain_timing();
        if (capture_stream) cudaStreamDestroy(capture_stream);
        if (pin_tri) cudaFreeHost(pin_tri);
        if (pin_ev) cudaEventDestroy(pin_ev);
        for (auto e : event_pool) cudaEventDestroy(e);
        if (basis_pool) cudaMemPoolDestroy(basis_pool);
    }

    int fail(int code, const char *fmt, ...) {
        char buf[512];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof buf, fmt, ap);
        va_end(ap);
        last_error = buf;
        return code;
    }
    int cuda(cudaError_t e, const char *where) {
        if (e == cudaSuccess) return EDK_OK;
        return fail(e == cudaErrorMemoryAllocation ? EDK_ERR_NOMEM : EDK_ERR_CUDA, "%s: %s", where,
                    cudaGetErrorString(e));
    }
    int ensure_tri(size_t n) {
        if (n <= tri_cap) return EDK_OK;
        size_t cap = std::max<size_t>(n, 1024);
        int rc = cuda(tri_diag.ensure(sizeof(double) * cap), "alloc tri");
        if (rc) return rc;
        rc = cuda(tri_sub.ensure(sizeof(double) * cap), "alloc tri");
        if (rc) return rc;
        rc = cuda(coef.ensure(sizeof(double) * cap), "alloc coef");
        if (rc) return rc;
        tri_cap = cap;
        return EDK_OK;
    }
};

namespace {

int ctx_init(edk_ctx *c)
{
    cudaError_t e = cudaSetDevice(c->device);
    if (e != cudaSuccess) return c->cuda(e, "cudaSetDevice");
    cudaDeviceProp prop;
    e = cudaGetDeviceProperties(&prop, c->device);
    if (e != cudaSuccess) return c->cuda(e, "cudaGetDeviceProperties");
    c->num_sms = prop.multiProcessorCount;
    c->reduce_grid = c->num_sms * 8;
    int rc;
    // the row kernel can use up to 2 blocks per SM of the reduction grid size
    if ((rc = c->cuda(c->partials.ensure(sizeof(double) * 4 * (size_t)c->num_sms * 16), "alloc"))) return rc;
    if ((rc = c->cuda(c->counter.ensure(64), "alloc"))) return rc;
    if ((rc = c->cuda(c->sums.ensure(sizeof(double) * 16), "alloc"))) return rc;
    if ((rc = c->cuda(c->flags.ensure(sizeof(int) * 16), "alloc"))) return rc;
    if ((rc = c->cuda(cudaMemsetAsync(c->counter.p, 0, 64, c->stream), "memset"))) return rc;
    if ((rc = c->cuda(cudaMemsetAsync(c->flags.p, 0, sizeof(int) * 16, c->stream), "memset"))) return rc;
    if ((rc = c->cuda(upload(c->ran_tab, default_ran_tab(), c->stream), "upload ran_tab"))) return rc;
    if ((rc = c->ensure_tri(1024))) return rc;
    return EDK_OK;
}

}  // namespace

// ---------------------------------------------------------------------------
// sector Hamiltonian
// ---------------------------------------------------------------------------
// Krylov vectors kept between pass 1 and pass 2 (edk_lanczos_opts.keep_basis):
// v_1, v_2, ... in chunks allocated from the context's pool as pass 1 reaches
// them.  Large sectors use chunks of kBasisChunkBytes (as many vectors as fit;
// one vector when it is larger), so the pool hands a freed chunk to the next
// pass whatever its sector and element type; a chain that needs less than one
// such chunk gets one chunk of its own size.
constexpr size_t kBasisChunkBytes = (size_t)4 << 30;
struct Basis {
    int dtype = -1;
    int64_t dim = 0;
    int cap = 0;                 // vectors allowed by the memory budget
    int nvec = 0;                // valid vectors after pass 1
    bool valid = false;
    const void *start = nullptr; // identity of the pass-1 start (start_dev, host ran_tab)
    const double *tab = nullptr;
    // contents of the pass-1 start: |start_dev| (as the start kernel summed it)
    // and the sum of the host ran_tab entries; pass 2 compares them before it
    // uses the kept vectors
    double start_norm = -1.0;
    double tab_sum = 0.0;
    cudaStream_t st = nullptr;
    cudaMemPool_t pool = nullptr;
    std::vector<void *> chunks;
    size_t vec_bytes() const { return (size_t)dim * (dtype == EDK_F64 ? 8 : 4); }
    // slots start on 256-byte boundaries, like separate allocations
    size_t stride() const { return (vec_bytes() + 255) & ~(size_t)255; }
    size_t chunk = 0;            // bytes per chunk, a multiple of stride()
    int per_chunk() const { return (int)(chunk / stride()); }
    size_t chunk_bytes() const { return chunk; }
    void *slot(int q) const
    {
        const int pc = per_chunk();
        return static_cast<char *>(chunks[(size_t)q / pc]) + (size_t)(q % pc) * stride();
    }
    // makes slot q usable; false when the budget or an allocation says no
    bool ensure(int q)
    {
        if (q >= cap || !pool) return false;
        while ((int64_t)chunks.size() * per_chunk() <= q) {
            void *p = nullptr;
            if (cudaMallocFromPoolAsync(&p, chunk_bytes(), pool, st) != cudaSuccess) {
                (void)cudaGetLastError();
                return false;
            }
            chunks.push_back(p);
        }
        return true;
    }
    void release(cudaStream_t s)
    {
        for (void *p : chunks) cudaFreeAsync(p, s);
        chunks.clear();
        valid = false;
        nvec = cap = 0;
    }
};

struct edk_h {
    edk_ctx *ctx = nullptr;
    ModelHost model;
    int nup = 0, ndn = 0;
    int64_t dup = 0, ddn = 0, dim = 0;
    SpinTableHost tab[2];
    std::vector<int32_t> rank;
    std::vector<int32_t> int_off;
    std::vector<double> int_coef;
    int hund = 0;
    // device copies
    struct SpinDev {
        DevBuf ptr, tgt, val, diag, imp, move, ell, ell_val, pal, lean, lean_kw, lean_b;
    } sd[2];
    DevBuf int_off_d, int_coef_d, jj_d, umask_d, row_order_d;
    // density terms of the split form (HAIMupdo_multr_split), built on first use
    DevBuf split_off_d, split_coef_d;
    bool split_ready = false;
    HamDev H;
    // apply_c maps keyed by (spin, dagger, site)
    struct CMap {
        int spin, dagger, site;
        int64_t dim_sigma_tgt;
        DevBuf src, sg;
    };
    std::vector<std::unique_ptr<CMap>> cmaps;
    // fast-kernel launch shape per element type, chosen by timing on first use
    // (index: shape_slot)
    FastShape fast_shape[8];
    bool fast_tuned[8] = {};
    // Nambu (Sz) sector: its tables replace the (N_up, N_dn) ones
    SzHost *sz = nullptr;
    int npart = -1;
    Basis basis;
    edk_h() = default;
    edk_h(const edk_h &) = delete;
    edk_h &operator=(const edk_h &) = delete;
    ~edk_h()
    {
        if (!basis.chunks.empty()) {
            basis.release(ctx->stream);
            cudaStreamSynchronize(ctx->stream);
        }
        if (sz) sz_destroy(sz);
    }
};

namespace {

int upload_spin(edk_h *h, int s)
{
    edk_ctx *c = h->ctx;
    const SpinTableHost &t = h->tab[s];
    auto &d = h->sd[s];
    cudaStream_t st = c->stream;
    int rc;
    if ((rc = c->cuda(upload(d.ptr, t.ptr, st), "upload ptr"))) return rc;
    if ((rc = c->cuda(upload(d.tgt, t.tgt, st), "upload tgt"))) return rc;
    if ((rc = c->cuda(upload(d.val, t.val, st), "upload val"))) return rc;
    if ((rc = c->cuda(upload(d.diag, t.diag, st), "upload diag"))) return rc;
    if ((rc = c->cuda(upload(d.imp, t.imp, st), "upload imp"))) return rc;
    if ((rc = c->cuda(upload(d.move, t.move, st), "upload move"))) return rc;
    if ((rc = c->cuda(upload(d.ell, t.ell, st), "upload ell"))) return rc;
    if ((rc = c->cuda(upload(d.ell_val, t.ell_val, st), "upload ell_val"))) return rc;
    if ((rc = c->cuda(upload(d.pal, t.palette, st), "upload pal"))) return rc;
    if ((rc = c->cuda(upload(d.lean, t.lean, st), "upload lean"))) return rc;
    if ((rc = c->cuda(upload(d.lean_kw, t.lean_kw, st), "upload lean_kw"))) return rc;
    if ((rc = c->cuda(upload(d.lean_b, t.lean_b, st), "upload lean_b"))) return rc;
    SpinTabDev &o = (s == 0) ? h->H.up : h->H.dn;
    o.ptr = d.ptr.as<int32_t>();
    o.tgt = d.tgt.as<int32_t>();
    o.val = d.val.as<double>();
    o.diag = d.diag.as<double>();
    o.imp = d.imp.as<uint8_t>();
    o.move = d.move.as<int32_t>();
    o.ell_k = t.ell_k;
    o.packed = t.packed ? 1 : 0;
    o.npal = (int)t.palette.size();
    o.ell = d.ell.as<uint32_t>();
    o.ell_val = d.ell_val.as<double>();
    o.pal = d.pal.as<double>();
    o.lean_ks = t.lean.empty() ? 0 : t.lean_ks;
    o.lean = t.lean.empty() ? nullptr : d.lean.as<uint32_t>();
    o.lean_kw = t.lean.empty() ? nullptr : d.lean_kw.as<uint8_t>();
    o.lean_b = t.lean.empty() ? nullptr : d.lean_b.as<uint32_t>();
    return EDK_OK;
}

int check_model(edk_ctx *c, const edk_model *m)
{
    if (!m) return c->fail(EDK_ERR_INVALID, "null model");
    if (m->nc < 1 || m->nc > kMaxNc) return c->fail(EDK_ERR_INVALID, "nc=%d outside [1,%d]", m->nc, kMaxNc);
    if (m->nb < 0 || m->nc + m->nb > kMaxNs)
        return c->fail(EDK_ERR_INVALID, "nc+nb=%d outside [1,%d]", m->nc + m->nb, kMaxNs);
    if (!m->ec || !m->u || !m->jj || (m->nb > 0 && (!m->eb || !m->vbc)))
        return c->fail(EDK_ERR_INVALID, "null model matrix");
    // hermiticity of U (impurity_class.f90:839-840) and of the one-body blocks
    for (int a = 0; a < m->nc; ++a)
        for (int b = 0; b < m->nc; ++b) {
            if (m->u[a * m->nc + b] != m->u[b * m->nc + a])
                return c->fail(EDK_ERR_INVALID, "U is not symmetric");
            for (int s = 0; s < 2; ++s)
                if (m->ec[s * m->nc * m->nc + a * m->nc + b] != m->ec[s * m->nc * m->nc + b * m->nc + a])
                    return c->fail(EDK_ERR_INVALID, "Ec is not symmetric");
        }
    for (int s = 0; s < 2; ++s)
        for (int a = 0; a < m->nb; ++a)
            for (int b = 0; b < m->nb; ++b)
                if (m->eb[s * m->nb * m->nb + a * m->nb + b] != m->eb[s * m->nb * m->nb + b * m->nb + a])
                    return c->fail(EDK_ERR_INVALID, "Eb is not symmetric");
    const bool hund_possible = std::fabs(m->jhund) > 1e-5;
    if (hund_possible && m->jhund < 0) return c->fail(EDK_ERR_INVALID, "negative Hund coupling");
    return EDK_OK;
}

int work_ptrs(edk_h *h, int dtype, void *(&w)[5])
{
    const size_t es = dtype == EDK_F64 ? 8 : 4;
    const size_t limit = h->ctx->work_limit;
    if (limit > 0 && 5 * es * (size_t)h->dim > limit)
        return h->ctx->fail(EDK_ERR_NOMEM, "Krylov workspace of %zu bytes exceeds the context's limit of %zu bytes",
                            5 * es * (size_t)h->dim, limit);
    for (int i = 0; i < 5; ++i) {
        int rc = h->ctx->cuda(h->ctx->work[dtype][i].ensure(es * (size_t)h->dim), "alloc Krylov workspace");
        if (rc) return rc;
        w[i] = h->ctx->work[dtype][i].p;
    }
    return EDK_OK;
}

RowArgs base_args(edk_h *h)
{
    RowArgs a;
    edk_ctx *c = h->ctx;
    a.partials = c->partials.as<double>();
    a.counter = c->counter.as<unsigned>();
    a.sums_out = c->sums.as<double>();
    a.flags = c->flags.as<int>();
    a.tri_diag = c->tri_diag.as<double>();
    a.tri_sub = c->tri_sub.as<double>();
    return a;
}

// The fast kernel's launch shape for this sector and element type.  On the
// first call with an output vector, every feasible shape is timed (a warm-up launch,
// then the best of three: single launches, or a few in a row of a short kernel)
// writing into that vector, which the real launch then overwrites; the
// fastest is kept on the Hamiltonian.
constexpr int kMaxShapes = 32;

// FP32 hop sums for a launch of this sector and element type: FP32 vectors
// of sectors at least as large as the context's threshold.
int sum32_for(const edk_h *h, int dtype)
{
    const edk_ctx *c = h->ctx;
    return dtype == EDK_F32 && c->fp32_sums && h->dim >= c->fp32_sums_min_dim && !h->sz ? 1 : 0;
}

// What a timed launch shape is kept under: all that the candidates depend on.
std::string shape_key(const edk_h *h, int dtype, int sum32, bool hv)
{
    char key[160];
    std::snprintf(key, sizeof key, "%d:%lld:%lld:%d:%d:%d:%d:%d:%d", dtype, (long long)h->H.dup, (long long)h->H.ddn,
                  h->H.up.ell_k, h->H.dn_kmax, h->H.nc, sum32, h->H.hund, hv);
    return key;
}

// Index of edk_h::fast_shape.  Plain H*v has a shape of its own: the one that is
// fastest for a fused step can be a quarter slower for it (853,776 states with Hund
// terms: steps of 37.2 to 38.6 us whose shapes take 21.4 to 26.8 us per H*v).
int shape_slot(int dtype, int sum32, bool hv) { return dtype + 2 * sum32 + (hv ? 4 : 0); }

// aligned: every vector of the call is aligned to twice the element size,
// which the register-staged kernel (kind 0) needs; without it only the
// bulk-copy kernel (kind 1) is a candidate, taken untimed and not remembered.
int fast_shape_for(edk_h *h, int dtype, const RowArgs &a, bool aligned, FastShape &out)
{
    edk_ctx *c = h->ctx;
    const int eb = dtype == EDK_F64 ? 8 : 4;
    FastShape cand[kMaxShapes];
    const bool hv = a.mode == kModeHv;
    const int slot = shape_slot(dtype, a.sum32, hv);
    if (c->kernel_path >= 16) {
        // a fixed candidate, for measurements
        const int n = fast_shapes(h->H, eb, c->num_sms, cand, kMaxShapes, a.sum32);
        if (n == 0) return c->fail(EDK_ERR_INVALID, "fast row kernel: no launch shape");
        out = cand[(c->kernel_path - 16) % n];
        return EDK_OK;
    }
    if (h->fast_tuned[slot]) { out = h->fast_shape[slot]; return EDK_OK; }
    if (!aligned) {
        const int n = fast_shapes(h->H, eb, c->num_sms, cand, kMaxShapes, a.sum32);
        for (int i = 0; i < n; ++i)
            if (!shape_needs_pairs(cand[i].kind)) { out = cand[i]; return EDK_OK; }
        if (n == 0) return c->fail(EDK_ERR_INVALID, "fast row kernel: no launch shape");
        out = cand[0];
        return EDK_OK;
    }
    // kept by another handle of the sector's shape
    auto kept = [&](const std::string &k) -> const FastShape * {
        for (const auto &kv : c->fast_by_shape)
            if (kv.first == k) return &kv.second;
        return nullptr;
    };
    const std::string key = shape_key(h, dtype, a.sum32, hv);
    if (c->kernel_path == 0)
        if (const FastShape *f = kept(key)) {
            out = h->fast_shape[slot] = *f;
            h->fast_tuned[slot] = true;
            return EDK_OK;
        }
    const int n = fast_shapes(h->H, eb, c->num_sms, cand, kMaxShapes, a.sum32);
    if (n == 0) return c->fail(EDK_ERR_INVALID, "fast row kernel: no launch shape");
    out = cand[0];
    // inside a caller's capture nothing can be timed: a later call does it.  H*v takes
    // the steps' shape there if it is known.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(c->stream, &capture) != cudaSuccess) (void)cudaGetLastError();
    if (capture != cudaStreamCaptureStatusNone) {
        const int step = shape_slot(dtype, a.sum32, false);
        if (h->fast_tuned[step]) out = h->fast_shape[step];
        else if (const FastShape *f = kept(shape_key(h, dtype, a.sum32, false))) out = *f;
        return EDK_OK;
    }
    if (c->kernel_path != 0 || n == 1 || !a.x || !a.y) {
        if (n == 1 || c->kernel_path != 0) { h->fast_shape[slot] = out; h->fast_tuned[slot] = true; }
        return EDK_OK;
    }
    // H*v is timed as it is.  For the other modes candidates are timed as the launch
    // they mostly serve, a fused Lanczos step, against scratch coefficients, flags and reduction buffers of their
    // own (so the live Lanczos state is untouched) and a zeroed scratch vector
    // that stands in for v_k, v_{k-1} and the second output: x is gathered,
    // the call's y is written (the real launch then overwrites it).  The
    // flags and the block counter are cleared before every timed launch.
    // Without room for the scratch vector, H*v mode.
    RowArgs t = a;
    t.mode = kModeHv;
    DevBuf tv, tstate;
    const size_t vbytes = (size_t)h->dim * eb;
    if (!hv && tv.ensure(vbytes) == cudaSuccess && tstate.ensure(sizeof(double) * (16 + 4 * (size_t)c->num_sms * 16) + 256) ==
                                                cudaSuccess) {
        double *tri = tstate.as<double>();                 // tri_diag [0..7], tri_sub [8..15]
        double *part = tri + 16;
        const double init[16] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0};
        int rc0 = c->cuda(cudaMemcpyAsync(tri, init, sizeof init, cudaMemcpyHostToDevice, c->stream), "tune state");
        unsigned char *tail = reinterpret_cast<unsigned char *>(part + 4 * (size_t)c->num_sms * 16);
        if (!rc0) rc0 = c->cuda(cudaMemsetAsync(tail, 0, 256, c->stream), "tune state");
        if (!rc0) rc0 = c->cuda(cudaMemsetAsync(tv.p, 0, vbytes, c->stream), "tune state");
        if (!rc0) rc0 = c->cuda(cudaStreamSynchronize(c->stream), "tune state");
        if (rc0) return rc0;
        t.mode = kModeStep;
        t.k = 1;
        t.kdev = nullptr;
        t.gamma1 = 0.0;
        t.cutoff = 0.0;                                    // launches in a row: none ends the chain
        t.tri_diag = tri;
        t.tri_sub = tri + 8;
        t.partials = part;
        t.counter = reinterpret_cast<unsigned *>(tail);
        t.sums_out = reinterpret_cast<double *>(tail + 64);
        t.flags = reinterpret_cast<int *>(tail + 128);
        t.vk = tv.p;
        t.vkm1 = tv.p;
        t.vout = tv.p;
        t.psi = nullptr;
        t.psi_coef = nullptr;
    } else if (!hv) {
        (void)cudaGetLastError();
    }
    // each candidate: one warm-up launch, then the best of three timed ones (a single
    // timed launch let clock and cache noise pick a shape 40 % slower).  Kernels below
    // 60 us are timed eight in a row, as a chain runs them: of one launch alone the
    // events' and the start's own time is half, and its noise picked other shapes from
    // context to context: steps of 13.6 to 15.2 us at 152,460 states with Hund terms
    // (13.5 now), 33.3 to 35.5 at 853,776 (33.0), 7.0 to 8.2 at 4,900 (7.0), 12.1 to
    // 12.7 at 213,444 (11.7).  It takes 1 to 2 ms more per sector shape, once.
    cudaEvent_t ea = c->get_event(), eb_ = c->get_event();
    float best = 3.0e38f;
    for (int i = 0; i < n; ++i) {
        float cbest = 3.0e38f;
        int row = 1;
        for (int rep = 0; rep < 4; ++rep) {
            if (t.mode == kModeStep) cudaMemsetAsync(reinterpret_cast<void *>(t.counter), 0, 256, c->stream);
            cudaEventRecord(ea, c->stream);
            cudaError_t e = cudaSuccess;
            for (int q = 0; q < row && e == cudaSuccess; ++q, c->launches++)
                e = launch_rows_fast(h->H, dtype, t, c->num_sms, cand[i], c->stream);
            cudaEventRecord(eb_, c->stream);
            if (e != cudaSuccess) { (void)cudaGetLastError(); cbest = 3.0e38f; break; }
            float ms = 0.f;
            if (cudaEventSynchronize(eb_) != cudaSuccess || cudaEventElapsedTime(&ms, ea, eb_) != cudaSuccess) break;
            if (rep == 1 && ms < 0.06f) {      // (the first launch may have loaded the kernel)
                row = 8;
                continue;
            }
            if (rep >= 1) cbest = std::min(cbest, ms / row);
        }
        if (cbest < best) { best = cbest; out = cand[i]; }
    }
    c->event_pool.push_back(ea);
    c->event_pool.push_back(eb_);
    int rc = c->cuda(cudaGetLastError(), "fast row kernel autotune");
    if (rc) return rc;
    h->fast_shape[slot] = out;
    h->fast_tuned[slot] = true;
    c->fast_by_shape.push_back({key, out});
    return EDK_OK;
}

int rows(edk_h *h, int dtype, const RowArgs &a_in)
{
    edk_ctx *c = h->ctx;
    const int eb = dtype == EDK_F64 ? 8 : 4;
    RowArgs a = a_in;
    // FP32 hop sums where the context allows them (FP32 vectors of large sectors)
    a.sum32 = sum32_for(h, dtype);
    // the two-pass step (kind 5) keeps its partial sums in a scratch vector of
    // the context; it is sized before any capture, by the sector's first
    // launch.  Without room for it the other kinds serve (kind 5 launches
    // fail without scratch, so the timing skips them).
    if (a.sum32 && h->H.up.lean && !c->capturing && c->tile_scratch.bytes < sizeof(float) * (size_t)h->dim) {
        if (c->tile_scratch.ensure(sizeof(float) * (size_t)h->dim) != cudaSuccess) {
            (void)cudaGetLastError();
            c->tile_scratch.p = nullptr;   // nothing was allocated
            c->tile_scratch.bytes = 0;
        }
    }
    if (a.sum32 && c->tile_scratch.bytes >= sizeof(float) * (size_t)h->dim) a.scratch = c->tile_scratch.p;
    LaunchCfg cfg;
    if (!h->sz) {
        cfg = plan_rows(h->H, eb, c->num_sms);
        // the fast kernel uses 2-element vector accesses: every vector must be
        // aligned to twice the element size
        auto al = [&](const void *p) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) % (2 * eb)) == 0; };
        const bool aligned = al(a.x) && al(a.y) && al(a.vk) && al(a.vkm1) && al(a.vout) && al(a.psi);
        // kinds 0, 2 and 3 need those aligned column pairs; kinds 1 and 4 read
        // single elements at any alignment
        FastShape any[kMaxShapes];
        cfg.fast = c->kernel_path != 1 && fast_rows_ok(h->H, eb) && fast_shapes(h->H, eb, c->num_sms, any, kMaxShapes, a.sum32) > 0;
        if (cfg.fast) {
            int rc = fast_shape_for(h, dtype, a, aligned, cfg.fast_shape);
            if (rc) return rc;
            if (shape_needs_pairs(cfg.fast_shape.kind) && !aligned) cfg.fast = false;
            if (cfg.fast_shape.kind == 5 && !a.scratch) cfg.fast = false;   // chosen earlier, no scratch now
        }
    }
    cudaEvent_t ev_a = nullptr, ev_b = nullptr;
    const bool timed = c->timing && !c->capturing;
    if (timed) {
        ev_a = c->get_event();
        ev_b = c->get_event();
        cudaEventRecord(ev_a, c->stream);
    }
    cudaError_t e = h->sz ? launch_sz_rows(sz_dev(h->sz), dtype, a, c->num_sms, c->kernel_path == 1, c->stream)
                          : launch_rows(h->H, dtype, a, cfg, c->stream);
    if (timed) {
        cudaEventRecord(ev_b, c->stream);
        c->timed.push_back({a.mode + (dtype == EDK_F32 ? 4 : 0), ev_a, ev_b, (double)h->dim, 1});
        if (c->timed.size() > 16384) c->drain_timing();
    }
    c->launches++;
    return c->cuda(e, "row kernel");
}

}  // namespace

// ---------------------------------------------------------------------------
// Krylov sequences on the device
// ---------------------------------------------------------------------------
namespace {

// Buffers rotate through the steps: vbuf[0..1] hold v_{k-1}, v_k; sbuf[0..1]
// alternate as gather source s_{k+1} and output s_{k+2}.
struct Krylov {
    edk_h *h;
    int dtype;
    void *w[5];
    int ivk = 1, ivkm1 = 0, is = 2, is_out = 3;
    int k = 0;     // iterations completed (T_k known)
    const double *psi_coef = nullptr;
    void *psi = nullptr;
    double cutoff = 1e-25;
    double gamma1 = 0.0;    // shift of the first stored vector (energy scale of the chain)
    // two consecutive fused steps captured as a CUDA graph at step gk0; the
    // buffer rotation has period 2, so the graph replays from every step of
    // the same parity (the step index comes from a device counter)
    cudaGraphExec_t gexec = nullptr;
    int gk0 = -1;
    bool graph_off = false;
    // stored-basis mode: v_{q+1} lives in basis slot q (no buffer rotation, no graphs)
    Basis *basis = nullptr;
    ~Krylov() { if (gexec) cudaGraphExecDestroy(gexec); }
};

// v1 = start/|start| into w[1]; tri_sub[0] = |start|; psi = coef[0]*v1 when psi set
int krylov_start(Krylov &K, const void *start_dev, const double *ran_tab_dev, double *norm_out)
{
    edk_h *h = K.h;
    edk_ctx *c = h->ctx;
    int rc;
    rc = c->cuda(cudaMemsetAsync(c->flags.p, 0, sizeof(int) * 16, c->stream), "memset flags");
    if (rc) return rc;
    const int grid = c->reduce_grid;
    if (K.basis && !K.basis->ensure(0)) K.basis = nullptr;
    void *v1 = K.basis ? K.basis->slot(0) : K.w[K.ivk];
    rc = c->cuda(launch_start_vector(K.dtype, h->dim, ran_tab_dev, start_dev, v1,
                                     c->partials.as<double>(), c->counter.as<unsigned>(),
                                     c->sums.as<double>(), grid, c->stream), "start vector");
    c->launches++;
    if (rc) return rc;
    double nrm2 = 0.0;
    rc = c->cuda(cudaMemcpyAsync(&nrm2, c->sums.p, sizeof(double), cudaMemcpyDeviceToHost, c->stream), "d2h");
    if (rc) return rc;
    rc = c->cuda(cudaStreamSynchronize(c->stream), "sync");
    if (rc) return rc;
    if (norm_out) *norm_out = std::sqrt(nrm2);
    if (!std::isfinite(nrm2)) return c->fail(EDK_ERR_NOT_FINITE, "start vector has a non-finite element");
    if (!(std::sqrt(nrm2) >= K.cutoff)) return c->fail(EDK_ERR_ZERO_START, "start vector has zero norm");
    rc = c->cuda(launch_scale(K.dtype, h->dim, v1, c->sums.as<double>(), 0, K.psi, K.psi_coef,
                              c->tri_sub.as<double>(), grid, c->stream), "scale");
    c->launches++;
    K.k = 0;
    return rc;
}

// iteration k+1 of lanc_opt: k=0 -> H v1, else the fused step
int krylov_step(Krylov &K)
{
    edk_h *h = K.h;
    RowArgs a = base_args(h);
    a.cutoff = K.cutoff;
    a.gamma1 = K.gamma1;
    if (K.k == 0) {
        a.mode = kModeFirst;
        a.x = K.basis ? K.basis->slot(0) : K.w[K.ivk];
        a.y = K.w[K.is];
        int rc = rows(h, K.dtype, a);
        if (rc) return rc;
        K.k = 1;
        return EDK_OK;
    }
    if (K.basis && !K.basis->ensure(K.k)) {
        // the budget ends here: carry on with rotating buffers from v_k, v_{k-1}
        edk_ctx *c = h->ctx;
        const size_t b = K.basis->vec_bytes();
        int rc = c->cuda(cudaMemcpyAsync(K.w[K.ivk], K.basis->slot(K.k - 1), b, cudaMemcpyDeviceToDevice, c->stream),
                         "basis fallback");
        if (!rc && K.k >= 2)
            rc = c->cuda(cudaMemcpyAsync(K.w[K.ivkm1], K.basis->slot(K.k - 2), b, cudaMemcpyDeviceToDevice,
                                         c->stream), "basis fallback");
        if (rc) return rc;
        K.basis->valid = false;
        K.basis = nullptr;
    }
    a.mode = kModeStep;
    a.k = K.k;
    a.x = K.w[K.is];
    a.y = K.w[K.is_out];
    if (K.basis) {
        a.vk = K.basis->slot(K.k - 1);
        a.vkm1 = K.k >= 2 ? K.basis->slot(K.k - 2) : nullptr;
        a.vout = K.basis->slot(K.k);
    } else {
        a.vk = K.w[K.ivk];
        a.vkm1 = (K.k >= 2) ? K.w[K.ivkm1] : nullptr;
        a.vout = K.w[K.ivkm1];
    }
    a.psi = K.psi;
    a.psi_coef = K.psi_coef;
    int rc = rows(h, K.dtype, a);
    if (rc) return rc;
    if (!K.basis) std::swap(K.ivk, K.ivkm1);      // v_{k+1} now in the old v_{k-1} slot
    std::swap(K.is, K.is_out);
    K.k += 1;
    return EDK_OK;
}

// Fused steps until K.k == target.  From step 2 on, when the context asks for
// graphs, pairs of steps run as one CUDA
// graph launch (captured once per Krylov run; the first steps, which also time
// the row kernel's launch shapes, run as plain launches).
int krylov_run(Krylov &K, int target)
{
    edk_ctx *c = K.h->ctx;
    while (K.k < target) {
        const bool eligible = c->graphs && !K.graph_off && !K.basis && K.k >= 2 && target - K.k >= 2;
        if (eligible && !K.gexec) {
            // capture two steps with the device step counter, then restore the host state
            const Krylov save_state{K.h, K.dtype, {}, K.ivk, K.ivkm1, K.is, K.is_out, K.k};
            const int64_t launches0 = c->launches;
            cudaGraph_t g = nullptr;
            // capture on a private stream (the context's may be the legacy default stream,
            // which cannot be captured); nothing runs during capture
            if (!c->capture_stream &&
                cudaStreamCreateWithFlags(&c->capture_stream, cudaStreamNonBlocking) != cudaSuccess) {
                c->capture_stream = nullptr;
                K.graph_off = true;
                continue;
            }
            cudaStream_t user_stream = c->stream;
            c->stream = c->capture_stream;
            c->capturing = true;
            if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
                c->stream = user_stream;
                c->capturing = false;
                (void)cudaGetLastError();
                K.graph_off = true;
                continue;
            }
            int rc1 = EDK_OK;
            for (int s = 0; s < 2 && rc1 == EDK_OK; ++s) {
                RowArgs a = base_args(K.h);
                a.cutoff = K.cutoff;
                a.gamma1 = K.gamma1;
                a.mode = kModeStep;
                a.k = K.k;
                a.kdev = c->flags.as<int>() + 8;
                a.x = K.w[K.is];
                a.y = K.w[K.is_out];
                a.vk = K.w[K.ivk];
                a.vkm1 = K.w[K.ivkm1];
                a.vout = K.w[K.ivkm1];
                a.psi = K.psi;
                a.psi_coef = K.psi_coef;
                rc1 = rows(K.h, K.dtype, a);
                std::swap(K.ivk, K.ivkm1);
                std::swap(K.is, K.is_out);
                K.k += 1;
            }
            const cudaError_t e2 = cudaStreamEndCapture(c->stream, &g);
            c->stream = user_stream;
            c->capturing = false;
            K.ivk = save_state.ivk; K.ivkm1 = save_state.ivkm1; K.is = save_state.is; K.is_out = save_state.is_out;
            K.k = save_state.k;
            c->launches = launches0;
            c->last_error.clear();
            if (rc1 == EDK_OK && e2 == cudaSuccess && g &&
                cudaGraphInstantiate(&K.gexec, g, 0) == cudaSuccess) {
                K.gk0 = K.k;
            } else {
                K.gexec = nullptr;
                K.graph_off = true;          // fall back to plain launches for this run
                (void)cudaGetLastError();
            }
            if (g) cudaGraphDestroy(g);
            continue;
        }
        if (eligible && K.gexec && ((K.k - K.gk0) & 1) == 0) {
            int rc = c->cuda(launch_set_int(c->flags.as<int>() + 8, K.k, c->stream), "step counter");
            c->launches++;
            if (rc) return rc;
            while (target - K.k >= 2) {
                // with per-launch timing on, a replay is timed as a whole: two fused steps
                cudaEvent_t ev_a = nullptr, ev_b = nullptr;
                if (c->timing) {
                    ev_a = c->get_event();
                    ev_b = c->get_event();
                    cudaEventRecord(ev_a, c->stream);
                }
                if ((rc = c->cuda(cudaGraphLaunch(K.gexec, c->stream), "graph launch"))) return rc;
                if (c->timing) {
                    cudaEventRecord(ev_b, c->stream);
                    c->timed.push_back({kModeStep + (K.dtype == EDK_F32 ? 4 : 0), ev_a, ev_b,
                                        2.0 * (double)K.h->dim, 2});
                    if (c->timed.size() > 16384) c->drain_timing();
                }
                c->launches += 2;
                K.k += 2;
            }
            continue;
        }
        int rc = krylov_step(K);
        if (rc) return rc;
    }
    return EDK_OK;
}

struct TriHost {
    std::vector<double> diag, sub;
    int flags[2] = {0, 0};
};

int fetch_tri(edk_ctx *c, int n, TriHost &t)
{
    c->d2h_bytes += (int64_t)sizeof(double) * (2 * n + 3) + 8;
    t.diag.resize(n + 1);
    t.sub.resize(n + 2);
    int rc = c->cuda(cudaMemcpyAsync(t.diag.data(), c->tri_diag.p, sizeof(double) * (n + 1),
                                     cudaMemcpyDeviceToHost, c->stream), "d2h tri");
    if (rc) return rc;
    rc = c->cuda(cudaMemcpyAsync(t.sub.data(), c->tri_sub.p, sizeof(double) * (n + 2),
                                 cudaMemcpyDeviceToHost, c->stream), "d2h tri");
    if (rc) return rc;
    rc = c->cuda(cudaMemcpyAsync(t.flags, c->flags.p, sizeof(int) * 2, cudaMemcpyDeviceToHost,
                                 c->stream), "d2h flags");
    if (rc) return rc;
    return c->cuda(cudaStreamSynchronize(c->stream), "sync");
}

// The context's pinned buffer, of at least `need` doubles, and its event.
int ensure_pinned(edk_ctx *c, size_t need)
{
    if (need > c->pin_cap) {
        if (c->pin_tri) cudaFreeHost(c->pin_tri);
        c->pin_tri = nullptr;
        c->pin_cap = 0;
        const size_t cap = std::max<size_t>(need, 4096);
        int rc = c->cuda(cudaMallocHost(reinterpret_cast<void **>(&c->pin_tri), sizeof(double) * cap), "pinned tri");
        if (rc) return rc;
        c->pin_cap = cap;
    }
    if (!c->pin_ev) return c->cuda(cudaEventCreateWithFlags(&c->pin_ev, cudaEventDisableTiming), "event");
    return EDK_OK;
}

// Enqueue the copy of alpha_1..alpha_{n+1}, beta_0..beta_{n+1} and the flags
// into pinned host memory and record an event after it; the host can then
// queue more steps before waiting on the event (tri_wait).
int tri_enqueue(edk_ctx *c, int n)
{
    int rc = ensure_pinned(c, (size_t)(2 * n + 8));
    if (rc) return rc;
    c->d2h_bytes += (int64_t)sizeof(double) * (2 * n + 3) + 8;
    double *d = c->pin_tri, *sb = c->pin_tri + (n + 1);
    int *fl = reinterpret_cast<int *>(c->pin_tri + (2 * n + 3));
    rc = c->cuda(cudaMemcpyAsync(d, c->tri_diag.p, sizeof(double) * (n + 1), cudaMemcpyDeviceToHost, c->stream),
                     "d2h tri");
    if (rc) return rc;
    rc = c->cuda(cudaMemcpyAsync(sb, c->tri_sub.p, sizeof(double) * (n + 2), cudaMemcpyDeviceToHost, c->stream),
                 "d2h tri");
    if (rc) return rc;
    rc = c->cuda(cudaMemcpyAsync(fl, c->flags.p, sizeof(int) * 2, cudaMemcpyDeviceToHost, c->stream), "d2h flags");
    if (rc) return rc;
    return c->cuda(cudaEventRecord(c->pin_ev, c->stream), "event");
}

int tri_wait(edk_ctx *c, int n, TriHost &t)
{
    int rc = c->cuda(cudaEventSynchronize(c->pin_ev), "sync tri");
    if (rc) return rc;
    t.diag.assign(c->pin_tri, c->pin_tri + (n + 1));
    t.sub.assign(c->pin_tri + (n + 1), c->pin_tri + (2 * n + 3));
    const int *fl = reinterpret_cast<const int *>(c->pin_tri + (2 * n + 3));
    t.flags[0] = fl[0];
    t.flags[1] = fl[1];
    return EDK_OK;
}

// Order-dependent sum of a caller's ran_tab (10001 entries), 0 for none.
double host_tab_sum(const double *tab)
{
    if (!tab) return 0.0;
    double s = 0.0;
    for (int i = 0; i < 10001; ++i) s = s * 0.9999999 + tab[i];
    return s;
}

const double *ran_tab_for(edk_ctx *c, const double *user_tab, int *rc)
{
    *rc = EDK_OK;
    if (!user_tab) return c->ran_tab.as<double>();
    std::vector<double> t(user_tab, user_tab + 10001);
    *rc = c->cuda(upload(c->ran_tab_user, t, c->stream), "upload ran_tab");
    return c->ran_tab_user.as<double>();
}

}  // namespace

// ---------------------------------------------------------------------------
// C-ABI
// ---------------------------------------------------------------------------
extern "C" {

int64_t edk_binom(int n, int k) { return binom(n, k); }

int edk_basis(int ns, int npart, uint64_t *states_host)
{
    if (ns < 0 || ns > kMaxNs || npart < 0 || npart > ns || !states_host) return EDK_ERR_INVALID;
    auto s = enumerate_states(ns, npart);
    std::memcpy(states_host, s.data(), sizeof(uint64_t) * s.size());
    return EDK_OK;
}

int edk_rank_table(int ns, int32_t *rank_host)
{
    if (ns < 0 || ns > kMaxNs || !rank_host) return EDK_ERR_INVALID;
    auto r = rank_table(ns);
    std::memcpy(rank_host, r.data(), sizeof(int32_t) * r.size());
    return EDK_OK;
}

int edk_default_ran_tab(double *tab_host)
{
    if (!tab_host) return EDK_ERR_INVALID;
    const auto t = default_ran_tab();
    std::memcpy(tab_host, t.data(), sizeof(double) * t.size());
    return EDK_OK;
}

int edk_build_table(const edk_model *m, int spin, int npart, int64_t *dim, int64_t *nnz,
                    int64_t *ptr_host, int32_t *tgt_host, double *val_host, double *diag_host)
{
    edk_ctx tmp;
    if (check_model(&tmp, m) || spin < 0 || spin > 1) return EDK_ERR_INVALID;
    const int ns = m->nc + m->nb;
    if (npart < 0 || npart > ns) return EDK_ERR_INVALID;
    ModelHost mh;
    mh.nc = m->nc;
    mh.nb = m->nb;
    mh.ec.assign(m->ec, m->ec + 2 * m->nc * m->nc);
    if (m->nb > 0) {
        mh.eb.assign(m->eb, m->eb + 2 * m->nb * m->nb);
        mh.vbc.assign(m->vbc, m->vbc + 2 * m->nb * m->nc);
    }
    mh.u.assign(m->u, m->u + m->nc * m->nc);
    mh.jj.assign(m->jj, m->jj + m->nc * m->nc);
    mh.jhund = m->jhund;
    mh.cutoff = m->cutoff_hamilt_param;
    const auto rank = rank_table(ns);
    const SpinTableHost t = build_spin_table(mh, spin, npart, rank);
    if (dim) *dim = (int64_t)t.states.size();
    if (nnz) *nnz = (int64_t)t.tgt.size();
    if (ptr_host)
        for (size_t i = 0; i < t.ptr.size(); ++i) ptr_host[i] = t.ptr[i];
    if (tgt_host) std::memcpy(tgt_host, t.tgt.data(), sizeof(int32_t) * t.tgt.size());
    if (val_host) std::memcpy(val_host, t.val.data(), sizeof(double) * t.val.size());
    if (diag_host) std::memcpy(diag_host, t.diag.data(), sizeof(double) * t.diag.size());
    return EDK_OK;
}

int edk_ctx_create(int device, void *stream, edk_ctx **out)
{
    if (!out) return EDK_ERR_INVALID;
    auto *c = new (std::nothrow) edk_ctx;
    if (!c) return EDK_ERR_NOMEM;
    c->device = device;
    c->stream = static_cast<cudaStream_t>(stream);
    int rc = ctx_init(c);
    if (rc) {
        delete c;
        *out = nullptr;
        return rc;
    }
    *out = c;
    return EDK_OK;
}

int edk_ctx_destroy(edk_ctx *ctx)
{
    if (!ctx) return EDK_OK;
    cudaStreamSynchronize(ctx->stream);
    edk_ctx_clear_cache(ctx);
    delete ctx;
    return EDK_OK;
}

int edk_ctx_set_stream(edk_ctx *ctx, void *stream)
{
    if (!ctx) return EDK_ERR_INVALID;
    ctx->stream = static_cast<cudaStream_t>(stream);
    return EDK_OK;
}

const char *edk_ctx_last_error(const edk_ctx *ctx) { return ctx ? ctx->last_error.c_str() : "null context"; }

int64_t edk_ctx_launch_count(const edk_ctx *ctx) { return ctx ? ctx->launches : 0; }

cudaStream_t edk_internal_stream(edk_ctx *ctx) { return ctx->stream; }

int edk_internal_ctx_device(const edk_ctx *ctx) { return ctx->device; }

void edk_internal_fp32_sums(edk_ctx *ctx, int *enable, int64_t *min_dim)
{
    *enable = ctx->fp32_sums;
    *min_dim = ctx->fp32_sums_min_dim;
}

int edk_internal_num_sms(const edk_ctx *ctx) { return ctx->num_sms; }

// A buffer of at least `bytes` for work on the context's stream, null when
// there is no memory for it.  It holds until the next request for the slot.
void *edk_internal_scratch(edk_ctx *ctx, int slot, size_t bytes)
{
    DevBuf &b = ctx->scratch[slot];
    if (b.ensure(bytes) == cudaSuccess) return b.p;
    (void)cudaGetLastError();
    b.p = nullptr;
    b.bytes = 0;
    return nullptr;
}

// After a call has synchronised: buffers above 256 MB are given back, the
// others stay for the next call.
void edk_internal_scratch_done(edk_ctx *ctx)
{
    for (DevBuf &b : ctx->scratch)
        if (b.bytes > (size_t)256 << 20) b.release();
}

// All of them, for a call that goes on without.
void edk_internal_scratch_free(edk_ctx *ctx)
{
    for (DevBuf &b : ctx->scratch) b.release();
}

int edk_internal_fail(edk_ctx *ctx, int code, const char *msg) { return ctx->fail(code, "%s", msg); }

// The context's pinned buffer (it holds until the next call that reads
// coefficients) and the event that goes with it.
int edk_internal_pinned(edk_ctx *ctx, size_t doubles, double **buf, cudaEvent_t *ev)
{
    const int rc = ensure_pinned(ctx, doubles);
    *buf = ctx->pin_tri;
    *ev = ctx->pin_ev;
    return rc;
}

edk_ctx *edk_internal_h_ctx(edk_h *h) { return h->ctx; }

void edk_internal_h_info(const edk_h *h, int *nc, int *nb, int *nup, int *ndn)
{
    *nc = h->model.nc;
    *nb = h->model.nb;
    *nup = h->nup;
    *ndn = h->ndn;
}

void edk_internal_add_launches(edk_ctx *ctx, int64_t n) { ctx->launches += n; }

int edk_internal_h_is_sz(const edk_h *h) { return h->sz ? 1 : 0; }

// A Hamiltonian of another (nup, ndn) sector of the same model.
int edk_internal_h_sibling(edk_h *h, int nup, int ndn, edk_h **out)
{
    const ModelHost &mh = h->model;
    edk_model m{mh.nc, mh.nb, mh.ec.data(), mh.eb.data(), mh.vbc.data(), mh.u.data(), mh.jj.data(),
                mh.jhund, mh.cutoff};
    return edk_h_create(h->ctx, &m, nup, ndn, out);
}

// The basis states of one spin species of the sector (increasing order).
const uint64_t *edk_internal_h_states(const edk_h *h, int spin) { return h->tab[spin].states.data(); }

const int32_t *edk_internal_h_rank(const edk_h *h) { return h->rank.data(); }

// The context's stream-ordered pool (null when the device has none).
cudaMemPool_t edk_internal_pool(edk_ctx *ctx) { return ctx->get_basis_pool(); }

int edk_ctx_set_graphs(edk_ctx *ctx, int enable)
{
    if (!ctx) return EDK_ERR_INVALID;
    ctx->graphs = enable != 0;
    return EDK_OK;
}

int edk_ctx_set_kernel_path(edk_ctx *ctx, int path)
{
    if (!ctx || path < 0 || (path > 3 && path < 16) || path >= 16 + kMaxShapes) return EDK_ERR_INVALID;
    ctx->kernel_path = path;
    return EDK_OK;
}

int edk_ctx_timing(edk_ctx *ctx, int enable)
{
    if (!ctx) return EDK_ERR_INVALID;
    if (enable && !ctx->timing) {
        ctx->drain_timing();
        for (int i = 0; i < 8; ++i) { ctx->t_count[i] = 0; ctx->t_ms[i] = 0.0; ctx->t_elems[i] = 0.0; }
    }
    ctx->timing = enable != 0;
    return EDK_OK;
}

int edk_ctx_timing_report(edk_ctx *ctx, int which, int64_t *launches, double *total_ms)
{
    if (!ctx || which < 0 || which > 7) return EDK_ERR_INVALID;
    ctx->drain_timing();
    if (launches) *launches = ctx->t_count[which];
    if (total_ms) *total_ms = ctx->t_ms[which];
    return EDK_OK;
}

int edk_ctx_timing_elements(edk_ctx *ctx, int which, double *elements)
{
    if (!ctx || which < 0 || which > 7 || !elements) return EDK_ERR_INVALID;
    ctx->drain_timing();
    *elements = ctx->t_elems[which];
    return EDK_OK;
}

int edk_ctx_transfer_bytes(const edk_ctx *ctx, int64_t *h2d, int64_t *d2h)
{
    if (!ctx) return EDK_ERR_INVALID;
    if (h2d) *h2d = ctx->h2d_bytes;
    if (d2h) *d2h = ctx->d2h_bytes;
    return EDK_OK;
}

int edk_ctx_set_workspace_limit(edk_ctx *ctx, int64_t bytes)
{
    if (!ctx || bytes < 0) return EDK_ERR_INVALID;
    ctx->work_limit = (size_t)bytes;
    return EDK_OK;
}

int edk_ctx_set_fp32_sums(edk_ctx *ctx, int enable, int64_t min_dim)
{
    if (!ctx || min_dim < 0) return EDK_ERR_INVALID;
    ctx->fp32_sums = enable ? 1 : 0;
    ctx->fp32_sums_min_dim = min_dim;
    return EDK_OK;
}

int edk_ctx_trim(edk_ctx *ctx)
{
    if (!ctx) return EDK_ERR_INVALID;
    int rc = ctx->cuda(cudaStreamSynchronize(ctx->stream), "sync");
    if (rc) return rc;
    edk_internal_scratch_free(ctx);
    if (!ctx->basis_pool) return EDK_OK;
    return ctx->cuda(cudaMemPoolTrimTo(ctx->basis_pool, 0), "cudaMemPoolTrimTo");
}

int edk_ctx_clear_cache(edk_ctx *ctx)
{
    if (!ctx) return EDK_ERR_INVALID;
    for (auto &kv : ctx->hcache) edk_h_destroy(kv.second);
    ctx->hcache.clear();
    return EDK_OK;
}

edk_h *edk_internal_cache_get(edk_ctx *ctx, const char *key, size_t len)
{
    const std::string k(key, len);
    for (auto &kv : ctx->hcache)
        if (kv.first == k) return kv.second;
    return nullptr;
}

void edk_internal_cache_put(edk_ctx *ctx, const char *key, size_t len, edk_h *h)
{
    ctx->hcache.push_back({std::string(key, len), h});
}

void edk_internal_count(edk_ctx *ctx, int64_t h2d, int64_t d2h)
{
    ctx->h2d_bytes += h2d;
    ctx->d2h_bytes += d2h;
}

int edk_h_create(edk_ctx *ctx, const edk_model *m, int nup, int ndn, edk_h **out)
{
    if (!ctx || !out) return EDK_ERR_INVALID;
    *out = nullptr;
    int rc = check_model(ctx, m);
    if (rc) return rc;
    const int ns = m->nc + m->nb;
    if (nup < 0 || nup > ns || ndn < 0 || ndn > ns)
        return ctx->fail(EDK_ERR_INVALID, "sector (%d,%d) outside [0,%d]", nup, ndn, ns);
    std::unique_ptr<edk_h> h(new (std::nothrow) edk_h);
    if (!h) return EDK_ERR_NOMEM;
    h->ctx = ctx;
    ModelHost &mh = h->model;
    mh.nc = m->nc;
    mh.nb = m->nb;
    mh.ec.assign(m->ec, m->ec + 2 * m->nc * m->nc);
    mh.eb.assign(m->eb ? m->eb : m->ec, (m->eb ? m->eb : m->ec) + 2 * m->nb * m->nb);
    mh.vbc.assign(m->vbc ? m->vbc : m->ec, (m->vbc ? m->vbc : m->ec) + 2 * m->nb * m->nc);
    mh.u.assign(m->u, m->u + m->nc * m->nc);
    mh.jj.assign(m->jj, m->jj + m->nc * m->nc);
    mh.jhund = m->jhund;
    mh.cutoff = m->cutoff_hamilt_param;
    h->nup = nup;
    h->ndn = ndn;
    h->rank = rank_table(ns);
    h->tab[0] = build_spin_table(mh, 0, nup, h->rank);
    h->tab[1] = build_spin_table(mh, 1, ndn, h->rank);
    h->dup = (int64_t)h->tab[0].states.size();
    h->ddn = (int64_t)h->tab[1].states.size();
    h->dim = h->dup * h->ddn;
    if (h->dup >= (1ll << 31) || h->ddn >= (1ll << 31))
        return ctx->fail(EDK_ERR_UNSUPPORTED, "spin sector dimension beyond 2^31");
    density_terms(mh, h->int_off, h->int_coef);
    bool offc = false;
    for (int a = 0; a < mh.nc; ++a)
        for (int b = 0; b < mh.nc; ++b)
            if (a != b && mh.u[a * mh.nc + b] != 0.0) offc = true;
    h->hund = (std::fabs(mh.jhund) > 1e-5 && offc) ? 1 : 0;
    // device copies
    if ((rc = upload_spin(h.get(), 0))) return rc;
    if ((rc = upload_spin(h.get(), 1))) return rc;
    cudaStream_t st = ctx->stream;
    std::vector<uint8_t> umask(mh.nc * mh.nc);
    for (int i = 0; i < mh.nc * mh.nc; ++i) umask[i] = mh.u[i] != 0.0;
    auto order = row_schedule(h->tab[1].states, mh.nc, mh.nb);
    if ((rc = ctx->cuda(upload(h->int_off_d, h->int_off, st), "upload"))) return rc;
    if ((rc = ctx->cuda(upload(h->int_coef_d, h->int_coef, st), "upload"))) return rc;
    if ((rc = ctx->cuda(upload(h->jj_d, mh.jj, st), "upload"))) return rc;
    if ((rc = ctx->cuda(upload(h->umask_d, umask, st), "upload"))) return rc;
    if ((rc = ctx->cuda(upload(h->row_order_d, order, st), "upload"))) return rc;
    HamDev &H = h->H;
    H.dup = h->dup;
    H.ddn = h->ddn;
    H.nc = mh.nc;
    H.nmove = mh.nc * (mh.nc - 1);
    H.hund = h->hund;
    H.ncfg = 1 << mh.nc;
    for (int64_t r = 0; r < h->ddn; ++r)
        H.dn_kmax = std::max<int>(H.dn_kmax, h->tab[1].ptr[r + 1] - h->tab[1].ptr[r]);
    H.int_off = h->int_off_d.as<int32_t>();
    H.int_coef = h->int_coef_d.as<double>();
    H.jj = h->jj_d.as<double>();
    H.umask = h->umask_d.as<uint8_t>();
    H.row_order = h->row_order_d.as<int32_t>();
    {
        // bytes of the device tables just uploaded
        int64_t b = 0;
        for (int s = 0; s < 2; ++s) {
            const SpinTableHost &t = h->tab[s];
            b += (int64_t)(t.ptr.size() * 4 + t.tgt.size() * 4 + t.val.size() * 12 + t.diag.size() * 12 +
                           t.imp.size() + t.move.size() * 4 + t.ell.size() * 4 + t.ell_val.size() * 12 +
                           t.palette.size() * 12 + t.lean.size() * 4 + t.lean_kw.size() + t.lean_b.size() * 4);
        }
        b += (int64_t)(order.size() * 4 + h->int_coef.size() * 12 + h->int_off.size() * 4);
        ctx->h2d_bytes += b;
    }
    *out = h.release();
    return EDK_OK;
}

int edk_h_create_sz(edk_ctx *ctx, const edk_model_sz *m, int npart, edk_h **out)
{
    if (!ctx || !m || !out) return EDK_ERR_INVALID;
    *out = nullptr;
    std::unique_ptr<edk_h> h(new (std::nothrow) edk_h);
    if (!h) return EDK_ERR_NOMEM;
    h->ctx = ctx;
    std::string err;
    int rc = sz_create(m, npart, ctx->stream, &h->sz, &err);
    if (rc) return ctx->fail(rc, "%s", err.c_str());
    ModelHost &mh = h->model;
    mh.nc = m->base.nc;
    mh.nb = m->base.nb;
    mh.jhund = m->base.jhund;
    mh.cutoff = m->base.cutoff_hamilt_param;
    h->npart = npart;
    h->dim = sz_dev(h->sz).sec.dim;
    h->dup = h->dim;
    h->ddn = 1;
    ctx->h2d_bytes += sz_upload_bytes(h->sz);
    *out = h.release();
    return EDK_OK;
}

int edk_h_sz_info(const edk_h *h, int32_t *npart, double *energy_shift)
{
    if (!h) return EDK_ERR_INVALID;
    if (npart) *npart = h->sz ? h->npart : -1;
    if (energy_shift) *energy_shift = h->sz ? sz_shift(h->sz) : 0.0;
    return EDK_OK;
}

int edk_apply_csz(edk_h *src, int dtype, int site, int spin, int dagger, int projected, int site2, int sign2,
                  const void *in_dev, void *out_dev, int64_t *out_dim, int32_t *out_npart)
{
    if (!src || !in_dev || !out_dev || spin < 0 || spin > 1 || (dtype != EDK_F64 && dtype != EDK_F32))
        return EDK_ERR_INVALID;
    edk_ctx *c = src->ctx;
    if (!src->sz) return c->fail(EDK_ERR_INVALID, "edk_apply_csz needs a Nambu sector (edk_h_create_sz)");
    const SzDev &S = sz_dev(src->sz);
    if (site < 0 || site >= S.nc || site2 >= S.nc || site2 == site)
        return c->fail(EDK_ERR_INVALID, "site outside the impurity (or site2 == site)");
    const int ns = S.ns;
    // spin up: the up orbital as written; spin down: the hole orbital with c, c+ exchanged
    const int create = spin == 0 ? (dagger != 0) : (dagger == 0);
    const int npt = src->npart + (create ? 1 : -1);
    if (npt < 0 || npt > 2 * ns) return c->fail(EDK_ERR_INVALID, "target Nambu sector outside [0, 2 ns]");
    std::string err;
    const SzSectorDev *tgt = nullptr;
    int rc = sz_sector(src->sz, npt, c->stream, &tgt, &err);
    if (rc) return c->fail(rc, "%s", err.c_str());
    auto op = [&](int st_site, int sgn) {
        SzOp o;
        const int up_bit = S.nb + st_site, hole_bit = ns + S.nb + st_site;
        o.bit = 1u << (spin == 0 ? up_bit : hole_bit);
        o.create = create;
        o.sgn = sgn;
        if (projected) {
            // apply_Csz_N_updo (apply_C.f90:444-458): up needs the site's down
            // occupied (hole empty), down needs its up occupied
            o.pmask = 1u << (spin == 0 ? hole_bit : up_bit);
            o.pwant = spin == 0 ? 0u : o.pmask;
        }
        return o;
    };
    SzOp ops[2] = {op(site, 1), SzOp()};
    int nop = 1;
    if (site2 >= 0) { ops[1] = op(site2, sign2 < 0 ? -1 : 1); nop = 2; }
    if (out_dim) *out_dim = tgt->dim;
    if (out_npart) *out_npart = npt;
    rc = c->cuda(launch_sz_apply_c(dtype, S, *tgt, nop, ops, in_dev, out_dev, c->num_sms, c->stream), "apply_csz");
    c->launches++;
    return rc;
}

int edk_apply_csz_ab(edk_h *src, int dtype, int site, int proj, int site2, int proj2, int spin, int dagger,
                     const void *in_dev, void *out_dev, int64_t *out_dim, int32_t *out_npart)
{
    if (!src || !in_dev || !out_dev || spin < 0 || spin > 1 || (dtype != EDK_F64 && dtype != EDK_F32))
        return EDK_ERR_INVALID;
    edk_ctx *c = src->ctx;
    if (!src->sz) return c->fail(EDK_ERR_INVALID, "edk_apply_csz_ab needs a Nambu sector (edk_h_create_sz)");
    const SzDev &S = sz_dev(src->sz);
    if (site < 0 || site >= S.nc || site2 < 0 || site2 >= S.nc)
        return c->fail(EDK_ERR_INVALID, "site outside the impurity");
    const int ns = S.ns;
    const int create = spin == 0 ? (dagger != 0) : (dagger == 0);
    const int npt = src->npart + (create ? 1 : -1);
    if (npt < 0 || npt > 2 * ns) return c->fail(EDK_ERR_INVALID, "target Nambu sector outside [0, 2 ns]");
    std::string err;
    const SzSectorDev *tgt = nullptr;
    int rc = sz_sector(src->sz, npt, c->stream, &tgt, &err);
    if (rc) return c->fail(rc, "%s", err.c_str());
    // the two operators of symmetric_combineAB (green_class_compute_symmetric_combination.f90:155-262),
    // each c[+] of apply_Csz_updo or, projected, of apply_Csz_N_updo (apply_C.f90:404-483)
    auto op = [&](int st_site, int projected) {
        SzOp o;
        const int up_bit = S.nb + st_site, hole_bit = ns + S.nb + st_site;
        o.bit = 1u << (spin == 0 ? up_bit : hole_bit);
        o.create = create;
        o.sgn = 1;
        if (projected) {
            o.pmask = 1u << (spin == 0 ? hole_bit : up_bit);
            o.pwant = spin == 0 ? 0u : o.pmask;
        }
        return o;
    };
    SzOp ops[2] = {op(site, proj), op(site2, proj2)};
    if (out_dim) *out_dim = tgt->dim;
    if (out_npart) *out_npart = npt;
    rc = c->cuda(launch_sz_apply_c(dtype, S, *tgt, 2, ops, in_dev, out_dev, c->num_sms, c->stream), "apply_csz_ab");
    c->launches++;
    return rc;
}

int edk_apply_cnambu(edk_h *src, int dtype, int orb, int dagger, int orb2, int sign2, const void *in_dev,
                     void *out_dev, int64_t *out_dim, int32_t *out_npart)
{
    if (!src || !in_dev || !out_dev || (dtype != EDK_F64 && dtype != EDK_F32)) return EDK_ERR_INVALID;
    edk_ctx *c = src->ctx;
    if (!src->sz) return c->fail(EDK_ERR_INVALID, "edk_apply_cnambu needs a Nambu sector (edk_h_create_sz)");
    const SzDev &S = sz_dev(src->sz);
    const int ns = S.ns, nc = S.nc;
    if (orb < 0 || orb >= 2 * nc || orb2 >= 2 * nc || orb2 == orb)
        return c->fail(EDK_ERR_INVALID, "Nambu orbital outside [0, 2nc) (or orb2 == orb)");
    const int npt = src->npart + (dagger ? 1 : -1);
    if (npt < 0 || npt > 2 * ns) return c->fail(EDK_ERR_INVALID, "target Nambu sector outside [0, 2 ns]");
    std::string err;
    const SzSectorDev *tgt = nullptr;
    int rc = sz_sector(src->sz, npt, c->stream, &tgt, &err);
    if (rc) return c->fail(rc, "%s", err.c_str());
    // IMPiorb of the Nambu AIM2 (quantum_algebra_Anderson_Impurity_class2.f90:88-93)
    auto bit = [&](int o) { return 1u << (o < nc ? S.nb + o : ns + S.nb + (o - nc)); };
    SzOp ops[2];
    ops[0].bit = bit(orb);
    ops[0].create = dagger ? 1 : 0;
    int nop = 1;
    if (orb2 >= 0) {
        ops[1].bit = bit(orb2);
        ops[1].create = dagger ? 1 : 0;
        ops[1].sgn = sign2 < 0 ? -1 : 1;
        nop = 2;
    }
    if (out_dim) *out_dim = tgt->dim;
    if (out_npart) *out_npart = npt;
    rc = c->cuda(launch_sz_apply_c(dtype, S, *tgt, nop, ops, in_dev, out_dev, c->num_sms, c->stream), "apply_cnambu");
    c->launches++;
    return rc;
}

int edk_h_destroy(edk_h *h)
{
    if (!h) return EDK_OK;
    cudaStreamSynchronize(h->ctx->stream);
    delete h;
    return EDK_OK;
}

int edk_h_launch_shapes(const edk_h *h, int dtype, int32_t *desc, int32_t cap)
{
    if (!h || (dtype != EDK_F64 && dtype != EDK_F32) || cap < 0 || (cap > 0 && !desc)) return -1;
    if (h->sz) return 0;
    FastShape cand[kMaxShapes];
    const int n = fast_shapes(h->H, dtype == EDK_F64 ? 8 : 4, h->ctx->num_sms, cand, kMaxShapes, sum32_for(h, dtype));
    for (int i = 0; i < n && i < cap; ++i) {
        desc[5 * i] = cand[i].r;
        desc[5 * i + 1] = cand[i].kmu;
        desc[5 * i + 2] = cand[i].kmd;
        desc[5 * i + 3] = cand[i].variant;
        desc[5 * i + 4] = cand[i].kind;
    }
    return n;
}

int edk_h_launch_shape_chosen(const edk_h *h, int dtype, int fp32_sums, int32_t *desc)
{
    if (!h || !desc || (dtype != EDK_F64 && dtype != EDK_F32)) return EDK_ERR_INVALID;
    if (h->sz) return 0;
    const int s32 = dtype == EDK_F32 && fp32_sums ? 1 : 0;
    // the fused step's, else plain H*v's
    FastShape out;
    bool found = false;
    for (int hv = 0; hv < 2 && !found; ++hv) {
        const int slot = shape_slot(dtype, s32, hv != 0);
        if (h->fast_tuned[slot]) {
            out = h->fast_shape[slot];
            found = true;
            continue;
        }
        const std::string key = shape_key(h, dtype, s32, hv != 0);
        for (const auto &kv : h->ctx->fast_by_shape)
            if (kv.first == key) { out = kv.second; found = true; }
    }
    if (!found) return 0;
    desc[0] = out.r;
    desc[1] = out.kmu;
    desc[2] = out.kmd;
    desc[3] = out.variant;
    desc[4] = out.kind;
    return 1;
}

int edk_h_dims(const edk_h *h, int64_t *dim, int64_t *dim_up, int64_t *dim_dn)
{
    if (!h) return EDK_ERR_INVALID;
    if (dim) *dim = h->dim;
    if (dim_up) *dim_up = h->dup;
    if (dim_dn) *dim_dn = h->ddn;
    return EDK_OK;
}

int edk_h_table(const edk_h *h, int spin, int64_t *nnz, int64_t *ptr_host, int32_t *tgt_host,
                double *val_host, double *diag_host)
{
    if (!h || spin < 0 || spin > 1) return EDK_ERR_INVALID;
    if (h->sz) return h->ctx->fail(EDK_ERR_UNSUPPORTED, "a Nambu sector has no spin tables");
    const SpinTableHost &t = h->tab[spin];
    if (nnz) *nnz = (int64_t)t.tgt.size();
    if (ptr_host)
        for (size_t i = 0; i < t.ptr.size(); ++i) ptr_host[i] = t.ptr[i];
    if (tgt_host) std::memcpy(tgt_host, t.tgt.data(), sizeof(int32_t) * t.tgt.size());
    if (val_host) std::memcpy(val_host, t.val.data(), sizeof(double) * t.val.size());
    if (diag_host) std::memcpy(diag_host, t.diag.data(), sizeof(double) * t.diag.size());
    return EDK_OK;
}

int edk_hmult(edk_h *h, int dtype, int64_t n, const void *x_dev, void *y_dev)
{
    if (!h || !x_dev || !y_dev || (dtype != EDK_F64 && dtype != EDK_F32)) return EDK_ERR_INVALID;
    if (n != h->dim) return h->ctx->fail(EDK_ERR_INVALID, "n=%lld differs from the sector dimension %lld",
                                         (long long)n, (long long)h->dim);
    if (x_dev == y_dev) return h->ctx->fail(EDK_ERR_INVALID, "x and y must not alias");
    RowArgs a = base_args(h);
    a.mode = kModeHv;
    a.x = x_dev;
    a.y = y_dev;
    return rows(h, dtype, a);
}

int edk_hmult_split(edk_h *h, int dtype, int64_t n, const void *x_dev, void *y_dev)
{
    if (!h || !x_dev || !y_dev || (dtype != EDK_F64 && dtype != EDK_F32)) return EDK_ERR_INVALID;
    edk_ctx *c = h->ctx;
    if (n != h->dim) return c->fail(EDK_ERR_INVALID, "n=%lld differs from the sector dimension %lld",
                                    (long long)n, (long long)h->dim);
    if (x_dev == y_dev) return c->fail(EDK_ERR_INVALID, "x and y must not alias");
    if (h->sz) return c->fail(EDK_ERR_UNSUPPORTED, "the split H*v is for (N_up, N_dn) sectors");
    // the reference STOPs here (HAIMupdo.f90:1243-1246)
    if (std::fabs(h->model.jhund) > 1e-5)
        return c->fail(EDK_ERR_UNSUPPORTED, "Jhund not implemented in the split H*v (|Jhund| > 1e-5)");
    int rc;
    if (!h->split_ready) {
        std::vector<int32_t> off;
        std::vector<double> coef;
        density_terms(h->model, off, coef, false);
        if ((rc = c->cuda(upload(h->split_off_d, off, c->stream), "upload split terms"))) return rc;
        if ((rc = c->cuda(upload(h->split_coef_d, coef, c->stream), "upload split terms"))) return rc;
        h->split_ready = true;
    }
    // two workspace vectors that are neither x nor y hold the transposes
    void *w[5];
    if ((rc = work_ptrs(h, dtype, w))) return rc;
    void *sc[2];
    int ns = 0;
    for (int i = 0; i < 5 && ns < 2; ++i)
        if (w[i] != x_dev && w[i] != y_dev) sc[ns++] = w[i];
    cudaError_t e = launch_split_hv(h->H, dtype, h->split_off_d.as<int32_t>(), h->split_coef_d.as<double>(), x_dev,
                                    y_dev, sc[0], sc[1], c->num_sms, c->stream);
    c->launches += 5;   // up pass, two transposes, down pass, transpose back
    return c->cuda(e, "split H*v");
}

int edk_hmult_host(edk_h *h, int dtype, int64_t n, const void *x_host, void *y_host)
{
    if (!h || !x_host || !y_host) return EDK_ERR_INVALID;
    if (n != h->dim) return h->ctx->fail(EDK_ERR_INVALID, "n differs from the sector dimension");
    void *w[5];
    int rc = work_ptrs(h, dtype, w);
    if (rc) return rc;
    edk_ctx *c = h->ctx;
    const size_t bytes = (size_t)n * (dtype == EDK_F64 ? 8 : 4);
    if ((rc = c->cuda(cudaMemcpyAsync(w[0], x_host, bytes, cudaMemcpyHostToDevice, c->stream), "h2d"))) return rc;
    if ((rc = edk_hmult(h, dtype, n, w[0], w[1]))) return rc;
    if ((rc = c->cuda(cudaMemcpyAsync(y_host, w[1], bytes, cudaMemcpyDeviceToHost, c->stream), "d2h"))) return rc;
    return c->cuda(cudaStreamSynchronize(c->stream), "sync");
}

int edk_lanczos_e0(edk_h *h, const edk_lanczos_opts *o, edk_lanczos_result *r)
{
    if (!h || !o || !r || !r->diag || !r->subdiag || !r->vecp) return EDK_ERR_INVALID;
    edk_ctx *c = h->ctx;
    if (o->dtype != EDK_F64 && o->dtype != EDK_F32) return c->fail(EDK_ERR_INVALID, "dtype");
    if (o->neigen < 1 || o->neigen > 64) return c->fail(EDK_ERR_INVALID, "neigen outside [1,64]");
    if (h->dim < 2) return c->fail(EDK_ERR_INVALID, "Lanczos needs dim >= 2 (dense ED below FULL_ED_SWITCH)");
    const int niter_max = (int)std::min<int64_t>(h->dim - 1, o->nitermax);
    if (niter_max < 1) return c->fail(EDK_ERR_INVALID, "nitermax < 1");
    int ne = (int)std::min<int64_t>(std::min<int64_t>(o->neigen, h->dim), niter_max);
    int rc = c->ensure_tri((size_t)niter_max + 4);
    if (rc) return rc;
    Krylov K{h, o->dtype};
    if ((rc = work_ptrs(h, o->dtype, K.w))) return rc;
    K.cutoff = o->cutoff_min_lanczos_vec > 0 ? o->cutoff_min_lanczos_vec : 1e-25;
    const double *tab = ran_tab_for(c, o->ran_tab, &rc);
    if (rc) return rc;
    Basis &B = h->basis;
    if (!B.chunks.empty()) {
        B.release(c->stream);
        cudaStreamSynchronize(c->stream);     // the freed chunks count as free below
    }
    if (o->keep_basis && (B.pool = c->get_basis_pool())) {
        // leave 1/16 of the device (at least 4 GB) to everything else; the
        // pool's idle chunks count as free
        size_t free_b = 0, total_b = 0;
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) { (void)cudaGetLastError(); free_b = 0; }
        free_b += c->basis_pool_idle();
        const size_t reserve = std::max<size_t>((size_t)4 << 30, total_b / 16);
        B.dtype = o->dtype;
        B.dim = h->dim;
        B.st = c->stream;
        const size_t s = B.stride();
        const size_t whole = s * ((size_t)niter_max + 1);
        B.chunk = s >= kBasisChunkBytes ? s : std::min(whole, kBasisChunkBytes / s * s);
        const size_t avail = free_b > reserve ? free_b - reserve : 0;
        const int64_t fit = (int64_t)(avail / B.chunk_bytes()) * B.per_chunk();
        B.cap = (int)std::min<int64_t>(fit, (int64_t)niter_max + 1 + B.per_chunk());
        if (B.cap >= 2) K.basis = &B;
    }
    double start_norm = -1.0;
    if ((rc = krylov_start(K, o->start_dev, tab, &start_norm))) return rc;
    const int every = std::max(1, o->check_every);
    std::vector<double> last(ne, 1e300), valp(ne), rdist(ne);
    std::vector<int> conv(ne, 0);
    TriHost T;
    int checked = 0, stop_at = 0, status = EDK_OK, target_rank = 0;
    if (o->use_target) ne = 1;
    // batches of `every` steps; the next batch is queued before the host checks
    // the previous one, so the device keeps running while the host bisects
    int queued = std::min(niter_max, K.k + every);
    if ((rc = krylov_run(K, queued))) return rc;
    if ((rc = tri_enqueue(c, queued))) return rc;
    while (!stop_at) {
        const int ready = queued;
        if (ready < niter_max) {
            queued = std::min(niter_max, K.k + every);
            if ((rc = krylov_run(K, queued))) return rc;
        }
        if ((rc = tri_wait(c, ready, T))) return rc;
        if (queued > ready && (rc = tri_enqueue(c, queued))) return rc;
        if (T.flags[1] == 2) return c->fail(EDK_ERR_TIMEOUT, "row kernel: a bounded wait for staged rows gave up");
        if (T.flags[1] == 2) return c->fail(EDK_ERR_TIMEOUT, "row kernel: a bounded wait for staged rows gave up");
    if (T.flags[1]) return c->fail(EDK_ERR_NOT_FINITE, "non-finite Lanczos coefficient");
        for (int it = checked + 1; it <= ready; ++it) {
            const int m = std::min(ne, it);
            if (o->use_target) {
                // refinement restart: follow the Ritz value nearest the target
                std::vector<double> all(it);
                tridiag_lowest(it, T.diag.data(), T.sub.data() + 1, it, all.data());
                int best = 0;
                for (int q = 1; q < it; ++q)
                    if (std::fabs(all[q] - o->target) < std::fabs(all[best] - o->target)) best = q;
                valp[0] = all[best];
                target_rank = best;
            } else {
                tridiag_lowest(it, T.diag.data(), T.sub.data() + 1, m, valp.data());
            }
            bool all = true;
            for (int j = 0; j < ne; ++j) {
                if (j < m) {
                    rdist[j] = valp[j] - last[j];
                    conv[j] = (std::fabs(rdist[j]) < o->tolerance) && it > 2;
                    if (conv[j] && o->residual_tol > 0.0) {
                        // Ritz residual |H V y - theta V y| = beta_{it+1} |y_it|
                        std::vector<double> y(it);
                        tridiag_vector(it, T.diag.data(), T.sub.data() + 1, valp[j], nullptr, 0, y.data());
                        conv[j] = std::fabs(T.sub[it] * y[it - 1]) < o->residual_tol;
                    }
                }
                if (!(j < m && conv[j])) all = false;
            }
            const bool broke = !(T.sub[it] >= K.cutoff);
            if (all || it == niter_max || broke) {
                stop_at = it;
                if (broke && !all && it < niter_max) status = EDK_KRYLOV_EXHAUSTED;
                break;
            }
            for (int j = 0; j < m; ++j) last[j] = valp[j];
        }
        checked = ready;
        if (!stop_at && ready >= niter_max) stop_at = niter_max;
    }
    // eigenpairs of T_{stop_at}
    const int n = stop_at;
    const int m = std::min(ne, n);
    std::vector<double> w(m), vecs((size_t)m * n);
    if (o->use_target) {
        std::vector<double> all(n);
        tridiag_lowest(n, T.diag.data(), T.sub.data() + 1, std::min(n, target_rank + 1), all.data());
        w[0] = all[std::min(n, target_rank + 1) - 1];
    } else {
        tridiag_lowest(n, T.diag.data(), T.sub.data() + 1, m, w.data());
    }
    int kept = 0;
    for (int j = 0; j < m; ++j) {
        const bool inwin = w[j] >= w[0] && w[j] <= w[0] + o->demax;
        if (!(j == 0 || (conv[j] && inwin))) continue;
        std::vector<double> v(n);
        // orthogonalise against kept vectors of nearby eigenvalues only
        std::vector<double> prev;
        int np = 0;
        for (int q = 0; q < kept; ++q)
            if (std::fabs(r->E[q] - w[j]) < 1e-8 * std::max(1.0, std::fabs(w[j]))) {
                prev.insert(prev.end(), r->vecp + (size_t)q * n, r->vecp + (size_t)(q + 1) * n);
                ++np;
            }
        tridiag_vector(n, T.diag.data(), T.sub.data() + 1, w[j], prev.data(), np, v.data());
        r->E[kept] = w[j];
        r->converged[kept] = conv[j];
        std::memcpy(r->vecp + (size_t)kept * n, v.data(), sizeof(double) * n);
        ++kept;
    }
    if (K.basis) {
        B.valid = true;
        B.nvec = K.k;
        B.start = o->start_dev;
        B.tab = o->ran_tab;
        B.start_norm = start_norm;
        B.tab_sum = host_tab_sum(o->ran_tab);
    } else if (!B.chunks.empty()) {
        B.release(c->stream);
    }
    r->nkept = kept;
    r->niter = n;
    r->status = status;
    std::memcpy(r->diag, T.diag.data(), sizeof(double) * n);
    std::memcpy(r->subdiag, T.sub.data(), sizeof(double) * (n + 1));
    return EDK_OK;
}

int edk_lanczos_gs(edk_h *h, const edk_lanczos_opts *o, int32_t niter, const double *coef_host, void *psi_dev)
{
    if (!h || !o || !coef_host || !psi_dev || niter < 1) return EDK_ERR_INVALID;
    edk_ctx *c = h->ctx;
    int rc = c->ensure_tri((size_t)niter + 4);
    if (rc) return rc;
    Krylov K{h, o->dtype};
    if ((rc = work_ptrs(h, o->dtype, K.w))) return rc;
    K.cutoff = o->cutoff_min_lanczos_vec > 0 ? o->cutoff_min_lanczos_vec : 1e-25;
    std::vector<double> cf(coef_host, coef_host + niter);
    cf.push_back(0.0);
    if ((rc = c->cuda(cudaMemcpyAsync(c->coef.p, cf.data(), sizeof(double) * cf.size(),
                                      cudaMemcpyHostToDevice, c->stream), "h2d coef"))) return rc;
    const double *tab = ran_tab_for(c, o->ran_tab, &rc);
    if (rc) return rc;
    Basis &B = h->basis;
    bool stored = o->keep_basis && B.valid && B.dtype == o->dtype && B.dim == h->dim && B.nvec >= niter &&
                  B.start == o->start_dev && B.tab == o->ran_tab && B.tab_sum == host_tab_sum(o->ran_tab);
    if (stored && o->start_dev) {
        // the same pointer must still hold the same start vector: compare its norm
        // with the one pass 1 summed (same grid and order, so equal to rounding)
        double n2 = 0.0;
        rc = c->cuda(launch_norm2(o->dtype, h->dim, o->start_dev, c->partials.as<double>(), c->counter.as<unsigned>(),
                                  c->sums.as<double>() + 12, c->reduce_grid, c->stream), "norm2 start");
        c->launches++;
        if (!rc) rc = c->cuda(cudaMemcpyAsync(&n2, c->sums.as<double>() + 12, sizeof(double), cudaMemcpyDeviceToHost,
                                              c->stream), "d2h");
        if (!rc) rc = c->cuda(cudaStreamSynchronize(c->stream), "sync");
        if (rc) return rc;
        const double n1 = B.start_norm;
        if (!(std::fabs(std::sqrt(n2) - n1) <= 1e-12 * n1)) stored = false;
    }
    DevBuf dptr;   // outlives the final stream synchronisation
    if (stored) {
        // psi = sum_q coef[q] v_{q+1} from the vectors pass 1 kept
        std::vector<const void *> ptrs(niter);
        for (int q = 0; q < niter; ++q) ptrs[q] = B.slot(q);
        if ((rc = c->cuda(upload(dptr, ptrs, c->stream), "upload basis pointers"))) return rc;
        rc = c->cuda(launch_combine(o->dtype, h->dim, dptr.as<const void *const>(), c->coef.as<double>(), niter,
                                    psi_dev, c->reduce_grid, c->stream), "combine basis");
        c->launches++;
        if (rc) return rc;
    } else {
        K.psi = psi_dev;
        K.psi_coef = c->coef.as<double>();
        if ((rc = krylov_start(K, o->start_dev, tab, nullptr))) return rc;
        // iterations 1..niter-1 produce v_2..v_niter (the last H*v is not needed
        // by the eigenvector but keeps one kernel for every step)
        if ((rc = krylov_run(K, niter))) return rc;
    }
    if (!B.chunks.empty() && o->keep_basis == 1) B.release(c->stream);
    // normalise psi
    if ((rc = c->cuda(launch_norm2(o->dtype, h->dim, psi_dev, c->partials.as<double>(),
                                   c->counter.as<unsigned>(), c->sums.as<double>() + 8, c->reduce_grid,
                                   c->stream), "norm2"))) return rc;
    c->launches++;
    rc = c->cuda(launch_scale(o->dtype, h->dim, psi_dev, c->sums.as<double>() + 8, 0, nullptr, nullptr,
                              nullptr, c->reduce_grid, c->stream), "scale");
    c->launches++;
    if (rc) return rc;
    return c->cuda(cudaStreamSynchronize(c->stream), "sync");
}

int edk_apply_c(edk_h *src, int dtype, int site, int spin, int dagger, int site2, int sign2,
                const void *in_dev, void *out_dev, int64_t *out_dim)
{
    if (!src || !in_dev || !out_dev || spin < 0 || spin > 1) return EDK_ERR_INVALID;
    edk_ctx *c = src->ctx;
    if (src->sz) return c->fail(EDK_ERR_INVALID, "a Nambu sector takes edk_apply_csz");
    const ModelHost &m = src->model;
    if (site < 0 || site >= m.nc || site2 >= m.nc) return c->fail(EDK_ERR_INVALID, "site outside impurity");
    const int ns = m.nc + m.nb;
    const int np = spin == 0 ? src->nup : src->ndn;
    const int npt = np + (dagger ? 1 : -1);
    if (npt < 0 || npt > ns) return c->fail(EDK_ERR_INVALID, "target sector outside [0,ns]");
    const int64_t dsig_t = binom(ns, npt);
    const int64_t dother = spin == 0 ? src->ddn : src->dup;
    if (out_dim) *out_dim = dsig_t * dother;
    // inverse maps: for each target state the source state and sign
    auto get_map = [&](int st_site, edk_h::CMap **mp) -> int {
        for (auto &cm : src->cmaps)
            if (cm->spin == spin && cm->dagger == dagger && cm->site == st_site) { *mp = cm.get(); return EDK_OK; }
        std::unique_ptr<edk_h::CMap> cm(new edk_h::CMap);
        cm->spin = spin;
        cm->dagger = dagger;
        cm->site = st_site;
        cm->dim_sigma_tgt = dsig_t;
        std::vector<int32_t> srcmap((size_t)dsig_t, -1);
        std::vector<int8_t> sg((size_t)dsig_t, 0);
        const auto &states = src->tab[spin].states;
        const int bit = m.nb + st_site;
        for (size_t i = 0; i < states.size(); ++i) {
            const uint64_t s = states[i];
            const bool occ = (s >> bit) & 1ull;
            if (dagger == occ) continue;                     // nil ket
            const uint64_t o = s ^ (1ull << bit);
            // create/destroy sign: occupied orbitals above the bit (apply_C.f90:566-581)
            const int sign = (__builtin_popcountll(o >> (bit + 1)) & 1) ? -1 : 1;
            const int32_t j = src->rank[o];
            srcmap[j] = (int32_t)i;
            sg[j] = (int8_t)sign;
        }
        int rc2 = c->cuda(upload(cm->src, srcmap, c->stream), "upload cmap");
        if (rc2) return rc2;
        rc2 = c->cuda(upload(cm->sg, sg, c->stream), "upload cmap");
        if (rc2) return rc2;
        *mp = cm.get();
        src->cmaps.push_back(std::move(cm));
        return EDK_OK;
    };
    edk_h::CMap *m1 = nullptr, *m2 = nullptr;
    int rc = get_map(site, &m1);
    if (rc) return rc;
    if (site2 >= 0) {
        if ((rc = get_map(site2, &m2))) return rc;
    }
    const int64_t dup_src = src->dup;
    const int64_t dup_tgt = spin == 0 ? dsig_t : src->dup;
    rc = c->cuda(launch_apply_c(dtype, spin, dother, dup_src, dup_tgt, dsig_t, m1->src.as<int32_t>(),
                                m1->sg.as<int8_t>(), m2 ? m2->src.as<int32_t>() : nullptr,
                                m2 ? m2->sg.as<int8_t>() : nullptr, sign2 < 0 ? -1 : 1, in_dev, out_dev,
                                c->stream),
                 "apply_c");
    c->launches++;
    return rc;
}

int edk_green_chain(edk_h *t, int dtype, const void *start_dev, int32_t nitergreen, double e0, int iph,
                    int32_t nw, const double *wn_host, double cutoff_dynamic, double *G_host,
                    double *diag_host, double *subdiag_host, int32_t *niter_done)
{
    if (!t || !start_dev || !wn_host || !G_host || nw < 1 || (iph != 1 && iph != 2)) return EDK_ERR_INVALID;
    edk_ctx *c = t->ctx;
    const int niter = (int)std::min<int64_t>(nitergreen, t->dim);
    if (niter < 1) return c->fail(EDK_ERR_INVALID, "nitergreen < 1");
    int rc = c->ensure_tri((size_t)niter + 4);
    if (rc) return rc;
    Krylov K{t, dtype};
    if ((rc = work_ptrs(t, dtype, K.w))) return rc;
    K.gamma1 = e0;          // the chain's alphas are energies near the state's
    double nrm = 0.0;
    // the start vector is copied into the workspace and normalised there
    rc = krylov_start(K, start_dev, nullptr, &nrm);
    std::memset(G_host, 0, sizeof(double) * 2 * nw);
    if (niter_done) *niter_done = 0;
    if (rc == EDK_ERR_ZERO_START || nrm * nrm < cutoff_dynamic) {
        c->last_error.clear();
        return EDK_OK;
    }
    if (rc) return rc;
    if ((rc = krylov_run(K, niter))) return rc;
    TriHost T;
    if ((rc = fetch_tri(c, K.k, T))) return rc;
    if (T.flags[1] == 2) return c->fail(EDK_ERR_TIMEOUT, "row kernel: a bounded wait for staged rows gave up");
    if (T.flags[1]) return c->fail(EDK_ERR_NOT_FINITE, "non-finite Lanczos coefficient");
    int n = niter;
    for (int it = 1; it < niter; ++it)
        if (!(T.sub[it] >= K.cutoff)) { n = it; break; }
    if (niter_done) *niter_done = n;
    if (diag_host) std::memcpy(diag_host, T.diag.data(), sizeof(double) * n);
    if (subdiag_host) std::memcpy(subdiag_host, T.sub.data(), sizeof(double) * n);
    const double ph = iph == 1 ? 1.0 : -1.0;
    const double scale = nrm * nrm;
    int32_t nn = n;
    return edk_cf_eval(c, 1, n, &nn, T.diag.data(), T.sub.data(), &e0, &ph, &scale, nw, wn_host, G_host);
}

int edk_cf_eval(edk_ctx *c, int32_t nchain, int32_t ld, const int32_t *n_host, const double *diag_host,
                const double *subdiag_host, const double *e_host, const double *ph_host,
                const double *scale_host, int32_t nw, const double *wn_host, double *G_host)
{
    if (!c || nchain < 1 || ld < 1 || nw < 1 || !n_host || !diag_host || !subdiag_host || !G_host)
        return EDK_ERR_INVALID;
    for (int i = 0; i < nchain; ++i)
        if (n_host[i] < 0 || n_host[i] > ld) return c->fail(EDK_ERR_INVALID, "chain length outside [0,ld]");
    cudaStream_t st = c->stream;
    int rc;
    auto up = [&](DevBuf &b, const void *src, size_t bytes) {
        int r2 = c->cuda(b.ensure(bytes), "alloc cf");
        if (r2) return r2;
        return c->cuda(cudaMemcpyAsync(b.p, src, bytes, cudaMemcpyHostToDevice, st), "h2d cf");
    };
    if ((rc = up(c->cf_n, n_host, sizeof(int32_t) * nchain))) return rc;
    if ((rc = up(c->cf_diag, diag_host, sizeof(double) * (size_t)nchain * ld))) return rc;
    if ((rc = up(c->cf_sub, subdiag_host, sizeof(double) * (size_t)nchain * ld))) return rc;
    if ((rc = up(c->cf_e, e_host, sizeof(double) * nchain))) return rc;
    if ((rc = up(c->cf_ph, ph_host, sizeof(double) * nchain))) return rc;
    if ((rc = up(c->cf_scale, scale_host, sizeof(double) * nchain))) return rc;
    if ((rc = up(c->cf_wn, wn_host, sizeof(double) * nw))) return rc;
    c->h2d_bytes += (int64_t)(sizeof(int32_t) * nchain + sizeof(double) * ((size_t)2 * nchain * ld + 3 * nchain + nw));
    c->d2h_bytes += (int64_t)(sizeof(double) * 2 * (size_t)nchain * nw);
    if ((rc = c->cuda(c->cf_G.ensure(sizeof(double) * 2 * (size_t)nchain * nw), "alloc"))) return rc;
    if ((rc = c->cuda(c->cf_flag.ensure(sizeof(int)), "alloc"))) return rc;
    if ((rc = c->cuda(cudaMemsetAsync(c->cf_flag.p, 0, sizeof(int), st), "memset"))) return rc;
    rc = c->cuda(launch_cf(nchain, ld, c->cf_n.as<int32_t>(), c->cf_diag.as<double>(), c->cf_sub.as<double>(),
                           c->cf_e.as<double>(), c->cf_ph.as<double>(), c->cf_scale.as<double>(), nw,
                           c->cf_wn.as<double>(), c->cf_G.as<double>(), c->cf_flag.as<int>(), st), "cf");
    c->launches++;
    if (rc) return rc;
    int flag = 0;
    if ((rc = c->cuda(cudaMemcpyAsync(G_host, c->cf_G.p, sizeof(double) * 2 * (size_t)nchain * nw,
                                      cudaMemcpyDeviceToHost, st), "d2h"))) return rc;
    if ((rc = c->cuda(cudaMemcpyAsync(&flag, c->cf_flag.p, sizeof(int), cudaMemcpyDeviceToHost, st), "d2h"))) return rc;
    if ((rc = c->cuda(cudaStreamSynchronize(st), "sync"))) return rc;
    if (flag) return c->fail(EDK_ERR_CF_ZERO_DEN, "zero denominator in the continued fraction");
    return EDK_OK;
}

int edk_double_occ(edk_h *h, int dtype, const void *psi_dev, int site, double *docc, double *norm2)
{
    if (!h || !psi_dev || site < 0 || site >= h->model.nc) return EDK_ERR_INVALID;
    edk_ctx *c = h->ctx;
    if (h->sz) return c->fail(EDK_ERR_UNSUPPORTED, "double occupancy of a Nambu sector");
    int rc = c->cuda(launch_double_occ(dtype, h->H, 1 << site, 1 << site, psi_dev, c->partials.as<double>(),
                                       c->counter.as<unsigned>(), c->sums.as<double>() + 4, c->reduce_grid,
                                       c->stream), "double occ");
    c->launches++;
    if (rc) return rc;
    double s[2];
    if ((rc = c->cuda(cudaMemcpyAsync(s, c->sums.as<double>() + 4, sizeof s, cudaMemcpyDeviceToHost,
                                      c->stream), "d2h"))) return rc;
    if ((rc = c->cuda(cudaStreamSynchronize(c->stream), "sync"))) return rc;
    if (docc) *docc = s[0];
    if (norm2) *norm2 = s[1];
    return EDK_OK;
}

int edk_residual(edk_h *h, const void *psi_dev, double e, double *res_norm, double *psi_norm)
{
    if (!h || !psi_dev) return EDK_ERR_INVALID;
    edk_ctx *c = h->ctx;
    RowArgs a = base_args(h);
    a.mode = kModeResid;
    a.x = psi_dev;
    a.eshift = e;
    int rc = rows(h, EDK_F64, a);
    if (rc) return rc;
    double s[4];
    if ((rc = c->cuda(cudaMemcpyAsync(s, c->sums.p, sizeof s, cudaMemcpyDeviceToHost, c->stream), "d2h"))) return rc;
    if ((rc = c->cuda(cudaStreamSynchronize(c->stream), "sync"))) return rc;
    if (res_norm) *res_norm = std::sqrt(s[0]);
    if (psi_norm) *psi_norm = std::sqrt(s[2]);
    return EDK_OK;
}

}  // extern "C"


// ---------------------------------------------------------------------------
// batched Green chains (edk_batch.cu)
// ---------------------------------------------------------------------------
namespace edk {

int gs_batch(edk_ctx *c, int nsec, edk_h *const *hs, int nitermax, int neigen, double tolerance, double demax,
             const double *ran_tab, int every, GsBatchSector *out)
{
    if (nsec <= 0) return EDK_OK;
    cudaStream_t st = c->stream;
    int rc = EDK_OK;
    const double *tab = ran_tab_for(c, ran_tab, &rc);
    if (rc) return rc;
    // items largest first (longest-processing-time order)
    std::vector<int> order(nsec);
    for (int i = 0; i < nsec; ++i) order[i] = i;
    std::sort(order.begin(), order.end(), [&](int a, int b) { return hs[a]->dim > hs[b]->dim; });
    int64_t maxdim = 0, maxdup = 0;
    int nmax = 1;
    std::vector<HamDev> hd(nsec);
    std::vector<GsItem> items(nsec);
    for (int q = 0; q < nsec; ++q) {
        const edk_h *h = hs[order[q]];
        hd[q] = h->H;
        GsItem &b = items[q];
        b.ham = q;
        b.dim = h->dim;
        b.niter_max = (int32_t)std::min<int64_t>(nitermax, h->dim - 1);
        b.ne = (int32_t)std::min<int64_t>(std::min<int64_t>(neigen, kGsMaxNe), b.niter_max);
        b.tolerance = tolerance;
        maxdim = std::max(maxdim, h->dim);
        maxdup = std::max(maxdup, h->dup);
        nmax = std::max(nmax, (int)b.niter_max);
    }
    const size_t ld = (size_t)nmax + 2;
    DevBuf d_hams, d_items, d_alpha, d_beta, d_res, d_ptrs, d_coef;
    if ((rc = c->cuda(d_alpha.ensure(sizeof(double) * ld * nsec), "alloc"))) return rc;
    if ((rc = c->cuda(d_beta.ensure(sizeof(double) * ld * nsec), "alloc"))) return rc;
    if ((rc = c->cuda(d_res.ensure(sizeof(int32_t) * 2 * nsec), "alloc"))) return rc;
    for (int q = 0; q < nsec; ++q) {
        items[q].alpha = d_alpha.as<double>() + (size_t)q * ld;
        items[q].beta = d_beta.as<double>() + (size_t)q * ld;
        items[q].result = d_res.as<int32_t>() + 2 * q;
    }
    const int R = 2 * maxdup * 8 + 16 * (int64_t)nmax <= 200 * 1024 ? 2 : 1;
    if (maxdup * 8 + 16 * (int64_t)nmax > 200 * 1024)
        return c->fail(EDK_ERR_UNSUPPORTED, "batched ground states: rows of at most 12288 states");
    const int grid = (int)std::min<int64_t>(nsec, c->num_sms);
    if ((rc = c->cuda(c->b_work.ensure(sizeof(double) * 4 * (size_t)maxdim * grid), "alloc batch workspace")))
        return rc;
    if ((rc = c->cuda(c->b_queue.ensure(sizeof(int)), "alloc"))) return rc;
    if ((rc = c->cuda(upload(d_hams, hd, st), "upload hams"))) return rc;
    if ((rc = c->cuda(upload(d_items, items, st), "upload items"))) return rc;
    c->h2d_bytes += (int64_t)(hd.size() * sizeof(HamDev) + items.size() * sizeof(GsItem));
    auto launch = [&](int pass) -> int {
        int r2 = c->cuda(cudaMemsetAsync(c->b_queue.p, 0, sizeof(int), st), "memset");
        if (r2) return r2;
        r2 = c->cuda(launch_gs_batch(R, d_hams.as<HamDev>(), d_items.as<GsItem>(), nsec, c->b_queue.as<int>(),
                                     c->b_work.p, maxdim, maxdup, nmax, tab, 1e-25, std::max(1, every), pass, grid,
                                     st),
                     "batched ground states");
        c->launches++;
        if (r2) return r2;
        return c->cuda(cudaStreamSynchronize(st), "sync");
    };
    // ---- pass 1 ----
    if ((rc = launch(1))) return rc;
    std::vector<double> al(ld * nsec), be(ld * nsec);
    std::vector<int32_t> res(2 * nsec);
    cudaMemcpyAsync(al.data(), d_alpha.p, sizeof(double) * ld * nsec, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(be.data(), d_beta.p, sizeof(double) * ld * nsec, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(res.data(), d_res.p, sizeof(int32_t) * 2 * nsec, cudaMemcpyDeviceToHost, st);
    if ((rc = c->cuda(cudaStreamSynchronize(st), "sync"))) return rc;
    c->d2h_bytes += (int64_t)(sizeof(double) * 2 * ld * nsec + sizeof(int32_t) * 2 * nsec);
    // ---- eigenpairs of every tridiagonal, the kept states (as edk_lanczos_e0) ----
    std::vector<double> coef;
    std::vector<void *> ptrs;
    std::vector<int64_t> coef_off(nsec), ptr_off(nsec);
    for (int q = 0; q < nsec; ++q) {
        GsBatchSector &o = out[order[q]];
        const int n = res[2 * q];
        o.niter = n;
        o.status = res[2 * q + 1];
        if (o.status == 2 || n < 1) return c->fail(EDK_ERR_ZERO_START, "batched ground states: zero start vector");
        const double *d = al.data() + q * ld, *e = be.data() + q * ld + 1;
        for (int k = 0; k < n; ++k)
            if (!std::isfinite(d[k]) || !std::isfinite(e[k])) return c->fail(EDK_ERR_NOT_FINITE, "non-finite Lanczos coefficient");
        const int ne = items[q].ne;
        const int m = std::min(ne, n);
        std::vector<double> w(m), wp(m, 1e300);
        tridiag_lowest(n, d, e, m, w.data());
        if (n > 2) tridiag_lowest(n - 1, d, e, std::min(m, n - 1), wp.data());
        coef_off[q] = (int64_t)coef.size();
        ptr_off[q] = (int64_t)ptrs.size();
        int kept = 0;
        std::vector<double> kv;   // kept coefficient vectors
        for (int j = 0; j < m; ++j) {
            const bool conv = n > 2 && j < n - 1 && std::fabs(w[j] - wp[j]) < tolerance;
            const bool inwin = w[j] >= w[0] && w[j] <= w[0] + demax;
            if (!(j == 0 || (conv && inwin))) continue;
            std::vector<double> prev, v(n);
            int np = 0;
            for (int p = 0; p < kept; ++p)
                if (std::fabs(o.E[p] - w[j]) < 1e-8 * std::max(1.0, std::fabs(w[j]))) {
                    prev.insert(prev.end(), kv.begin() + (size_t)p * n, kv.begin() + (size_t)(p + 1) * n);
                    ++np;
                }
            tridiag_vector(n, d, e, w[j], prev.data(), np, v.data());
            o.E[kept] = w[j];
            o.converged[kept] = conv ? 1 : 0;
            kv.insert(kv.end(), v.begin(), v.end());
            void *p = nullptr;
            if (cudaMalloc(&p, (size_t)hs[order[q]]->dim * 8) != cudaSuccess) {
                (void)cudaGetLastError();
                return c->fail(EDK_ERR_NOMEM, "batched ground states: state vector");
            }
            o.psi[kept] = p;
            ptrs.push_back(p);
            ++kept;
        }
        o.nkept = kept;
        coef.insert(coef.end(), kv.begin(), kv.end());
    }
    // ---- pass 2: the kept states of every sector ----
    if ((rc = c->cuda(upload(d_coef, coef, st), "upload coef"))) return rc;
    if ((rc = c->cuda(upload(d_ptrs, ptrs, st), "upload state pointers"))) return rc;
    for (int q = 0; q < nsec; ++q) {
        const GsBatchSector &o = out[order[q]];
        items[q].niter_max = o.niter;
        items[q].ne = o.nkept;
        items[q].coef = d_coef.as<double>() + coef_off[q];
        items[q].psi = d_ptrs.as<void *const>() + ptr_off[q];
    }
    if ((rc = c->cuda(upload(d_items, items, st), "upload items"))) return rc;
    c->h2d_bytes += (int64_t)(coef.size() * 8 + ptrs.size() * 8 + items.size() * sizeof(GsItem));
    return launch(2);
}

}  // namespace edk

extern "C" int edk_green_batch(edk_ctx *c, int dtype, int32_t nchain, const edk_chain *ch, int32_t nitergreen,
                               int32_t nw, const double *wn_host, double cutoff_dynamic, int32_t nout,
                               double *G_out, int32_t mode, edk_batch_stats *stats)
{
    if (!c || nchain < 0 || (nchain > 0 && !ch) || nitergreen < 1 || nw < 1 || !wn_host || nout < 1 || !G_out)
        return EDK_ERR_INVALID;
    if (dtype != EDK_F64 && dtype != EDK_F32) return c->fail(EDK_ERR_INVALID, "dtype");
    std::memset(G_out, 0, sizeof(double) * 2 * (size_t)nout * nw);
    if (stats) std::memset(stats, 0, sizeof *stats);
    if (nchain == 0) return EDK_OK;
    for (int i = 0; i < nchain; ++i)
        if (!ch[i].target || !ch[i].start_dev || ch[i].out < 0 || ch[i].out >= nout || (ch[i].iph != 1 && ch[i].iph != 2))
            return c->fail(EDK_ERR_INVALID, "chain %d: bad target/start/out/iph", i);
    if (mode != 1)
        for (int i = 0; i < nchain; ++i)
            if (ch[i].target->sz)
                return c->fail(EDK_ERR_UNSUPPORTED, "chain %d: Nambu targets run with mode 1", i);
    cudaStream_t st = c->stream;
    int rc;
    if (mode == 1) {
        // per-chain launches: one grid per Lanczos step (edk_green_chain)
        std::vector<double> G(2 * (size_t)nw);
        int64_t steps = 0;
        for (int i = 0; i < nchain; ++i) {
            int32_t nd = 0;
            if ((rc = edk_green_chain(ch[i].target, dtype, ch[i].start_dev, nitergreen, ch[i].e0, ch[i].iph, nw,
                                      wn_host, cutoff_dynamic, G.data(), nullptr, nullptr, &nd)))
                return rc;
            steps += nd;
            double *o = G_out + (size_t)ch[i].out * 2 * nw;
            for (int w = 0; w < 2 * nw; ++w) o[w] += ch[i].weight * G[w];
        }
        if (stats) { stats->steps = steps; stats->chains = nchain; }
        return EDK_OK;
    }
    // ---- persistent work queue (a cluster of blocks per chain) ----
    std::vector<const edk_h *> hs;
    std::vector<HamDev> hd;
    std::vector<BatchItem> items(nchain);
    std::vector<int> order(nchain);
    int64_t maxdim = 0, maxdup = 0;
    for (int i = 0; i < nchain; ++i) {
        const edk_h *h = ch[i].target;
        int idx = -1;
        for (size_t q = 0; q < hs.size(); ++q)
            if (hs[q] == h) idx = (int)q;
        if (idx < 0) { idx = (int)hs.size(); hs.push_back(h); hd.push_back(h->H); }
        maxdim = std::max(maxdim, h->dim);
        maxdup = std::max(maxdup, h->dup);
        order[i] = i;
    }
    if (maxdup * (dtype == EDK_F64 ? 8 : 4) > 96 * 1024)
        return c->fail(EDK_ERR_UNSUPPORTED, "batched chains need rows of at most 96 KB (use mode 1)");
    // largest chains first (longest-processing-time order)
    std::sort(order.begin(), order.end(), [&](int a, int b) {
        const int64_t wa = ch[a].target->dim * std::min<int64_t>(nitergreen, ch[a].target->dim);
        const int64_t wb = ch[b].target->dim * std::min<int64_t>(nitergreen, ch[b].target->dim);
        return wa > wb;
    });
    const size_t ld = (size_t)nitergreen + 1;
    if ((rc = c->cuda(c->b_alpha.ensure(sizeof(double) * ld * nchain), "alloc"))) return rc;
    if ((rc = c->cuda(c->b_beta.ensure(sizeof(double) * ld * nchain), "alloc"))) return rc;
    if ((rc = c->cuda(c->b_done.ensure(sizeof(int32_t) * nchain), "alloc"))) return rc;
    for (int q = 0; q < nchain; ++q) {
        const int i = order[q];
        const edk_h *h = ch[i].target;
        int idx = 0;
        for (size_t z = 0; z < hs.size(); ++z)
            if (hs[z] == h) idx = (int)z;
        BatchItem &b = items[q];
        b.ham = idx;
        b.niter = (int32_t)std::min<int64_t>(nitergreen, h->dim);
        b.dim = h->dim;
        b.start = ch[i].start_dev;
        b.gamma1 = ch[i].e0;
        b.cutoff_dynamic = cutoff_dynamic;
        b.alpha = c->b_alpha.as<double>() + (size_t)q * ld;
        b.beta = c->b_beta.as<double>() + (size_t)q * ld;
        b.done = c->b_done.as<int32_t>() + q;
    }
    if ((rc = c->cuda(upload(c->b_hams, hd, st), "upload hams"))) return rc;
    if ((rc = c->cuda(upload(c->b_items, items, st), "upload items"))) return rc;
    if ((rc = c->cuda(c->b_queue.ensure(sizeof(int)), "alloc"))) return rc;
    c->h2d_bytes += (int64_t)(hd.size() * sizeof(HamDev) + items.size() * sizeof(BatchItem));
    const size_t es = dtype == EDK_F64 ? 8 : 4;

    // ---- autotune the launch shape for this problem class ----
    // (the number of chains, to a power of two: it decides how many blocks one gets)
    int nclass = 0;
    while ((1 << nclass) < nchain && nclass < 10) ++nclass;
    char key[96];
    snprintf(key, sizeof key, "%d:%lld:%lld:%d", dtype, (long long)maxdup, (long long)maxdim, nclass);
    edk_ctx::BatchShape shape{0, 0, 0};
    for (auto &kv : c->batch_tuned)
        if (kv.first == key && c->kernel_path < 16) shape = kv.second;
    auto run = [&](const edk_ctx::BatchShape &s, int nitems, double *ms) -> int {
        const int nclus = std::min(s.clusters, nitems), grid = nclus * s.cluster;
        int r2 = c->cuda(c->b_work.ensure(es * 4 * (size_t)maxdim * nclus), "alloc batch workspace");
        if (r2) return r2;
        r2 = c->cuda(cudaMemsetAsync(c->b_queue.p, 0, sizeof(int), st), "memset");
        if (r2) return r2;
        cudaEvent_t a = c->get_event(), b = c->get_event();
        cudaEventRecord(a, st);
        r2 = c->cuda(launch_batch(dtype, s.cluster, c->b_hams.as<HamDev>(), c->b_items.as<BatchItem>(), nitems,
                                  c->b_queue.as<int>(), c->b_work.p, maxdim, maxdup, 1e-25, grid, s.block, st),
                     "batch kernel");
        c->launches++;
        cudaEventRecord(b, st);
        cudaEventSynchronize(b);
        float t = 0.f;
        cudaEventElapsedTime(&t, a, b);
        c->event_pool.push_back(a);
        c->event_pool.push_back(b);
        if (ms) *ms = t;
        return r2;
    };
    int tuned = 0;
    if (shape.block == 0) {
        // candidates: block size x blocks per chain, timed on the largest items with
        // the chain length cut to 6 steps
        std::vector<edk_ctx::BatchShape> cand;
        for (int cluster : {1, 2, 4, 8, 16})
            for (int block : {128, 256, 512}) {
                // each resident chain holds four work vectors
                const int active = std::min(batch_max_clusters(dtype, cluster, block, maxdup), 4 * c->num_sms);
                if (active >= 1) cand.push_back(edk_ctx::BatchShape{block, cluster, active});
            }
        if (cand.empty()) return c->fail(EDK_ERR_UNSUPPORTED, "no batch launch shape fits");
        if (c->kernel_path >= 16) {
            shape = cand[(size_t)(c->kernel_path - 16) % cand.size()];
        } else {
            const int nsample = std::min<int>(nchain, c->num_sms * 2);
            std::vector<BatchItem> sample(items.begin(), items.begin() + nsample);
            for (auto &b : sample) b.niter = std::min<int32_t>(b.niter, 6);
            if ((rc = c->cuda(upload(c->b_items, sample, st), "upload sample"))) return rc;
            double best = 1e300;
            for (const auto &s : cand) {
                double ms = 0;
                if ((rc = run(s, nsample, &ms))) return rc;
                ++tuned;
                if (ms < best) { best = ms; shape = s; }
            }
            c->batch_tuned.push_back({key, shape});
        }
        if ((rc = c->cuda(upload(c->b_items, items, st), "upload items"))) return rc;
    }
    double ms = 0;
    if ((rc = run(shape, nchain, &ms))) return rc;
    // ---- continued fractions for every chain ----
    std::vector<double> al(ld * nchain), be(ld * nchain);
    std::vector<int32_t> done(nchain);
    cudaMemcpyAsync(al.data(), c->b_alpha.p, sizeof(double) * ld * nchain, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(be.data(), c->b_beta.p, sizeof(double) * ld * nchain, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(done.data(), c->b_done.p, sizeof(int32_t) * nchain, cudaMemcpyDeviceToHost, st);
    if ((rc = c->cuda(cudaStreamSynchronize(st), "sync"))) return rc;
    c->d2h_bytes += (int64_t)(sizeof(double) * 2 * ld * nchain + sizeof(int32_t) * nchain);
    std::vector<int32_t> n(nchain);
    std::vector<double> e(nchain), ph(nchain), scale(nchain);
    int64_t steps = 0;
    for (int q = 0; q < nchain; ++q) {
        const int i = order[q];
        int m = done[q];
        for (int k = 1; k < m; ++k)
            if (!(be[q * ld + k] >= 1e-25)) { m = k; break; }
        n[q] = m;
        steps += done[q];
        e[q] = ch[i].e0;
        ph[q] = ch[i].iph == 1 ? 1.0 : -1.0;
        scale[q] = m > 0 ? be[q * ld] * be[q * ld] : 0.0;
    }
    std::vector<double> G(2 * (size_t)nchain * nw);
    if ((rc = edk_cf_eval(c, nchain, (int32_t)ld, n.data(), al.data(), be.data(), e.data(), ph.data(), scale.data(),
                          nw, wn_host, G.data())))
        return rc;
    for (int q = 0; q < nchain; ++q) {
        const int i = order[q];
        double *o = G_out + (size_t)ch[i].out * 2 * nw;
        for (int w = 0; w < 2 * nw; ++w) o[w] += ch[i].weight * G[(size_t)q * 2 * nw + w];
    }
    if (stats) {
        stats->steps = steps;
        stats->chains = nchain;
        stats->kernel_ms = ms;
        stats->block = shape.block;
        stats->rows = 1;                              // rows a thread sums at a time
        stats->blocks_per_sm = std::max(1, std::min(shape.clusters, nchain) * shape.cluster / c->num_sms);
        stats->tuned_shapes = tuned;
    }
    return EDK_OK;
}
