// Device kernels of the Nambu (Sz) sectors: H*v of HAIMsz_multr /
// HAIMsz_mult_fly_r (HAIMsz.f90:453-808) fused with the Lanczos modes of the
// row kernel, and c / c+ of apply_Csz_updo / apply_Csz_N_updo
// (apply_C.f90:344-483).
//
// One thread block per row of equal high half h (the down holes), threads
// over the row's low halves, so the x reads of the own row and of targets
// that keep h are coalesced.  Per element:
//   acc = QUART_INT_SZ * x                               (table by impurity configuration)
//   tabulated order: acc += (sum of the occupied orbitals' diagonal energies) * x
//   on-the-fly order: acc += e_o * x for each occupied orbital o in turn
//   acc += (+-t) * x[rank(target)] for each term c+_tgt c_src in the list whose
//          source is occupied and target empty (sign: parity of the occupied
//          orbitals strictly between)
// in the reference's order with separate multiply and add, so the FP64 result
// equals a sequential FP64 evaluation bit for bit.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <type_traits>
#include "edk_internal.h"
#include "edk_device.cuh"

namespace edk {

namespace {

constexpr int kSzBlock = 256;      // threads of a block at most (sz_wide_kernel has its own)

// One hole-hole or pairing term of a row's list whose high-half condition
// holds on the row.  Pairing: the state must have `want` in bit 17 of its
// entry of the orbital's table (SzDev::pair), which gives the target column.
struct RowTerm {
    uint64_t xoff;         // byte offset of the target row
    uint32_t tab;          // pairing: byte offset of the low orbital's table
    uint32_t want;         // pairing: the low orbital's bit | 0 or 1 << 17
};


// The row's lists, built by the block's first warp: the terms of each run whose
// high half applies, in term order (seg[run] .. seg[run + 1] are the run's), and
// the diagonal energies that the row adds after SzDev::pdiag (tabulated order:
// the occupied hole baths; on the fly: every up orbital, with its low bit, and
// the occupied holes).
template <typename T>
__device__ __forceinline__ void sz_row_lists(const SzDev &S, uint32_t h, const SzRun *runs, RowTerm *rt, double *hv,
                                             int *seg, double *de, uint32_t *db, int *nde)
{
    const int lane = threadIdx.x & 31, ns = S.ns;
    const uint32_t lowmask = (1u << ns) - 1u, lt = (1u << lane) - 1u;
    int n = 0;
    for (int t0 = 0; t0 < S.nterm; t0 += 32) {
        const int t = t0 + lane;
        bool pass = false;
        SzTerm tm;
        int run = 0, kind = 0;
        uint32_t hsrc = 0u, htgt = 0u;
        if (t < S.nterm) {
            tm = S.terms[t];
            run = S.term_run[t];
            kind = runs[run].kind;
            hsrc = tm.src >> ns;
            htgt = tm.tgt >> ns;
            // a pairing term whose target row does not exist has no state to act on
            const int kt = S.sec.npart - __popc(h ^ hsrc ^ htgt);
            pass = kind != 0 && (h & hsrc) == hsrc && (h & htgt) == 0u && kt >= 0 && kt <= ns;
        }
        const unsigned b = __ballot_sync(0xffffffffu, pass);
        const int pos = n + __popc(b & lt);
        if (t < S.nterm && runs[run].first == t) seg[run] = pos;
        if (pass) {
            RowTerm o;
            const uint32_t low = (tm.src | tm.tgt) & lowmask;
            o.xoff = (uint64_t)S.sec.off_h[h ^ hsrc ^ htgt] * sizeof(T);
            o.tab = kind == 2 ? (uint32_t)S.pair_row[31 - __clz(low)] << (ns + 2) : 0u;
            o.want = kind == 2 ? low | (tm.src & lowmask ? 1u << 17 : 0u) : 0u;
            rt[pos] = o;
            hv[pos] = (__popc(h & (tm.btw >> ns)) & 1) ? -tm.h : tm.h;
        }
        n += __popc(b);
    }
    if (lane == 0) seg[S.nrun] = n;
    n = 0;
    for (int t0 = S.order == 0 ? 2 * S.nc + S.nb : 0; t0 < S.ndiag; t0 += 32) {
        const int t = t0 + lane;
        uint32_t bit = 0u;
        if (t < S.ndiag) bit = S.diag_bit[t];
        const bool pass = (bit & lowmask) != 0u || (h & (bit >> ns)) != 0u;
        const unsigned b = __ballot_sync(0xffffffffu, pass);
        if (pass) {
            const int pos = n + __popc(b & lt);
            de[pos] = S.diag_e[t];
            db[pos] = bit & lowmask;
        }
        n += __popc(b);
    }
    if (lane == 0) *nde = n;
}

// g with its sign flipped where bit 16 of the table entry is set
__device__ __forceinline__ double with_sign(double g, uint32_t t)
{
    return __hiloint2double(__double2hiint(g) ^ (int)((t & 0x10000u) << 15), __double2loint(g));
}

// Row kernel: one block per row, two columns per thread, the own row staged in
// shared memory when STAGE.  Same arithmetic, in the same order, as
// sz_row_simple_kernel.  What bounds it is instructions and the gathers'
// latency, not bytes, so everything that depends on the low half alone comes
// from tables read along the row: the diagonal up to the hole baths
// (SzDev::pdiag), the up-up runs' targets (their entries carry the offset of
// the signed value, so a hop is two shared loads, a multiply and an add) and the
// pairing terms' target columns and signs (SzDev::pair).  The lists take one
// warp a few ballots per row instead of block-wide compactions.
template <typename T, bool STAGE, int NTMAX, int MINB>
__global__ void __launch_bounds__(NTMAX, MINB) sz_row_kernel(const SzDev S, const RowArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int n_diag;
    const int nq = 1 << (2 * S.nc);
    RowTerm *rt = reinterpret_cast<RowTerm *>(smem_raw);
    double *hv = reinterpret_cast<double *>(rt + S.nterm);
    double *h2 = hv + S.nterm;                                      // {h, -h} of every term, 0
    double *qs = h2 + 2 * S.nterm + 1;
    double *de = qs + nq;
    SzRun *runs = reinterpret_cast<SzRun *>(de + S.ndiag);
    uint32_t *db = reinterpret_cast<uint32_t *>(runs + S.nrun);
    int *seg = reinterpret_cast<int *>(db + S.ndiag);
    T *xs = reinterpret_cast<T *>(smem_raw + S.smem_lists);
    chain_next();
    for (int t = threadIdx.x; t < nq; t += blockDim.x) qs[t] = S.quart[t];
    for (int t = threadIdx.x; t < S.nterm; t += blockDim.x) { h2[2 * t] = S.terms[t].h; h2[2 * t + 1] = -S.terms[t].h; }
    if (threadIdx.x == 0) h2[2 * S.nterm] = 0.0;
    for (int t = threadIdx.x; t < S.nrun; t += blockDim.x) runs[t] = S.runs[t];
    // the first row's lists before the wait (no kernel writes the tables they come from)
    __syncthreads();
    if (threadIdx.x < 32 && blockIdx.x < S.sec.nrows)
        sz_row_lists<T>(S, S.sec.row_h[blockIdx.x], runs, rt, hv, seg, de, db, &n_diag);
    chain_wait();
    const int ks = step_index(a);
    StepScalars sc;
    if (!step_scalars(a, ks, sc)) return;

    const T *x = static_cast<const T *>(a.x);
    const int ns = S.ns, nb = S.nb, nc = S.nc, nrun = S.nrun, NT = blockDim.x, lane = threadIdx.x & 31;
    const uint32_t cm = (1u << nc) - 1u;
    const uint32_t nlow = 1u << ns;
    const unsigned char *h2b = reinterpret_cast<const unsigned char *>(h2);
    const uint32_t pad = (uint32_t)S.nterm << 20;                   // entries past a state's last: the 0 in h2
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int r = blockIdx.x; r < S.sec.nrows; r += gridDim.x) {
        const uint32_t h = S.sec.row_h[r];
        const int k = S.sec.npart - __popc(h);
        const int c0 = S.class_start[k], len = S.class_start[k + 1] - c0;
        const uint32_t base = S.sec.off_h[h];
        __syncthreads();                       // the previous row is done with the lists
        if (r != blockIdx.x && threadIdx.x < 32) sz_row_lists<T>(S, h, runs, rt, hv, seg, de, db, &n_diag);
        if (STAGE) stage_row<T>(xs, x + base, len);
        __syncthreads();
        const int nd = n_diag;
        const uint32_t hcfg = (h >> nb) & cm;
        const uint32_t *__restrict__ ell = S.ell + c0;
        const uint32_t *__restrict__ pair = S.pair + c0;
        const double *__restrict__ pdiag = S.pdiag + ((size_t)hcfg << ns) + c0;
        const T *xrow = x + base;
        const uint32_t *__restrict__ kell = S.kell + k * nrun;
        // a warp owns 64 adjacent columns, two per lane: c and c + step (step = 32 where the
        // warp's columns all exist, so that it folds into the loads' immediate offsets;
        // lanes past the row's end repeat its last column and store nothing)
        auto columns = [&](int cw, auto full) {
            constexpr bool FULL = decltype(full)::value;
            const int c = FULL ? cw + lane : min(cw + lane, len - 1);
            const int step = FULL ? 32 : min(cw + 32 + lane, len - 1) - c;
            const uint32_t l[2] = {(uint32_t)S.low_states[c0 + c], (uint32_t)S.low_states[c0 + c + step]};
            const T xo[2] = {STAGE ? xs[c] : xrow[c], STAGE ? xs[c + step] : xrow[c + step]};
            double acc[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) acc[e] = fmul(qs[((l[e] >> nb) & cm) | (hcfg << nc)], (double)xo[e]);
            if (S.order == 0) {
                double d[2] = {__ldg(pdiag + c), __ldg(pdiag + c + step)};
                for (int o = 0; o < nd; ++o) {
                    d[0] = fadd(d[0], de[o]);
                    d[1] = fadd(d[1], de[o]);
                }
                acc[0] = hmadd<T>(acc[0], d[0], xo[0]);
                acc[1] = hmadd<T>(acc[1], d[1], xo[1]);
            } else {
                for (int o = 0; o < nd; ++o)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        if (!db[o] || (l[e] & db[o])) acc[e] = hmadd<T>(acc[e], de[o], xo[e]);
            }
            for (int run = 0; run < nrun; ++run) {
                const int kind = runs[run].kind, e0 = seg[run], e1 = seg[run + 1];
                // Loads are unconditional (a lane without the term reads an element that is
                // there), only the sums are predicated.
                if (kind == 0) {
                    // this state's active terms from the run's table
                    const uint32_t *tab = ell + (runs[run].ell_off + c);
                    const int n = (int)kell[run];
#pragma unroll 4
                    for (int q = 0; q < n; ++q, tab += nlow) {
                        const uint32_t u[2] = {__ldg(tab), __ldg(tab + step)};
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const double g = *reinterpret_cast<const double *>(h2b + (u[e] >> 16));
                            const uint32_t col = u[e] & 0xFFFFu;
                            const T xv = STAGE ? xs[col] : xrow[col];
                            if (u[e] < pad) acc[e] = hmadd<T>(acc[e], g, xv);
                        }
                    }
                } else if (kind == 1) {
                    // the same column of another row
                    const unsigned char *xc = reinterpret_cast<const unsigned char *>(x + c);
#pragma unroll 4
                    for (int q = e0; q < e1; ++q) {
                        const T *p = reinterpret_cast<const T *>(xc + rt[q].xoff);
                        const T x0 = p[0], x1 = p[step];
                        const double g = hv[q];
                        acc[0] = hmadd<T>(acc[0], g, x0);
                        acc[1] = hmadd<T>(acc[1], g, x1);
                    }
                } else {
                    // pairing: bit 17 of the table entry is the orbital's occupation, bit 16
                    // the parity of the orbitals above it, the rest the target column.
                    // Adjacent columns agree in their high orbitals, so a vote over the
                    // warp's columns drops the terms none of them has.
                    const uint32_t any = __reduce_or_sync(0xffffffffu, l[0] | l[1]);
                    const uint32_t all = __reduce_and_sync(0xffffffffu, l[0] & l[1]);
                    const unsigned char *xb = reinterpret_cast<const unsigned char *>(x);
                    const unsigned char *pc = reinterpret_cast<const unsigned char *>(pair + c);
                    for (int b0 = e0; b0 < e1; b0 += 32) {
                        bool need = false;
                        if (b0 + lane < e1) {
                            const uint32_t w = rt[b0 + lane].want;
                            need = (w >> 17) ? (any & w) != 0u : (all & w) == 0u;
                        }
                        unsigned m = __ballot_sync(0xffffffffu, need);
                        while (m) {
                            // two terms at a time (the second repeats the first at the end)
                            const int qa = b0 + __ffs(m) - 1;
                            m &= m - 1u;
                            const bool more = m != 0u;
                            const int qb = more ? b0 + __ffs(m) - 1 : qa;
                            m &= m - 1u;
                            const RowTerm oa = rt[qa], ob = rt[qb];
                            const uint32_t *pa = reinterpret_cast<const uint32_t *>(pc + oa.tab);
                            const uint32_t *pb = reinterpret_cast<const uint32_t *>(pc + ob.tab);
                            uint32_t ta[2] = {__ldg(pa), __ldg(pa + step)}, tb[2] = {__ldg(pb), __ldg(pb + step)};
                            const T *ra = reinterpret_cast<const T *>(xb + oa.xoff);
                            const T *rb = reinterpret_cast<const T *>(xb + ob.xoff);
                            T va[2], vb[2];
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                ta[e] ^= oa.want & 0x20000u;
                                tb[e] ^= ob.want & 0x20000u;
                                va[e] = ra[ta[e] & 0x20000u ? 0u : ta[e] & 0xFFFFu];
                                vb[e] = rb[tb[e] & 0x20000u ? 0u : tb[e] & 0xFFFFu];
                            }
                            const double ga = hv[qa], gb = hv[qb];
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                if (!(ta[e] & 0x20000u)) acc[e] = hmadd<T>(acc[e], with_sign(ga, ta[e]), va[e]);
                                if (more && !(tb[e] & 0x20000u))
                                    acc[e] = hmadd<T>(acc[e], with_sign(gb, tb[e]), vb[e]);
                            }
                        }
                    }
                }
            }
            if (FULL || cw + lane < len) row_epilogue<T>(a, sc, (int64_t)base + c, acc[0], xo[0], s0, s1, s2);
            if (FULL || cw + 32 + lane < len)
                row_epilogue<T>(a, sc, (int64_t)base + c + step, acc[1], xo[1], s0, s1, s2);
        };
        for (int cw = 2 * (int)(threadIdx.x - lane); cw < len; cw += 2 * NT) {
            if (cw + 64 <= len) columns(cw, std::true_type());
            else columns(cw, std::false_type());
        }
    }
    if (a.mode == kModeHv) return;
    double v[3] = {s0, s1, s2};
    if (grid_sum<3>(v, a.partials, a.counter, a.sums_out))
        if (a.mode == kModeFirst || a.mode == kModeStep) lanczos_finalize(a, ks, v, sc.gam1);
}

// One element global -> shared, asynchronous, where i < n (predicated, no branch).
__device__ __forceinline__ void copy_async(double *dst, const double *src, int i, int n)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\t@p cp.async.ca.shared.global [%0], [%1], 8;\n\t}"
                 ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(i), "r"(n) : "memory");
}
__device__ __forceinline__ void copy_async(float *dst, const float *src, int i, int n)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\t@p cp.async.ca.shared.global [%0], [%1], 4;\n\t}"
                 ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(i), "r"(n) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Row kernel for rows of which three fit in shared memory: the block keeps all
// columns of its row in registers (at most kSlots per thread, tid + i NT) and
// walks the row's terms together.  The target row of a pairing term is copied
// whole into one of two buffers while the term before it is summed, so its
// gather is a shared load; in sz_row_kernel each such gather waits for a table
// entry and then for x, two dependent loads from L2 or DRAM per pair of terms, and
// that latency is most of its time.  Hole-hole terms read the other row directly,
// one coalesced load per column.  The loops over a thread's columns are unrolled
// for the row's number of them, so offsets are immediates and the tests that
// remain are predicates: with a branch per column and term the kernel issued three
// times the instructions.  The loads of a column past the row's end repeat the
// thread's first column, the shared load of a state without the term reads an
// element that is not used (a buffer is as long as the longest class it may index).
constexpr int kSlots = 8;

template <typename T, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) sz_wide_kernel(const SzDev S, const RowArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int n_diag;
    const int nq = 1 << (2 * S.nc);
    RowTerm *rt = reinterpret_cast<RowTerm *>(smem_raw);
    double *hv = reinterpret_cast<double *>(rt + S.nterm);
    double *h2 = hv + S.nterm;                                      // {h, -h} of every term, 0
    double *qs = h2 + 2 * S.nterm + 1;
    double *de = qs + nq;
    SzRun *runs = reinterpret_cast<SzRun *>(de + S.ndiag);
    uint32_t *db = reinterpret_cast<uint32_t *>(runs + S.nrun);
    int *seg = reinterpret_cast<int *>(db + S.ndiag);
    T *xs = reinterpret_cast<T *>(smem_raw + S.smem_lists);         // own row, two buffers
    const int pitch = S.sec.pitch, tid = threadIdx.x;
    chain_next();
    for (int t = tid; t < nq; t += NT) qs[t] = S.quart[t];
    for (int t = tid; t < S.nterm; t += NT) { h2[2 * t] = S.terms[t].h; h2[2 * t + 1] = -S.terms[t].h; }
    if (tid == 0) h2[2 * S.nterm] = 0.0;
    for (int t = tid; t < S.nrun; t += NT) runs[t] = S.runs[t];
    // the first row's lists before the wait (no kernel writes the tables they come from)
    __syncthreads();
    if (tid < 32 && blockIdx.x < S.sec.nrows)
        sz_row_lists<T>(S, S.sec.row_h[blockIdx.x], runs, rt, hv, seg, de, db, &n_diag);
    chain_wait();
    const int ks = step_index(a);
    StepScalars sc;
    if (!step_scalars(a, ks, sc)) return;

    const T *x = static_cast<const T *>(a.x);
    const int ns = S.ns, nb = S.nb, nc = S.nc, nrun = S.nrun;
    const uint32_t cm = (1u << nc) - 1u, nlow = 1u << ns;
    const unsigned char *h2b = reinterpret_cast<const unsigned char *>(h2);
    const unsigned char *xb = reinterpret_cast<const unsigned char *>(x);
    const uint32_t pad = (uint32_t)S.nterm << 20;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int r = blockIdx.x; r < S.sec.nrows; r += gridDim.x) {
        const uint32_t h = S.sec.row_h[r];
        const int k = S.sec.npart - __popc(h);
        const int c0 = S.class_start[k], len = S.class_start[k + 1] - c0;
        // lengths of the rows that a pairing term can reach
        const int len_less = k > 0 ? c0 - S.class_start[k - 1] : 0;
        const int len_more = k < ns ? S.class_start[k + 2] - S.class_start[k + 1] : 0;
        const uint32_t base = S.sec.off_h[h];
        __syncthreads();                       // the previous row is done with the lists and buffers
#pragma unroll
        for (int i = 0; i < kSlots; ++i) copy_async(xs + tid + i * NT, x + base + tid + i * NT, tid + i * NT, len);
        copy_commit();
        if (r != blockIdx.x && tid < 32) sz_row_lists<T>(S, h, runs, rt, hv, seg, de, db, &n_diag);
        copy_wait<0>();
        __syncthreads();
        const int nd = n_diag;
        const uint32_t hcfg = (h >> nb) & cm;
        const uint32_t *__restrict__ kell = S.kell + k * nrun;
        auto row = [&](auto slots) {
            constexpr int NS = decltype(slots)::value;
            const int cb = min(tid, len - 1);                   // the thread's first column
            const bool last = tid + (NS - 1) * NT < len;
            const int ol = last ? (NS - 1) * NT : 0;            // offset of its last one
            auto off = [&](int i) { return i < NS - 1 ? i * NT : ol; };
            const uint16_t *__restrict__ low = S.low_states + c0 + cb;
            const double *__restrict__ pdiag = S.pdiag + ((size_t)hcfg << ns) + c0 + cb;
            double acc[NS];
            {
                double d[NS];
                uint32_t l[NS];
#pragma unroll
                for (int i = 0; i < NS; ++i) {
                    l[i] = (uint32_t)__ldg(low + off(i));
                    d[i] = S.order == 0 ? __ldg(pdiag + off(i)) : 0.0;
                }
#pragma unroll
                for (int i = 0; i < NS; ++i)
                    acc[i] = fmul(qs[((l[i] >> nb) & cm) | (hcfg << nc)], (double)xs[cb + off(i)]);
                if (S.order == 0) {
                    for (int o = 0; o < nd; ++o) {
                        const double e = de[o];
#pragma unroll
                        for (int i = 0; i < NS; ++i) d[i] = fadd(d[i], e);
                    }
#pragma unroll
                    for (int i = 0; i < NS; ++i) acc[i] = hmadd<T>(acc[i], d[i], xs[cb + off(i)]);
                } else {
                    for (int o = 0; o < nd; ++o) {
                        const double e = de[o];
                        const uint32_t bit = db[o];
#pragma unroll
                        for (int i = 0; i < NS; ++i) {
                            const double v = hmadd<T>(acc[i], e, xs[cb + off(i)]);
                            acc[i] = !bit || (l[i] & bit) ? v : acc[i];
                        }
                    }
                }
            }
            for (int run = 0; run < nrun; ++run) {
                const int kind = runs[run].kind, e0 = seg[run], e1 = seg[run + 1];
                if (kind == 0) {
                    // this state's active terms from the run's table
                    const uint32_t *tab = S.ell + (runs[run].ell_off + c0 + cb);
                    const int n = (int)kell[run];
#pragma unroll 2
                    for (int q = 0; q < n; ++q, tab += nlow) {
                        uint32_t u[NS];
#pragma unroll
                        for (int i = 0; i < NS; ++i) u[i] = __ldg(tab + off(i));
#pragma unroll
                        for (int i = 0; i < NS; ++i) {
                            const double g = *reinterpret_cast<const double *>(h2b + (u[i] >> 16));
                            const T v = xs[u[i] & 0xFFFFu];
                            if (u[i] < pad) acc[i] = hmadd<T>(acc[i], g, v);
                        }
                    }
                } else if (kind == 1) {
                    // the same column of another row
                    const unsigned char *xc = reinterpret_cast<const unsigned char *>(x + cb);
#pragma unroll 2
                    for (int q = e0; q < e1; ++q) {
                        const T *p = reinterpret_cast<const T *>(xc + rt[q].xoff);
                        T v[NS];
#pragma unroll
                        for (int i = 0; i < NS; ++i) v[i] = p[off(i)];
                        const double g = hv[q];
#pragma unroll
                        for (int i = 0; i < NS; ++i) acc[i] = hmadd<T>(acc[i], g, v[i]);
                    }
                } else {
                    // pairing: bit 17 of the table entry is the orbital's occupation, bit 16 the
                    // parity of the orbitals above it, the rest the target column
                    const unsigned char *pc = reinterpret_cast<const unsigned char *>(S.pair + c0 + cb);
                    auto fetch = [&](int q) {
                        const RowTerm o = rt[q];
                        const int lt = (o.want >> 17) ? len_less : len_more;
                        const T *src = reinterpret_cast<const T *>(xb + o.xoff) + tid;
                        T *dst = xs + pitch * (1 + (q & 1)) + tid;
#pragma unroll
                        for (int i = 0; i < kSlots; ++i) copy_async(dst + i * NT, src + i * NT, tid + i * NT, lt);
                    };
                    if (e0 < e1) fetch(e0);
                    copy_commit();
                    for (int q = e0; q < e1; ++q) {
                        const RowTerm o = rt[q];
                        const uint32_t *p = reinterpret_cast<const uint32_t *>(pc + o.tab);
                        uint32_t t[NS];
#pragma unroll
                        for (int i = 0; i < NS; ++i) t[i] = __ldg(p + off(i));
                        if (q + 1 < e1) fetch(q + 1);
                        copy_commit();
                        copy_wait<1>();            // term q is in, q + 1 on its way
                        __syncthreads();
                        const T *buf = xs + pitch * (1 + (q & 1));
                        const double g = hv[q];
#pragma unroll
                        for (int i = 0; i < NS; ++i) {
                            const T v = buf[t[i] & 0xFFFFu];
                            if (!((t[i] ^ o.want) & 0x20000u)) acc[i] = hmadd<T>(acc[i], with_sign(g, t[i]), v);
                        }
                        __syncthreads();           // before the buffer is filled again
                    }
                    copy_wait<0>();
                }
            }
#pragma unroll
            for (int i = 0; i < NS; ++i)
                if (i < NS - 1 || last)
                    row_epilogue<T>(a, sc, (int64_t)base + tid + i * NT, acc[i], xs[tid + i * NT], s0, s1, s2);
        };
        switch ((len + NT - 1) / NT) {
        case 1: row(std::integral_constant<int, 1>()); break;
        case 2: row(std::integral_constant<int, 2>()); break;
        case 3: row(std::integral_constant<int, 3>()); break;
        case 4: row(std::integral_constant<int, 4>()); break;
        case 5: row(std::integral_constant<int, 5>()); break;
        case 6: row(std::integral_constant<int, 6>()); break;
        case 7: row(std::integral_constant<int, 7>()); break;
        default: row(std::integral_constant<int, 8>()); break;
        }
    }
    if (a.mode == kModeHv) return;
    double v[3] = {s0, s1, s2};
    if (grid_sum<3>(v, a.partials, a.counter, a.sums_out))
        if (a.mode == kModeFirst || a.mode == kModeStep) lanczos_finalize(a, ks, v, sc.gam1);
}

// Reference form: every state walks the whole term list (kernel path 1).
template <typename T>
__global__ void __launch_bounds__(kSzBlock) sz_row_simple_kernel(const SzDev S, const RowArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SzTerm *ts = reinterpret_cast<SzTerm *>(smem_raw);
    const int nq = 1 << (2 * S.nc);
    double *qs = reinterpret_cast<double *>(ts + S.nterm);
    double *des = qs + nq;
    uint32_t *dbs = reinterpret_cast<uint32_t *>(des + S.ndiag);
    for (int t = threadIdx.x; t < S.nterm; t += blockDim.x) ts[t] = S.terms[t];
    chain_next();
    for (int t = threadIdx.x; t < nq; t += blockDim.x) qs[t] = S.quart[t];
    for (int t = threadIdx.x; t < S.ndiag; t += blockDim.x) { des[t] = S.diag_e[t]; dbs[t] = S.diag_bit[t]; }

    chain_wait();
    const int ks = step_index(a);
    StepScalars sc;
    if (!step_scalars(a, ks, sc)) return;
    __syncthreads();

    const T *x = static_cast<const T *>(a.x);
    const int ns = S.ns, nb = S.nb, nc = S.nc, nterm = S.nterm, ndiag = S.ndiag;
    const uint32_t lowmask = (1u << ns) - 1u, cm = (1u << nc) - 1u;
    const uint32_t *__restrict__ off_h = S.sec.off_h;
    const uint16_t *__restrict__ rank_low = S.rank_low;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int r = blockIdx.x; r < S.sec.nrows; r += gridDim.x) {
        const uint32_t h = S.sec.row_h[r];
        const int k = S.sec.npart - __popc(h);
        const int c0 = S.class_start[k], len = S.class_start[k + 1] - c0;
        const int64_t base = off_h[h];
        const uint32_t hs = h << ns;
        for (int c = threadIdx.x; c < len; c += blockDim.x) {
            const uint32_t s = (uint32_t)S.low_states[c0 + c] | hs;
            const int64_t i = base + c;
            const T xo = x[i];
            const uint32_t cfg = ((s >> nb) & cm) | (((s >> (ns + nb)) & cm) << nc);
            double acc = fmul(qs[cfg], (double)xo);
            if (S.order == 0) {
                double d = 0.0;
                for (int o = 0; o < ndiag; ++o)
                    if (s & dbs[o]) d = fadd(d, des[o]);
                acc = hmadd<T>(acc, d, xo);
            } else {
                for (int o = 0; o < ndiag; ++o)
                    if (s & dbs[o]) acc = hmadd<T>(acc, des[o], xo);
            }
            for (int t = 0; t < nterm; ++t) {
                const uint32_t src = ts[t].src, tgt = ts[t].tgt;
                if (!(s & src) || (s & tgt)) continue;
                const uint32_t s2t = s ^ src ^ tgt;
                const int64_t j = (int64_t)off_h[s2t >> ns] + rank_low[s2t & lowmask];
                const double hv = (__popc(s & ts[t].btw) & 1) ? -ts[t].h : ts[t].h;
                acc = hmadd<T>(acc, hv, x[j]);
            }
            row_epilogue<T>(a, sc, i, acc, xo, s0, s1, s2);
        }
    }
    if (a.mode == kModeHv) return;
    double v[3] = {s0, s1, s2};
    if (grid_sum<3>(v, a.partials, a.counter, a.sums_out))
        if (a.mode == kModeFirst || a.mode == kModeStep) lanczos_finalize(a, ks, v, sc.gam1);
}

// Gather form of the reference's scatter: every target state looks up its
// source; the map is one-to-one, so each target receives at most one term per
// operator, in operator order.
template <typename T>
__global__ void sz_apply_c_kernel(const SzDev S, const SzSectorDev tgt, int nop, SzOp o0, SzOp o1,
                                  const T *__restrict__ in, T *__restrict__ out)
{
    const int ns = S.ns;
    const uint32_t lowmask = (1u << ns) - 1u;
    for (int r = blockIdx.x; r < tgt.nrows; r += gridDim.x) {
        const uint32_t h = tgt.row_h[r];
        const int k = tgt.npart - __popc(h);
        const int c0 = S.class_start[k], len = S.class_start[k + 1] - c0;
        const int64_t base = tgt.off_h[h];
        for (int c = threadIdx.x; c < len; c += blockDim.x) {
            const uint32_t t = (uint32_t)S.low_states[c0 + c] | (h << ns);
            T acc = T(0);
            for (int q = 0; q < nop; ++q) {
                const SzOp o = q == 0 ? o0 : o1;
                if (((t & o.bit) != 0u) != (o.create != 0)) continue;
                const uint32_t s = t ^ o.bit;
                if ((s & o.pmask) != o.pwant) continue;
                // create / destroy sign: occupied orbitals above the bit, on the result
                const uint32_t above = t & ~((o.bit << 1) - 1u);
                const int sg = (__popc(above) & 1) ? -o.sgn : o.sgn;
                const T v = in[(int64_t)S.sec.off_h[s >> ns] + S.rank_low[s & lowmask]];
                if (q == 0) acc = sg > 0 ? v : -v;
                else acc = sg > 0 ? fadd(acc, v) : fsub(acc, v);
            }
            out[base + c] = acc;
        }
    }
}

size_t sz_smem(const SzDev &S)
{
    return (size_t)S.nterm * sizeof(SzTerm) + sizeof(double) * ((size_t)1 << (2 * S.nc)) +
           (size_t)S.ndiag * (sizeof(double) + sizeof(uint32_t));
}

// Threads of a block for rows of at most maxlen columns.
int sz_block(int maxlen, int most = kSzBlock)
{
    int b = ((maxlen + 31) / 32) * 32;
    if (b > most) b = most;
    if (b < 32) b = 32;
    return b;
}

template <typename K>
cudaError_t launch_one(K kern, int grid, int block, size_t smem, const SzDev &S, const RowArgs &a, cudaStream_t st)
{
    int per_sm = 0;      // allows the shared memory; the callers size the grid themselves
    cudaError_t e = kernel_fit(reinterpret_cast<const void *>(kern), block, smem, &per_sm);
    if (e != cudaSuccess) return e;
    return launch_chained(kern, grid, block, smem, st, S, a);
}

}  // namespace

namespace {
// SzDev::pair, one table per blockIdx.y
__global__ void sz_pair_kernel(const SzDev S, uint32_t *pair)
{
    const uint32_t nlow = 1u << S.ns, p = blockIdx.x * blockDim.x + threadIdx.x, o = S.pair_orb[blockIdx.y];
    if (p >= nlow) return;
    const uint32_t l = (uint32_t)S.low_states[p], above = (nlow - 1u) & ~((2u << o) - 1u);
    pair[(size_t)blockIdx.y * nlow + p] = (uint32_t)S.rank_low[l ^ (1u << o)] | (uint32_t)(__popc(l & above) & 1) << 16 |
                                          ((l >> o) & 1u) << 17;
}
}  // namespace

cudaError_t launch_sz_pair(const SzDev &S, int nrow, uint32_t *pair, cudaStream_t st)
{
    sz_pair_kernel<<<dim3((unsigned)(((1u << S.ns) + 255u) / 256u), (unsigned)nrow), 256, 0, st>>>(S, pair);
    return cudaGetLastError();
}

cudaError_t launch_sz_rows(const SzDev &S, int dtype, const RowArgs &a, int num_sms, int simple, cudaStream_t st)
{
    const size_t eb = dtype == EDK_F64 ? 8 : 4;
    if (simple) {
        const int block = sz_block(S.sec.maxlen);
        int grid = num_sms * std::min(16, 2048 / block);
        if (grid > S.sec.nrows) grid = S.sec.nrows;
        if (grid < 1) grid = 1;
        const size_t smem = sz_smem(S);
        return dtype == EDK_F64 ? launch_one(sz_row_simple_kernel<double>, grid, block, smem, S, a, st)
                                : launch_one(sz_row_simple_kernel<float>, grid, block, smem, S, a, st);
    }
    // The wide kernel where three rows fit in shared memory with at most kSlots columns
    // per thread, and the rows are long: its blocks are sized for the longest class.
    // FP64 H*v, wide against row kernel: half filling 34 / 40 us at ns = 11, 354 / 444 at
    // 13, 1566 / 1780 at 14; 24 / 15 us at ns = 10; few particles, whose rows average far
    // below the longest, 118 / 60 us (ns = 14, 5 particles), 2808 / 1149 us (15, 9).
    const size_t wide = S.smem_lists + 3 * (size_t)S.sec.pitch * eb;
    if (wide <= 220 * 1024 && S.sec.maxlen >= 400 && S.sec.maxlen <= kSlots * 1024 &&
        2 * S.sec.dim >= (int64_t)S.sec.maxlen * S.sec.nrows) {
        // 1024 threads per SM (the register budget) in as many blocks as shared
        // memory and the number of rows allow
        int per_sm = std::max(1, std::min((int)((227 * 1024) / (wide + 2048)), (S.sec.nrows + num_sms - 1) / num_sms));
        int block = per_sm >= 8 ? 128 : per_sm >= 4 ? 256 : per_sm >= 2 ? 512 : 1024;
        while (block < 1024 && S.sec.maxlen > kSlots * block) block *= 2;
        per_sm = std::min(per_sm, 1024 / block);
        const int grid = std::max(1, std::min(num_sms * per_sm, S.sec.nrows));
        if (dtype == EDK_F64)
            return block == 128   ? launch_one(sz_wide_kernel<double, 128>, grid, block, wide, S, a, st)
                   : block == 256 ? launch_one(sz_wide_kernel<double, 256>, grid, block, wide, S, a, st)
                   : block == 512 ? launch_one(sz_wide_kernel<double, 512>, grid, block, wide, S, a, st)
                                  : launch_one(sz_wide_kernel<double, 1024>, grid, block, wide, S, a, st);
        return block == 128   ? launch_one(sz_wide_kernel<float, 128>, grid, block, wide, S, a, st)
               : block == 256 ? launch_one(sz_wide_kernel<float, 256>, grid, block, wide, S, a, st)
               : block == 512 ? launch_one(sz_wide_kernel<float, 512>, grid, block, wide, S, a, st)
                              : launch_one(sz_wide_kernel<float, 1024>, grid, block, wide, S, a, st);
    }
    // Two columns per thread; short rows in blocks of 128 threads, eight per SM, longer
    // ones in blocks of 256, three per SM (their rows in shared memory leave less L1;
    // 87 against 60 us at ns = 14, 5 particles, 15 against 20 us at ns = 10).  The own
    // row is staged when it leaves room for four blocks per SM.
    const bool smem_fits = S.smem_lists + (size_t)S.sec.maxlen * eb <= 52 * 1024;
    const bool small = S.sec.maxlen <= 256 && smem_fits;
    const int most = small ? 128 : 256, blocks = small ? 8 : 3;
    const int block = sz_block((S.sec.maxlen + 1) / 2, most);
    size_t smem = S.smem_lists;
    const size_t row_bytes = (size_t)S.sec.maxlen * eb;
    const bool stage = smem_fits;
    if (stage) smem += row_bytes;
    int per_sm = std::min(16, blocks * most / block);    // the register budget of the launch bounds
    per_sm = std::max(1, std::min(per_sm, (int)((228 * 1024) / (smem + 1024))));
    const int grid = std::max(1, std::min(num_sms * per_sm, S.sec.nrows));
    if (small)                                           // always staged
        return dtype == EDK_F64 ? launch_one(sz_row_kernel<double, true, 128, 8>, grid, block, smem, S, a, st)
                                : launch_one(sz_row_kernel<float, true, 128, 8>, grid, block, smem, S, a, st);
    if (dtype == EDK_F64)
        return stage ? launch_one(sz_row_kernel<double, true, 256, 3>, grid, block, smem, S, a, st)
                     : launch_one(sz_row_kernel<double, false, 256, 3>, grid, block, smem, S, a, st);
    return stage ? launch_one(sz_row_kernel<float, true, 256, 3>, grid, block, smem, S, a, st)
                 : launch_one(sz_row_kernel<float, false, 256, 3>, grid, block, smem, S, a, st);
}

cudaError_t launch_sz_apply_c(int dtype, const SzDev &src, const SzSectorDev &tgt, int nop, const SzOp *ops,
                              const void *in, void *out, int num_sms, cudaStream_t st)
{
    if (nop < 1 || nop > 2) return cudaErrorInvalidValue;
    const SzOp o0 = ops[0], o1 = nop > 1 ? ops[1] : SzOp();
    const int block = sz_block(tgt.maxlen);
    int grid = num_sms * (2048 / block);
    if (grid > tgt.nrows) grid = tgt.nrows;
    if (grid < 1) grid = 1;
    if (dtype == EDK_F64)
        sz_apply_c_kernel<double><<<grid, block, 0, st>>>(src, tgt, nop, o0, o1, static_cast<const double *>(in),
                                                          static_cast<double *>(out));
    else
        sz_apply_c_kernel<float><<<grid, block, 0, st>>>(src, tgt, nop, o0, o1, static_cast<const float *>(in),
                                                         static_cast<float *>(out));
    return cudaGetLastError();
}

}  // namespace edk
