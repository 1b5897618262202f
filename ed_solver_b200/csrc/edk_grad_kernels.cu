// Device kernels of the adjoint (parameter gradients): FP64 vector updates,
// multi-dot products, and the bilinear forms <a| dH/dtheta_q |b> of every
// requested parameter in one pass over a sector vector.
//
// The Hamiltonian is linear in its parameters, so dH/dtheta_q is a fixed
// operator: a one-body number operator n_p (Ec(c,c), Eb(k,k)), a symmetric
// one-body hop c+_p c_q + c+_q c_p (Ec(i,j), Eb(i,j), Vbc(k,c); the terms of
// HAIM_offdiag_arrays.f90:419-524), n_up n_dn of one impurity site (U(c,c),
// HAIMupdo.f90:784-796) or n_i n_j of two (U(i,j), HAIMupdo.f90:798-829).
// Hops act on one spin species through a per-parameter map of that spin's
// basis: (rank of the target + 1) * Jordan-Wigner sign, or 0.
#include "edk_device.cuh"
#include "edk_grad.h"

namespace edk {

namespace {

__global__ void lincomb_kernel(int64_t n, double *out, int accumulate, const double *x0, double c0,
                               const double *x1, double c1, const double *x2, double c2, const double *x3,
                               double c3)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double v = accumulate ? out[i] : 0.0;
        if (x0) v += c0 * x0[i];
        if (x1) v += c1 * x1[i];
        if (x2) v += c2 * x2[i];
        if (x3) v += c3 * x3[i];
        out[i] = v;
    }
}

__global__ void dots_kernel(int64_t n, const double *x0, const double *y0, const double *x1, const double *y1,
                            const double *x2, const double *y2, const double *x3, const double *y3,
                            double *partials, unsigned *counter, double *out)
{
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (x0) s[0] += x0[i] * y0[i];
        if (x1) s[1] += x1[i] * y1[i];
        if (x2) s[2] += x2[i] * y2[i];
        if (x3) s[3] += x3[i] * y3[i];
    }
    grid_sum<4>(s, partials, counter, out);
}

// One block per row; the rows of a and b are staged in shared memory when
// STAGE.  The warps share the parameters out between them (several warps per
// parameter where there are more warps), so a short row costs one or two
// parameters' latency instead of all of them; each warp accumulates its columns
// in a fixed order into its own slot, blocks write per-parameter partials and
// the last block sums them, a warp per parameter, in a fixed order.
template <bool STAGE>
__global__ void __launch_bounds__(512, 1) bilinear_kernel(int dup, int ddn, const double *a, const double *b,
                                                          const uint32_t *__restrict__ st_up,
                                                          const uint32_t *__restrict__ st_dn, int np,
                                                          const ParamDev *__restrict__ P, double *partials,
                                                          unsigned *counter, double *out, int accumulate)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ ParamDev sp[kMaxGradParams];
    __shared__ double s_part[kMaxGradParams][16];
    __shared__ bool last;
    chain_next();
    const int nwarp = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int share = nwarp > np ? nwarp / np : 1;              // warps per parameter
    const int sub = warp % share, first = warp / share, step = nwarp / share;
    const int c0 = lane + 32 * sub, cs = 32 * share;
    for (int q = threadIdx.x; q < np; q += blockDim.x) sp[q] = P[q];
    for (int t = threadIdx.x; t < np * 16; t += blockDim.x) s_part[t / 16][t % 16] = 0.0;
    chain_wait();
    double *as = reinterpret_cast<double *>(smem_raw);
    double *bs = as + dup;
    for (int row = blockIdx.x; row < ddn; row += gridDim.x) {
        __syncthreads();
        const double *arow = a + (size_t)row * dup, *brow = b + (size_t)row * dup;
        if (STAGE) {
            for (int c = threadIdx.x; c < dup; c += blockDim.x) {
                as[c] = arow[c];
                bs[c] = brow[c];
            }
            __syncthreads();
        }
        const double *ar = STAGE ? as : arow;
        const double *br = STAGE ? bs : brow;
        const uint32_t sdn = st_dn[row];
        for (int q = first; q < np && first < step; q += step) {
            const ParamDev p = sp[q];
            double t = 0.0;
            if (p.kind == kParamNumber) {
                const int fdn = ((p.spin_mask & 2) && (sdn & p.bp)) ? 1 : 0;
                for (int c = c0; c < dup; c += cs) {
                    const int f = (((p.spin_mask & 1) && (st_up[c] & p.bp)) ? 1 : 0) + fdn;
                    if (f) t += (double)f * ar[c] * br[c];
                }
            } else if (p.kind == kParamDouble) {
                if (sdn & p.bp)
                    for (int c = c0; c < dup; c += cs)
                        if (st_up[c] & p.bp) t += ar[c] * br[c];
            } else if (p.kind == kParamPair) {
                const int di = (sdn & p.bp) ? 1 : 0, dj = (sdn & p.bq) ? 1 : 0;
                for (int c = c0; c < dup; c += cs) {
                    const uint32_t su = st_up[c];
                    const int f = (((su & p.bp) ? 1 : 0) + di) * (((su & p.bq) ? 1 : 0) + dj);
                    if (f) t += (double)f * ar[c] * br[c];
                }
            } else {   // kParamHop
                if (p.mapu)
                    for (int c = c0; c < dup; c += cs) {
                        const int32_t m = p.mapu[c];
                        if (m) t += (m > 0 ? ar[c] : -ar[c]) * br[(m > 0 ? m : -m) - 1];
                    }
                if (p.mapd) {
                    const int32_t m = p.mapd[row];
                    if (m) {
                        const double *bo = b + (size_t)((m > 0 ? m : -m) - 1) * dup;
                        double u = 0.0;
                        for (int c = c0; c < dup; c += cs) u += ar[c] * bo[c];
                        t += m > 0 ? u : -u;
                    }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
            if (lane == 0) s_part[q][sub] += t;
        }
    }
    __syncthreads();
    for (int q = threadIdx.x; q < np; q += blockDim.x) {
        double v = 0.0;
        for (int w = 0; w < share; ++w) v += s_part[q][w];
        partials[(size_t)blockIdx.x * np + q] = v;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int q = warp; q < np; q += nwarp) {
        double v = 0.0;
        for (unsigned g = lane; g < gridDim.x; g += 32) v += __ldcg(&partials[(size_t)g * np + q]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) out[q] = accumulate ? out[q] + v : v;
    }
    if (threadIdx.x == 0) *counter = 0u;
}

// ---------------------------------------------------------------------------
// The vector passes of the forward recurrence, its replay, the reverse sweep
// and the conjugate gradients.  Their coefficients are read from device memory,
// where the dot products of the passes before them left them, so a whole chain
// is queued without a host round trip; passes that touch the same vectors are
// one kernel with their dot products.  Small sectors are bound by launches (a
// 63,504-state sector: 10 passes a Lanczos step instead of 22 launches, copies and
// six waits for the device), large ones by the vectors read and written.
// ---------------------------------------------------------------------------
#define EDK_EACH(i) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)

// w = H v_k - b_k v_{k-1} in place over H v_k; a_k = <w, v_k>
__global__ void fwd_w_kernel(int64_t n, double *w, const double *vkm1, const double *vk, int k, GradScalars S,
                             double *partials, unsigned *counter)
{
    chain_next();
    chain_wait();
    double s[1] = {0.0};
    const double b = -S.be[k];
    EDK_EACH(i) {
        const double v = w[i] + b * vkm1[i];
        w[i] = v;
        s[0] += v * vk[i];
    }
    grid_sum<1>(s, partials, counter, S.al + k);
}

// r = w - a_k v_k; b_{k+1} = |r|
__global__ void fwd_r_kernel(int64_t n, double *r, const double *w, const double *vk, int k, GradScalars S,
                             double *partials, unsigned *counter)
{
    chain_next();
    chain_wait();
    double s[1] = {0.0};
    const double a = -S.al[k];
    EDK_EACH(i) {
        const double v = w[i] + a * vk[i];
        r[i] = v;
        s[0] += v * v;
    }
    if (grid_sum<1>(s, partials, counter, S.be + k + 1)) S.be[k + 1] = sqrt(fmax(S.be[k + 1], 0.0));
}

// v_{k+1} = r / b_{k+1} (zero after a breakdown: the host cuts the chain there)
__global__ void fwd_scale_kernel(int64_t n, double *r, int k, GradScalars S)
{
    chain_next();
    chain_wait();
    const double b = S.be[k + 1], c = b > 1e-25 ? 1.0 / b : 0.0;
    EDK_EACH(i) r[i] = c * r[i];
}

// v_{k+1} = (H v_k - b_k v_{k-1} - a_k v_k) / b_{k+1}, in place over H v_k
__global__ void replay_kernel(int64_t n, double *v, const double *vkm1, const double *vk, int k, GradScalars S)
{
    chain_next();
    chain_wait();
    const double b = -S.be[k], a = -S.al[k], c = 1.0 / S.be[k + 1];
    EDK_EACH(i) {
        double t = v[i] + b * vkm1[i];
        t += a * vk[i];
        v[i] = c * t;
    }
}

// Reverse step k before H: with d1 = <vbar_{k+1}, v_{k+1}>, e1 = <vbar_{k+1}, v_k> and
// f1 = <v_{k+1}, v_k> in S.dot (from rev_next of step k + 1),
//   rbar = vbar_{k+1} / b_{k+1} + (bb_{k+1} - d1 / b_{k+1}) v_{k+1},
//   ab = abar_k - <rbar, v_k>,  wbar = rbar + ab v_k,
//   vbar_k += -a_k rbar + ab (b_{k+1} v_{k+1} + a_k v_k),  bb_k -= <wbar, v_{k-1}>.
__global__ void rev_wbar_kernel(int64_t n, int have_r, const double *vbn, double *vbc, double *wbar, const double *vkp,
                                const double *vkk, const double *vkm, int k, GradScalars S, double *partials,
                                unsigned *counter)
{
    chain_next();
    chain_wait();
    const double ak = S.al[k], bk1 = S.be[k + 1];
    double cr = 0.0, ib = 0.0, ab = S.ab[k];
    if (have_r) {
        ib = 1.0 / bk1;
        cr = S.bb[k + 1] - S.dot[0] / bk1;
        ab -= S.dot[1] * ib + cr * S.dot[2];
    }
    double s[1] = {0.0};
    EDK_EACH(i) {
        const double p = vkp[i], q = vkk[i];
        const double r = have_r ? ib * vbn[i] + cr * p : 0.0;
        const double w = r + ab * q;
        double v = vbc[i] - ak * r;
        v += (ab * bk1) * p;
        v += (ab * ak) * q;
        wbar[i] = w;
        vbc[i] = v;
        s[0] += w * vkm[i];
    }
    if (grid_sum<1>(s, partials, counter, S.dot + 3) && k >= 2) S.bb[k] -= S.dot[3];
}

// Reverse step k after H: vbar_k += H wbar (final), vbar_{k-1} starts at -b_k wbar in
// the buffer of vbar_{k+1}; the dot products of step k - 1.
__global__ void rev_next_kernel(int64_t n, double *vbn, double *vbc, const double *hw, const double *wbar,
                                const double *vkk, const double *vkm, int k, GradScalars S, double *partials,
                                unsigned *counter)
{
    chain_next();
    chain_wait();
    const double b = -S.be[k];
    double s[3] = {0.0, 0.0, 0.0};
    EDK_EACH(i) {
        const double v = vbc[i] + hw[i], p = vkk[i], q = vkm[i];
        vbc[i] = v;
        vbn[i] = b * wbar[i];
        s[0] += v * p;
        s[1] += v * q;
        s[2] += p * q;
    }
    grid_sum<3>(s, partials, counter, S.dot);
}

// phibar = (vbar_1 - <vbar_1, v_1> v_1) / b_1 + bb_1 v_1
__global__ void rev_start_kernel(int64_t n, double *phibar, const double *vb1, const double *v1, GradScalars S)
{
    chain_next();
    chain_wait();
    const double b1 = S.be[1], c = -S.dot[0] / b1 + S.bb[1], ib = 1.0 / b1;
    EDK_EACH(i) phibar[i] = ib * vb1[i] + c * v1[i];
}

// Conjugate gradients on (H - E0) x = r in the complement of psi.  S: rr, rr0,
// <ap, psi>, <p, psi>, pap, rn; done stops the passes that are already queued.
__global__ void cg_dots_kernel(int64_t n, const double *ap, const double *p, const double *psi, CgScalars *S,
                               double *partials, unsigned *counter)
{
    chain_next();
    chain_wait();
    if (S->done) return;
    double s[2] = {0.0, 0.0};
    EDK_EACH(i) {
        s[0] += ap[i] * psi[i];
        s[1] += p[i] * psi[i];
    }
    grid_sum<2>(s, partials, counter, S->t);
}
__global__ void cg_project_kernel(int64_t n, double *ap, const double *p, const double *psi, double e0, CgScalars *S,
                                  double *partials, unsigned *counter)
{
    chain_next();
    chain_wait();
    if (S->done) return;
    const double c = -(S->t[0] - e0 * S->t[1]);
    double s[1] = {0.0};
    EDK_EACH(i) {
        double v = ap[i] - e0 * p[i];
        v += c * psi[i];
        ap[i] = v;
        s[0] += p[i] * v;
    }
    if (grid_sum<1>(s, partials, counter, &S->pap) && !(S->pap > 0.0)) S->done = 1;
}
__global__ void cg_step_kernel(int64_t n, double *x, double *r, const double *p, const double *ap, CgScalars *S,
                               double *partials, unsigned *counter)
{
    chain_next();
    chain_wait();
    if (S->done) return;
    const double al = S->rr / S->pap;
    double s[1] = {0.0};
    EDK_EACH(i) {
        x[i] += al * p[i];
        const double v = r[i] - al * ap[i];
        r[i] = v;
        s[0] += v * v;
    }
    grid_sum<1>(s, partials, counter, &S->rn);
}
__global__ void cg_direction_kernel(int64_t n, double *p, const double *r, double tol2, int maxit, CgScalars *S,
                                    double *partials, unsigned *counter)
{
    chain_next();
    chain_wait();
    if (S->done) return;
    const double c = S->rn / S->rr;
    EDK_EACH(i) p[i] = r[i] + c * p[i];
    double s[1] = {0.0};
    if (grid_sum<1>(s, partials, counter, S->t)) {       // every block has read rr
        S->rr = S->rn;
        S->it += 1;
        if (!(S->rr > tol2 * S->rr0) || S->it >= maxit) S->done = 1;
    }
}

// ---- continued fraction and its vector-Jacobian product -------------------
struct Cd {
    double re, im;
};
__device__ __forceinline__ Cd operator+(Cd a, Cd b) { return Cd{a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ Cd operator-(Cd a, Cd b) { return Cd{a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ Cd operator*(Cd a, Cd b) { return Cd{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ Cd operator*(double s, Cd a) { return Cd{s * a.re, s * a.im}; }
__device__ __forceinline__ Cd inverse(Cd b)       // Smith's scaling
{
    if (fabs(b.re) >= fabs(b.im)) {
        const double r = b.im / b.re, d = 1.0 / (b.re + b.im * r);
        return Cd{d, -r * d};
    }
    const double r = b.re / b.im, d = 1.0 / (b.im + b.re * r);
    return Cd{r * d, -d};
}

// One frequency per thread: u of (z - ph (T - e0)) u = e1 by the Thomas
// recurrence, u[k * nw + w]; G, and the per-frequency parts of the cotangents.
__global__ void cf_solve_kernel(int K, double e0, double ph, int nw, const double *wn, const double *gbar, GradScalars S,
                                double2 *cp, double2 *u, double2 *gs, double *G, double *parts)
{
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= nw) return;
    const double b1 = S.be[1], s = b1 * b1;
    const Cd z{0.0, wn[w]};
    Cd den = inverse(Cd{-ph * (S.al[1] - e0), z.im});
    Cd c = K > 1 ? (-ph * S.be[2]) * den : Cd{0.0, 0.0}, d = den;
    cp[w] = make_double2(c.re, c.im);
    u[w] = make_double2(d.re, d.im);
    for (int k = 1; k < K; ++k) {
        const double off = -ph * S.be[k + 1];
        den = inverse(Cd{-ph * (S.al[k + 1] - e0), z.im} - off * c);
        c = k + 1 < K ? (-ph * S.be[k + 2]) * den : Cd{0.0, 0.0};
        d = (-off) * (d * den);
        cp[(size_t)k * nw + w] = make_double2(c.re, c.im);
        u[(size_t)k * nw + w] = make_double2(d.re, d.im);
    }
    Cd v = d, uu = v * v;
    for (int k = K - 2; k >= 0; --k) {
        const double2 dk = u[(size_t)k * nw + w], ck = cp[(size_t)k * nw + w];
        v = Cd{dk.x, dk.y} - Cd{ck.x, ck.y} * v;
        u[(size_t)k * nw + w] = make_double2(v.re, v.im);
        uu = uu + v * v;
    }
    G[2 * w] = s * v.re;
    G[2 * w + 1] = s * v.im;
    const Cd gc{gbar[2 * w], -gbar[2 * w + 1]};
    gs[w] = make_double2(s * gc.re, s * gc.im);
    parts[w] = (gc * ((-ph * s) * uu)).re;                  // E0
    parts[nw + w] = (gc * ((2.0 * b1) * v)).re;             // b_1
}

// Block k < K: abar_{k+1} and bb_{k+2}; block K: E0's cotangent and bb_1; added to
// those of the frequencies before.
__global__ void cf_reduce_kernel(int K, double ph, int nw, const double2 *u, const double2 *gs, const double *parts,
                                 GradScalars S)
{
    __shared__ double red[2][32];
    const int k = blockIdx.x;
    double s[2] = {0.0, 0.0};
    for (int w = threadIdx.x; w < nw; w += blockDim.x) {
        if (k == K) {
            s[0] += parts[w];
            s[1] += parts[nw + w];
            continue;
        }
        const double2 g = gs[w], p = u[(size_t)k * nw + w];
        const Cd gu = (ph * Cd{g.x, g.y}) * Cd{p.x, p.y};
        s[0] += (gu * Cd{p.x, p.y}).re;
        if (k + 1 < K) {
            const double2 q = u[(size_t)(k + 1) * nw + w];
            s[1] += 2.0 * (gu * Cd{q.x, q.y}).re;
        }
    }
    block_sum<2>(s, red);
    if (threadIdx.x == 0) {
        if (k == K) {
            S.dot[4] += s[0];
            S.bb[1] += s[1];
        } else {
            S.ab[k + 1] += s[0];
            if (k + 1 < K) S.bb[k + 2] += s[1];
        }
    }
}

// out[i] = tab[(i + offset) % 10000 + 1] (the reference's periodic start
// vector, rcvector_class.f90:43-60, shifted by `offset` for a block column)
__global__ void fill_periodic_kernel(int64_t n, const double *tab, int64_t offset, double *out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = tab[(i + offset) % 10000 + 1];
}

}  // namespace

cudaError_t launch_fill_periodic(int64_t n, const double *tab, int64_t offset, double *out, int grid, cudaStream_t st)
{
    fill_periodic_kernel<<<grid, 256, 0, st>>>(n, tab, offset, out);
    return cudaGetLastError();
}

cudaError_t launch_lincomb(int64_t n, double *out, bool accumulate, const double *x0, double c0,
                           const double *x1, double c1, const double *x2, double c2, const double *x3,
                           double c3, int grid, cudaStream_t st)
{
    lincomb_kernel<<<grid, 256, 0, st>>>(n, out, accumulate ? 1 : 0, x0, c0, x1, c1, x2, c2, x3, c3);
    return cudaGetLastError();
}

cudaError_t launch_dots(int64_t n, const double *x0, const double *y0, const double *x1, const double *y1,
                        const double *x2, const double *y2, const double *x3, const double *y3, double *partials,
                        unsigned *counter, double *out, int grid, cudaStream_t st)
{
    dots_kernel<<<grid, 256, 0, st>>>(n, x0, y0, x1, y1, x2, y2, x3, y3, partials, counter, out);
    return cudaGetLastError();
}

cudaError_t launch_bilinear(int64_t dup, int64_t ddn, const double *a, const double *b, const uint32_t *st_up,
                            const uint32_t *st_dn, int np, const ParamDev *P, double *partials, unsigned *counter,
                            double *out, int grid, bool accumulate, cudaStream_t st)
{
    if (np < 1 || np > kMaxGradParams) return cudaErrorInvalidValue;
    if (grid > ddn) grid = (int)ddn;
    if (grid < 1) grid = 1;
    const size_t smem = 2 * (size_t)dup * sizeof(double);
    // the kernel's static shared memory is about 11 KB of the 227 KB a block may use
    if (smem <= (size_t)(227 - 12) * 1024) {
        int per_sm = 0;
        cudaError_t e = kernel_fit(reinterpret_cast<const void *>(bilinear_kernel<true>), 512, smem, &per_sm);
        if (e != cudaSuccess) return e;
        return launch_chained(bilinear_kernel<true>, grid, 512, smem, st, (int)dup, (int)ddn, a, b, st_up, st_dn, np, P,
                              partials, counter, out, accumulate ? 1 : 0);
    }
    return launch_chained(bilinear_kernel<false>, grid, 512, 0, st, (int)dup, (int)ddn, a, b, st_up, st_dn, np, P,
                          partials, counter, out, accumulate ? 1 : 0);
}

// ---- passes of the adjoint (GradPass: sector length, grid, reduction scratch, stream) ----
static int pass_grid(const GradPass &p)
{
    const int64_t b = (p.n + 255) / 256;
    return (int)(b < p.grid ? (b > 0 ? b : 1) : p.grid);
}
cudaError_t pass_fwd_w(const GradPass &p, double *w, const double *vkm1, const double *vk, int k, const GradScalars &S)
{
    return launch_chained(fwd_w_kernel, pass_grid(p), 256, 0, p.st, p.n, w, vkm1, vk, k, S, p.partials, p.counter);
}
cudaError_t pass_fwd_r(const GradPass &p, double *r, const double *w, const double *vk, int k, const GradScalars &S)
{
    return launch_chained(fwd_r_kernel, pass_grid(p), 256, 0, p.st, p.n, r, w, vk, k, S, p.partials, p.counter);
}
cudaError_t pass_fwd_scale(const GradPass &p, double *r, int k, const GradScalars &S)
{
    return launch_chained(fwd_scale_kernel, pass_grid(p), 256, 0, p.st, p.n, r, k, S);
}
cudaError_t pass_replay(const GradPass &p, double *v, const double *vkm1, const double *vk, int k, const GradScalars &S)
{
    return launch_chained(replay_kernel, pass_grid(p), 256, 0, p.st, p.n, v, vkm1, vk, k, S);
}
cudaError_t pass_rev_wbar(const GradPass &p, bool have_r, const double *vbn, double *vbc, double *wbar,
                          const double *vkp, const double *vkk, const double *vkm, int k, const GradScalars &S)
{
    return launch_chained(rev_wbar_kernel, pass_grid(p), 256, 0, p.st, p.n, have_r ? 1 : 0, vbn, vbc, wbar, vkp, vkk, vkm, k, S, p.partials,
                                                    p.counter);
}
cudaError_t pass_rev_next(const GradPass &p, double *vbn, double *vbc, const double *hw, const double *wbar,
                          const double *vkk, const double *vkm, int k, const GradScalars &S)
{
    return launch_chained(rev_next_kernel, pass_grid(p), 256, 0, p.st, p.n, vbn, vbc, hw, wbar, vkk, vkm, k, S, p.partials, p.counter);
}
cudaError_t pass_rev_start(const GradPass &p, double *phibar, const double *vb1, const double *v1, const GradScalars &S)
{
    return launch_chained(rev_start_kernel, pass_grid(p), 256, 0, p.st, p.n, phibar, vb1, v1, S);
}
cudaError_t pass_cg(const GradPass &p, double *x, double *r, double *d, double *ap, const double *psi, double e0,
                    double tol2, int maxit, CgScalars *S)
{
    const int g = pass_grid(p);
    cudaError_t e = cudaSuccess;
    if (e == cudaSuccess) e = launch_chained(cg_dots_kernel, g, 256, 0, p.st, p.n, ap, d, psi, S, p.partials, p.counter);
    if (e == cudaSuccess) e = launch_chained(cg_project_kernel, g, 256, 0, p.st, p.n, ap, d, psi, e0, S, p.partials, p.counter);
    if (e == cudaSuccess) e = launch_chained(cg_step_kernel, g, 256, 0, p.st, p.n, x, r, d, ap, S, p.partials, p.counter);
    if (e == cudaSuccess) e = launch_chained(cg_direction_kernel, g, 256, 0, p.st, p.n, d, r, tol2, maxit, S, p.partials, p.counter);
    return e;
}
cudaError_t pass_cf(int K, double e0, double ph, int nw, const double *wn, const double *gbar, const GradScalars &S,
                    double2 *cp, double2 *u, double2 *gs, double *G, double *parts, cudaStream_t st)
{
    cf_solve_kernel<<<(nw + 31) / 32, 32, 0, st>>>(K, e0, ph, nw, wn, gbar, S, cp, u, gs, G, parts);
    cf_reduce_kernel<<<K + 1, 128, 0, st>>>(K, ph, nw, u, gs, parts, S);
    return cudaGetLastError();
}

}  // namespace edk
