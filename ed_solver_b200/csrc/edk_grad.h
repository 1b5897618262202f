// Internal declarations of the adjoint kernels (edk_grad_kernels.cu) used by
// the gradient drivers (edk_grad.cpp).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace edk {

constexpr int kMaxGradParams = 64;

enum ParamKind : int {
    kParamNumber = 0,   // n_p on the spins of spin_mask
    kParamHop = 1,      // c+_p c_q + c+_q c_p through the maps
    kParamDouble = 2,   // n_p,up n_p,dn
    kParamPair = 3,     // (n_p,up + n_p,dn)(n_q,up + n_q,dn)
};

struct ParamDev {
    int kind;
    int spin_mask;                  // bit 0 up, bit 1 down
    uint32_t bp, bq;                // orbital bit masks
    const int32_t *mapu, *mapd;     // hop maps per spin (null when that spin is not included)
};

cudaError_t launch_lincomb(int64_t n, double *out, bool accumulate, const double *x0, double c0,
                           const double *x1, double c1, const double *x2, double c2, const double *x3,
                           double c3, int grid, cudaStream_t st);
cudaError_t launch_dots(int64_t n, const double *x0, const double *y0, const double *x1, const double *y1,
                        const double *x2, const double *y2, const double *x3, const double *y3, double *partials,
                        unsigned *counter, double *out, int grid, cudaStream_t st);
cudaError_t launch_fill_periodic(int64_t n, const double *tab, int64_t offset, double *out, int grid, cudaStream_t st);
cudaError_t launch_bilinear(int64_t dup, int64_t ddn, const double *a, const double *b, const uint32_t *st_up,
                            const uint32_t *st_dn, int np, const ParamDev *P, double *partials, unsigned *counter,
                            double *out, int grid, bool accumulate, cudaStream_t st);

// Device scalars of one chain, indexed by the Lanczos step k >= 1: a_k, b_k
// (b_1 = |phi|), their cotangents ab_k and bb_k; dot: scratch of the passes
// (0-2: products for the next reverse step, 3: of this one, 4: E0's cotangent).
struct GradScalars {
    double *al, *be, *ab, *bb, *dot;
};
struct CgScalars {
    double rr, rr0, t[2], pap, rn;
    int it, done;
};
struct GradPass {
    int64_t n;
    int grid;
    double *partials;
    unsigned *counter;
    cudaStream_t st;
};
cudaError_t pass_fwd_w(const GradPass &p, double *w, const double *vkm1, const double *vk, int k, const GradScalars &S);
cudaError_t pass_fwd_r(const GradPass &p, double *r, const double *w, const double *vk, int k, const GradScalars &S);
cudaError_t pass_fwd_scale(const GradPass &p, double *r, int k, const GradScalars &S);
cudaError_t pass_replay(const GradPass &p, double *v, const double *vkm1, const double *vk, int k, const GradScalars &S);
cudaError_t pass_rev_wbar(const GradPass &p, bool have_r, const double *vbn, double *vbc, double *wbar,
                          const double *vkp, const double *vkk, const double *vkm, int k, const GradScalars &S);
cudaError_t pass_rev_next(const GradPass &p, double *vbn, double *vbc, const double *hw, const double *wbar,
                          const double *vkk, const double *vkm, int k, const GradScalars &S);
cudaError_t pass_rev_start(const GradPass &p, double *phibar, const double *vb1, const double *v1, const GradScalars &S);
// one iteration after ap = H d: four passes
cudaError_t pass_cg(const GradPass &p, double *x, double *r, double *d, double *ap, const double *psi, double e0,
                    double tol2, int maxit, CgScalars *S);
cudaError_t pass_cf(int K, double e0, double ph, int nw, const double *wn, const double *gbar, const GradScalars &S,
                    double2 *cp, double2 *u, double2 *gs, double *G, double *parts, cudaStream_t st);

}  // namespace edk
