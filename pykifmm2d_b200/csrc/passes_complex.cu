// passes_complex.cu -- the point passes of the complex form, FP64.
//
// The reference's complex mode (FMM(..., iscomplex=True), class_fmm.py:174)
// keeps every workspace in complex128 and runs the same passes.  Here a node's
// state is the real image of its complex check potential: Q = 2 Qc doubles,
// [Re u (Qc), Im u (Qc)], and every translation operator is the real image of
// the complex one (operators.cu), so M2M, M2L and L2L are the real FP64
// kernels unchanged.  P2M, L2P and P2P are in pass_f64.cuh and targets.cu; here
// are the densities' permutation and KF / KA / KAS
// (class_fmm.py:115-145) for a complex kernel.
// Densities and potentials are double2 (re, im) in HBM.
#include "passes.cuh"

namespace kifmm {

__device__ __forceinline__ void cacc(double2 &acc, double2 a, double2 b) {
    acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
    acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
}

__global__ void k_gather_tau_c(const double2 *__restrict__ tau, const int32_t *__restrict__ perm, int64_t n,
                               double2 *__restrict__ taus, unsigned long long *__restrict__ flags, int nflag) {
    pdl_wait();
    pdl_trigger();
    if (blockIdx.x == 0 && threadIdx.x < nflag) flags[threadIdx.x] = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        taus[i] = tau[perm[i]];
}

// ------------------------------------------------ kernel-function utilities
// KAS restricted to targets (class_fmm.py:134-143), complex: one block per target
__global__ void k_direct_c(int kind, double k, const double *__restrict__ x, const double *__restrict__ y,
                           const double2 *__restrict__ tau, int64_t n, const int64_t *__restrict__ tg,
                           double2 *__restrict__ out) {
    __shared__ double2 red[32];
    const int64_t j = tg[blockIdx.x];
    if (j < 0 || j >= n) {  // caller index out of range: report NaN, touch nothing
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
        if (threadIdx.x == 0) out[blockIdx.x] = make_double2(nan, nan);
        return;
    }
    const double px = x[j], py = y[j];
    double2 acc = make_double2(0.0, 0.0);
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        if (i == j) continue;
        const double dx = px - x[i], dy = py - y[i];
        cacc(acc, green_z(kind, k, dx * dx + dy * dy), tau[i]);
    }
    for (int o = 16; o; o >>= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        double2 v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : make_double2(0.0, 0.0);
        for (int o = 16; o; o >>= 1) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        }
        if (threadIdx.x == 0) out[blockIdx.x] = v;
    }
}

__global__ void k_kmatrix_c(int kind, double k, const double *sx, const double *sy, int64_t ns, const double *tx,
                            const double *ty, int64_t nt, double2 *out) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ns * nt; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = e / ns, i = e % ns;
        const double dx = tx[j] - sx[i], dy = ty[j] - sy[i];
        out[e] = green_z(kind, k, dx * dx + dy * dy);
    }
}

__global__ void k_kapply_c(int kind, double k, const double *sx, const double *sy, int64_t ns, const double *tx,
                           const double *ty, int64_t nt, const double2 *tau, double2 *out) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nt; j += (int64_t)gridDim.x * blockDim.x) {
        double2 acc = make_double2(0.0, 0.0);
        for (int64_t i = 0; i < ns; i++) {
            const double dx = tx[j] - sx[i], dy = ty[j] - sy[i];
            cacc(acc, green_z(kind, k, dx * dx + dy * dy), tau[i]);
        }
        out[j] = acc;
    }
}

// ------------------------------------------------------------ host side
void launch_gather_tau_c(kifmm_plan *P) {
    launch_pdl(k_gather_tau_c, dim3(grid_for(P->N, 256, P->num_sms * 8)), dim3(256), 0, P->stream,
               (const double2 *)P->tau_src, (const int32_t *)P->perm.p, P->N, (double2 *)P->taus.p,
               P->scal.p + KIFMM_SCAL_PASS_ERR, KIFMM_SCAL_WORDS - KIFMM_SCAL_PASS_ERR);
}

void direct_sum_device_c(const kifmm_kernel &kn, const double *x, const double *y, const double *tau, int64_t n,
                         const int64_t *tg, int64_t nt, double *out, cudaStream_t s) {
    if (nt <= 0) return;
    KIFMM_REQUIRE(nt < (1ll << 31), KIFMM_ERR_ARG, "direct_sum: too many targets");
    k_direct_c<<<(unsigned)nt, 256, 0, s>>>(kn.kind, kn.k, x, y, (const double2 *)tau, n, tg, (double2 *)out);
    KIFMM_LAUNCHED();
}

void kernel_matrix_device_c(const kifmm_kernel &kn, const double *sx, const double *sy, int64_t ns, const double *tx,
                            const double *ty, int64_t nt, double *out, cudaStream_t s) {
    if (ns * nt <= 0) return;
    k_kmatrix_c<<<grid_for(ns * nt, 256, 8192), 256, 0, s>>>(kn.kind, kn.k, sx, sy, ns, tx, ty, nt, (double2 *)out);
    KIFMM_LAUNCHED();
}

void kernel_apply_device_c(const kifmm_kernel &kn, const double *sx, const double *sy, int64_t ns, const double *tx,
                           const double *ty, int64_t nt, const double *tau, double *out, cudaStream_t s) {
    if (nt <= 0) return;
    k_kapply_c<<<grid_for(nt, 128, 8192), 128, 0, s>>>(kn.kind, kn.k, sx, sy, ns, tx, ty, nt, (const double2 *)tau,
                                                        (double2 *)out);
    KIFMM_LAUNCHED();
}

}  // namespace kifmm
