// pass_f64.cu -- the FP64 passes that touch points: P2M (class_fmm.py:57-71)
// and the L2P + P2P at the sources (class_fmm.py:73-111), for real densities
// (the "plain" form; the mixed form takes its P2M from here, its K0 far field,
// and with near_fp64 its leaf pass) and for complex ones.
#include <cstring>
#include <mutex>

#include "pass_f64.cuh"

namespace kifmm {

__device__ double2 g_logtab[LOGTAB_N];
const double2 *log_table(int device) {
    static std::mutex mu;
    static const double2 *tab[64] = {};
    KIFMM_REQUIRE(device >= 0 && device < 64, KIFMM_ERR_ARG, "device index out of range");
    std::lock_guard<std::mutex> lock(mu);
    if (!tab[device]) {
        double2 t[LOGTAB_N];
        for (int i = 0; i < LOGTAB_N; i++) {  // subintervals [a, b) of m
            const auto value = [](uint64_t hi) {
                double d;
                hi <<= 32;
                memcpy(&d, &hi, sizeof(d));
                return d;
            };
            const double a = value(LOG_M_HI + i * LOG_STEP_HI), b = value(LOG_M_HI + (i + 1) * LOG_STEP_HI);
            const bool one = a <= 1.0 && 1.0 < b;
            t[i].x = one ? 1.0 : (double)(1.0L / (((long double)a + b) * 0.5L));
            t[i].y = one ? 0.0 : (double)-logl((long double)t[i].x);
        }
        void *p = nullptr;
        KIFMM_CUDA(cudaMemcpyToSymbol(g_logtab, t, sizeof(t)));
        KIFMM_CUDA(cudaGetSymbolAddress(&p, g_logtab));
        tab[device] = (const double2 *)p;
    }
    return tab[device];
}

// Equivalent densities of the leaves' local expansions, phi = Inv_l u_down,
// on the FP64 tensor path: one block per 32 consecutive leaves of one level
// (leaf_list is level-major), warp w all Q rows for leaves 8w .. 8w + 7.  The
// level's inverse is read once per block instead of once per leaf.
// den[leaf_list index][Q]; without a list the level's nodes are taken and den is
// indexed by node.  Reads 4 Q^2 bytes per leaf-block from L2 and
// 16 Q bytes per leaf: latency-bound (a few microseconds at 65k leaves).
struct DenArgs {
    PassArgs A;
    const int32_t *list;
    double *den;
    int lmin, lmax;
    int64_t loff[MAX_LEVELS + 1];  // leaf_list range of each level
    int64_t toff[MAX_LEVELS + 1];  // first block of each level
};
constexpr int DEN_THREADS = 128, DEN_MT = 8;  // Q <= 8 DEN_MT
static size_t den_smem(int Q) {
    const int Kp = (Q + 3) & ~3, Mp = (Q + 7) & ~7;
    return ((size_t)Kp * pad4mod16(Mp) + 32 * (size_t)pad4mod16(Kp)) * sizeof(double);
}
__global__ void __launch_bounds__(DEN_THREADS) k_leaf_density(DenArgs D) {
    extern __shared__ __align__(16) double sm_den[];
    const PassArgs &A = D.A;
    const int Q = A.Q, Kp = (Q + 3) & ~3, Mp = (Q + 7) & ~7, ldm = pad4mod16(Mp), ldx = pad4mod16(Kp);
    double *mS = sm_den;                  // [Kp][ldm]: Inv[r][c] at c * ldm + r
    double *xS = mS + (size_t)Kp * ldm;   // [32][ldx]
    const int tid = threadIdx.x;
    const int64_t b = blockIdx.x;
    int l = D.lmin;
    while (l < D.lmax && D.toff[l + 1] <= b) l++;
    const int64_t w0 = D.loff[l] + (b - D.toff[l]) * 32;
    const int nt = (int)min((int64_t)32, D.loff[l + 1] - w0);
    const double *inv = A.ops + (size_t)l * A.stride + A.off_inv;
    for (int i = tid; i < Kp * Mp; i += DEN_THREADS) {
        const int r = i / Kp, c = i - r * Kp;
        mS[c * ldm + r] = r < Q && c < Q ? inv[r * Q + c] : 0.0;
    }
    pdl_wait();  // u_down comes from the L2L chain
    // only now: the leaf pass's blocks fill every SM, and waiting there through
    // the L2L chain they would keep other streams' kernels out
    pdl_trigger();
    for (int i = tid; i < 32 * Kp; i += DEN_THREADS) {
        const int n = i / Kp, c = i - n * Kp;
        xS[n * ldx + c] = n < nt && c < Q ? A.udown[(size_t)(D.list ? D.list[w0 + n] : w0 + n) * Q + c] : 0.0;
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, n0 = warp * 8;
    if (n0 >= nt) return;
    double acc[DEN_MT][2];
#pragma unroll
    for (int i = 0; i < DEN_MT; i++) acc[i][0] = acc[i][1] = 0.0;
    const double *xb = xS + (size_t)(n0 + g) * ldx + t, *ab = mS + (size_t)t * ldm + g;
    for (int k0 = 0; k0 < Kp; k0 += 4) {
        const double bv = xb[k0];
#pragma unroll
        for (int i = 0; i < DEN_MT; i++)
            if (8 * i < Mp) dmma_8x8x4(acc[i][0], acc[i][1], ab[(size_t)k0 * ldm + 8 * i], bv);
    }
#pragma unroll
    for (int i = 0; i < DEN_MT; i++) {
        const int r = 8 * i + g;
        if (r >= Q) continue;
#pragma unroll
        for (int j = 0; j < 2; j++)
            if (n0 + 2 * t + j < nt) D.den[(size_t)(w0 + n0 + 2 * t + j) * Q + r] = acc[i][j];
    }
}

static const double *launch_density(kifmm_plan *P, DenArgs &D) {
    D.lmin = 2;
    D.lmax = P->L - 1;
    int64_t tiles = 0;
    for (int l = 0; l <= MAX_LEVELS; l++) {
        D.toff[l] = tiles;
        if (l >= D.lmin && l <= D.lmax && l < MAX_LEVELS) tiles += (D.loff[l + 1] - D.loff[l] + 31) / 32;
    }
    if (tiles) {
        const size_t smem = den_smem(P->Q);
        ensure_dyn_smem(k_leaf_density, smem);
        launch_pdl(k_leaf_density, dim3((unsigned)tiles), dim3(DEN_THREADS), smem, P->stream, D);
    }
    return D.den;
}
// the equivalent densities of the leaf list
const double *launch_leaf_density(kifmm_plan *P, const PassArgs &A) {
    DenArgs D{};
    D.A = A;
    D.list = P->leaf_list.p;
    P->leaf_den.alloc((size_t)P->n_leaf_list * P->Q);
    D.den = P->leaf_den.p;
    for (int l = 0; l <= MAX_LEVELS; l++) D.loff[l] = P->leaf_loff[l];
    return launch_density(P, D);
}
// ... of every node (targets may lie in leaves without points)
const double *launch_node_density(kifmm_plan *P, const PassArgs &A) {
    DenArgs D{};
    D.A = A;
    P->node_den.alloc((size_t)P->n_nodes * P->Q);
    D.den = P->node_den.p;
    for (int l = 0; l <= MAX_LEVELS; l++) D.loff[l] = l < P->L ? P->lt.off[l] : P->n_nodes;
    return launch_density(P, D);
}

void launch_leaf_eval_d(kifmm_plan *P, const PassArgs &A, int check_self) {
    if (P->cplx) launch_leaf_eval_dc(P, A, check_self);
    else if (P->kern.kind == KIFMM_KERNEL_LAPLACE)
        launch_leaf_eval<KIFMM_KERNEL_LAPLACE, false, false>(P, A, check_self);
    else launch_leaf_eval<KIFMM_KERNEL_MOD_HELMHOLTZ, false, false>(P, A, check_self);
}
// the K0 far field, added to the near field in pots (there after near_done)
void launch_leaf_far_d(kifmm_plan *P, const PassArgs &A, cudaEvent_t near_done) {
    launch_leaf_eval<KIFMM_KERNEL_MOD_HELMHOLTZ, false, true>(P, A, 0, near_done);
}
void launch_p2m_d(kifmm_plan *P, const PassArgs &A) {
    if (P->cplx) launch_p2m_dc(P, A);
    else if (P->kern.kind == KIFMM_KERNEL_LAPLACE) launch_p2m_kind<KIFMM_KERNEL_LAPLACE, false>(P, A);
    else launch_p2m_kind<KIFMM_KERNEL_MOD_HELMHOLTZ, false>(P, A);
}

}  // namespace kifmm
