// pass_f64.cu -- the FP64 passes that touch points, real kernels: P2M
// (class_fmm.py:57-71) and the L2P + P2P at the sources (class_fmm.py:73-111),
// the "plain" form's leaf pass; the mixed form takes its P2M from here, its
// K0 far field, and with near_fp64 its leaf pass.
#include <algorithm>
#include <mutex>

#include "pair_f64.cuh"
#include "passes.cuh"

namespace kifmm {

__device__ double2 g_logtab[LOGTAB_N];
const double2 *log_table(int device) {
    static std::mutex mu;
    static const double2 *tab[64] = {};
    KIFMM_REQUIRE(device >= 0 && device < 64, KIFMM_ERR_ARG, "device index out of range");
    std::lock_guard<std::mutex> lock(mu);
    if (!tab[device]) {
        double2 t[LOGTAB_N];
        const long double c0 = (long double)LOG_H2 * LOG_H2 * LOG_H2 / 192.0L;
        for (int i = 0; i < LOGTAB_N; i++) {
            t[i].x = (double)(1.0L / (1.0L + ((long double)i + 0.5L) / LOGTAB_N));
            t[i].y = (double)(-logl((long double)t[i].x) - c0);
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
// den[leaf_list index][Q].  Reads 4 Q^2 bytes per leaf-block from L2 and
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
    pdl_trigger();
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
    for (int i = tid; i < 32 * Kp; i += DEN_THREADS) {
        const int n = i / Kp, c = i - n * Kp;
        xS[n * ldx + c] = n < nt && c < Q ? A.udown[(size_t)D.list[w0 + n] * Q + c] : 0.0;
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

// L2P + P2P of the leaves, one warp per item: an item is up to ts (<= 32)
// targets of one leaf.  The warp's targets form ng groups of TB targets; sp =
// 32 / ng lanes share a group, lane (gi, j) taking sources j, j + sp, ..., so
// that a leaf of 28 points (the mean on the 1M mixture) keeps 28 lanes busy and
// each source read from shared memory serves TB pairs.  The leaf's sources
// (its own points, then its colleagues') are staged in chunks; the L2P is the
// same loop over the Q equivalent points of the leaf's local expansion, in
// box-relative coordinates.  Bound by issue: 12 FP64 instructions (two slots
// each) and about 9 others per Laplace pair.  Warps draw items from a ticket
// (the leaves differ in work by more than 10x); each warp draws one ticket past
// the end, so atomicInc's wrap leaves the counter at zero for the next launch.
constexpr int L64_CHUNK = 64;  // sources staged per pass, two per lane
struct Leaf64Warp {
    double2 xy[L64_CHUNK];
    double z[L64_CHUNK];
    double red[8][32];
    int rng[18];
    int pad[2];
};
static_assert(sizeof(Leaf64Warp) % 16 == 0, "Leaf64Warp alignment");

// Sums of the lane's TB targets over sources u, u + sp, ... below n.  CHECKED
// tests each pair and gives those that the fast value is not for to the math
// library (coincident pairs are left out with skip_equal); without it the
// return value tells afterwards whether there was such a pair (one instruction
// a pair instead of five), and the caller runs the sources again, checked.
template <int KIND, int NT, int TB, bool CHECKED>
__device__ __forceinline__ bool pair_loop(const Leaf64Warp &W, const double2 *tl, int &u, int sp, int n,
                                          const double *tx, const double *ty, double k, double k2, unsigned hi_end,
                                          bool skip_equal, double *acc) {
    unsigned worst = 0;      // largest rank (K0)
    int least = 0x7fffffff;  // smallest high word (Laplace: r^2 is finite)
#pragma unroll 1
    for (; u < n; u += sp) {
        const double2 s = W.xy[u];
        const double z = W.z[u];
        bool all = true;
#pragma unroll
        for (int a = 0; a < TB; a++) {
            const double dx = tx[a] - s.x, dy = ty[a] - s.y;
            const double r2 = fma(dx, dx, dy * dy);
            const double t = KIND == KIFMM_KERNEL_LAPLACE ? r2 : r2 * k2;
            const double v = pair_value<KIND, NT>(t, tl);
            if (CHECKED) {
                const bool ok = pair_ordinary(t, hi_end);
                if (ok) acc[a] = fma(v, z, acc[a]);
                all = all && ok;
            } else {
                acc[a] = fma(v, z, acc[a]);
                if (KIND == KIFMM_KERNEL_LAPLACE) least = min(least, __double2hiint(t));
                else worst = max(worst, pair_rank(t));
            }
        }
        if (CHECKED && !all) {
#pragma unroll
            for (int a = 0; a < TB; a++) {
                const double dx = tx[a] - s.x, dy = ty[a] - s.y;
                const double r2 = fma(dx, dx, dy * dy);
                if (!pair_ordinary(KIND == KIFMM_KERNEL_LAPLACE ? r2 : r2 * k2, hi_end) &&
                    !(skip_equal && dx == 0.0 && dy == 0.0))
                    acc[a] = fma(pair_value_any<KIND>(r2, k), z, acc[a]);
            }
        }
    }
    return KIND == KIFMM_KERNEL_LAPLACE ? least < 0x00100000 : worst >= hi_end - 0x00100000u;
}
// ... where many pairs are past the series (leaves several 1/k wide): either
// value per pair
template <int KIND, int NT, int TB>
__device__ __forceinline__ void pair_loop_beyond(const Leaf64Warp &W, const double2 *tl, int u, int sp, int n,
                                                 const double *tx, const double *ty, double k, double k2,
                                                 unsigned hi_end, bool skip_equal, double *acc) {
#pragma unroll 1
    for (; u < n; u += sp) {
        const double2 s = W.xy[u];
        const double z = W.z[u];
#pragma unroll
        for (int a = 0; a < TB; a++) {
            const double dx = tx[a] - s.x, dy = ty[a] - s.y;
            const double r2 = fma(dx, dx, dy * dy), t = r2 * k2;
            if (pair_ordinary(t, hi_end)) acc[a] = fma(pair_value<KIND, NT>(t, tl), z, acc[a]);
            else if (!(skip_equal && dx == 0.0 && dy == 0.0)) acc[a] = fma(pair_value_any<KIND>(r2, k), z, acc[a]);
        }
    }
}
// the staged sources u, u + sp, ... below n, the first n_own of them checked
// (the leaf's own points, where the target meets itself)
template <int KIND, int NT, int TB, bool BEYOND>
__device__ __forceinline__ void pair_chunk(Leaf64Warp &W, const double2 *tl, int u, int sp, int n_own, int n,
                                           const double *tx, const double *ty, double k, double k2, unsigned hi_end,
                                           bool skip_equal, double *acc) {
    if (BEYOND) {
        pair_loop_beyond<KIND, NT, TB>(W, tl, u, sp, n, tx, ty, k, k2, hi_end, skip_equal, acc);
        return;
    }
    pair_loop<KIND, NT, TB, true>(W, tl, u, sp, n_own, tx, ty, k, k2, hi_end, skip_equal, acc);
    const int lane = threadIdx.x & 31, u0 = u;
#pragma unroll
    for (int a = 0; a < TB; a++) W.red[a][lane] = acc[a];
    if (pair_loop<KIND, NT, TB, false>(W, tl, u, sp, n, tx, ty, k, k2, hi_end, skip_equal, acc)) {
#pragma unroll
        for (int a = 0; a < TB; a++) acc[a] = W.red[a][lane];
        u = u0;
        pair_loop<KIND, NT, TB, true>(W, tl, u, sp, n, tx, ty, k, k2, hi_end, skip_equal, acc);
    }
}
// the near sources of the leaf (n_own of its own first), then the equivalent
// points of its local expansion
template <int KIND, int NT, int TB, bool BEYOND, bool FAR>
__device__ __forceinline__ double leaf_item(const PassArgs &A, Leaf64Warp &W, const double2 *tl, int t0, int nt,
                                            int n_own, int ns, int l, double cx, double cy, const double *den,
                                            unsigned hi_end, bool check_self, double k2, int lane) {
    const int ng = (nt + TB - 1) / TB, sp = 32 / ng, j = lane / ng, gi = lane - j * ng;
    double tx[TB], ty[TB], acc[TB];
#pragma unroll
    for (int a = 0; a < TB; a++) {
        const int i = gi + a * ng < nt ? gi + a * ng : gi;  // unused slots repeat the first
        tx[a] = A.xs[t0 + i];
        ty[a] = A.ys[t0 + i];
        acc[a] = 0.0;
    }
    const int u0 = j < sp ? j : 1 << 20;  // lanes past the last group idle
    for (int c0 = 0; !FAR && c0 < ns; c0 += L64_CHUNK) {
        const int cn = min(L64_CHUNK, ns - c0);
        __syncwarp();
#pragma unroll
        for (int h = 0; h < L64_CHUNK; h += 32) {
            const int q = h + lane;
            if (q < cn) {
                const int p = range_point(W.rng, c0 + q);
                W.xy[q] = make_double2(A.xs[p], A.ys[p]);
                W.z[q] = A.taus[p];
            }
        }
        __syncwarp();
        pair_chunk<KIND, NT, TB, BEYOND>(W, tl, u0, sp, min(n_own - c0, cn), cn, tx, ty, A.k, k2, hi_end, check_self,
                                         acc);
    }
    if (l >= 2) {
        const double *lg = A.ops + (size_t)l * A.stride + A.off_large;
        __syncwarp();
        for (int q = lane; q < A.Q; q += 32) {
            W.xy[q] = make_double2(lg[q], lg[A.Q + q]);
            W.z[q] = den[q];
        }
        __syncwarp();
#pragma unroll
        for (int a = 0; a < TB; a++) {
            tx[a] -= cx;
            ty[a] -= cy;
        }
        pair_chunk<KIND, NT, TB, BEYOND>(W, tl, u0, sp, 0, A.Q, tx, ty, A.k, k2, hi_end, false, acc);
    }
    __syncwarp();
#pragma unroll
    for (int a = 0; a < TB; a++) W.red[a][lane] = acc[a];
    __syncwarp();
    double v = 0.0;
    if (lane < nt) {
        const int slot = lane / ng, grp = lane - slot * ng;
        for (int m = 0; m < sp; m++) v += W.red[slot][grp + m * ng];
    }
    return v * pair_scale<KIND>();
}
template <int KIND, bool FAR, int NT, bool BEYOND = false>
__device__ __forceinline__ double leaf_item_tb(const PassArgs &A, Leaf64Warp &W, const double2 *tl, int t0, int nt,
                                               int n_own, int ns, int l, double cx, double cy, const double *den,
                                               unsigned hi_end, bool check_self, double k2, int lane) {
    // the number of targets per lane that leaves the fewest lanes idle: pair
    // slots per source TB / (32 / ceil(nt / TB)), compared by cross products
    const int s2 = 32 / ((nt + 1) >> 1), s3 = 32 / ((nt + 2) / 3), s4 = 32 / ((nt + 3) >> 2);
    if (s4 * 3 >= s3 * 4 && s4 * 2 >= s2 * 4)
        return leaf_item<KIND, NT, 4, BEYOND, FAR>(A, W, tl, t0, nt, n_own, ns, l, cx, cy, den, hi_end, check_self, k2,
                                                   lane);
    if (s3 * 2 >= s2 * 3)
        return leaf_item<KIND, NT, 3, BEYOND, FAR>(A, W, tl, t0, nt, n_own, ns, l, cx, cy, den, hi_end, check_self, k2,
                                                   lane);
    return leaf_item<KIND, NT, 2, BEYOND, FAR>(A, W, tl, t0, nt, n_own, ns, l, cx, cy, den, hi_end, check_self, k2, lane);
}

// 16 warps per SM at 128 registers measured 1-5% faster than 24 at 80 (the K0
// series spill there), and 64-source chunks the same as 96 or 128
constexpr int L64_MAX_WARPS = 8, L64_BLOCKS_PER_SM = 2;
// FAR: the L2P alone, added to the near field that pots already holds
template <int KIND, bool FAR>
__global__ void __launch_bounds__(32 * L64_MAX_WARPS, L64_BLOCKS_PER_SM)
    k_leaf_eval_d(PassArgs A, const double2 *__restrict__ logtab, const double *__restrict__ den, unsigned nitems,
                  int ntile, int ts, int check_self, unsigned *__restrict__ ticket) {
    extern __shared__ __align__(16) unsigned char sm_l64[];
    double2 *tab = (double2 *)sm_l64;
    Leaf64Warp &W = ((Leaf64Warp *)(tab + LOGTAB_N * LOGTAB_COPIES))[threadIdx.x >> 5];
    stage_log_table(tab, logtab);
    __syncthreads();
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const double2 *tl = tab + (lane & (LOGTAB_COPIES - 1));
    const double k2 = A.k * A.k;
    const unsigned last = nitems + gridDim.x * (blockDim.x >> 5) - 1;
    for (;;) {
        unsigned it = 0;
        if (lane == 0) it = atomicInc(ticket, last);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= nitems) return;
        const unsigned w = it / ntile;
        const int rv = A.leaf_rec[(size_t)w * LEAF_REC_WORDS + lane];
        const int l = __shfl_sync(0xffffffffu, rv, LR_LEVEL), b = __shfl_sync(0xffffffffu, rv, LR_BOT),
                  e = __shfl_sync(0xffffffffu, rv, LR_TOP), ns = __shfl_sync(0xffffffffu, rv, LR_NSRC);
        const uint64_t key = (uint64_t)(uint32_t)__shfl_sync(0xffffffffu, rv, LR_KEY_LO) |
                             ((uint64_t)(uint32_t)__shfl_sync(0xffffffffu, rv, LR_KEY_HI) << 32);
        __syncwarp();
        if (lane >= LR_RNG && lane < LR_RNG + 18) W.rng[lane - LR_RNG] = rv;
        __syncwarp();
        const double wl = ldexp(A.W, -l);
        const double cx = A.root + ((double)compact2(key >> 1) + 0.5) * wl;
        const double cy = A.root + ((double)compact2(key) + 0.5) * wl;
        // r^2 <= 8 w^2 over the 3x3 cells; to the equivalent points r < 2 w
        const double tmax = KIND == KIFMM_KERNEL_LAPLACE ? 0.0 : (FAR ? 4.0 : 8.0) * wl * wl * k2;
        if (FAR && l < 2) continue;
        const double *dn = den + (size_t)w * A.Q;
        for (int t0 = b + (int)(it - w * ntile) * ts; t0 < e; t0 += ntile * ts) {
            const int nt = min(ts, e - t0);
            double v;
            const int own = e - b;
            if (KIND == KIFMM_KERNEL_LAPLACE)
                v = leaf_item_tb<KIND, FAR, 1>(A, W, tl, t0, nt, own, ns, l, cx, cy, dn, LOG_HI_END, check_self, k2, lane);
            else if (tmax < 0.0625)
                v = leaf_item_tb<KIND, FAR, SERIES_NARROW>(A, W, tl, t0, nt, own, ns, l, cx, cy, dn, SERIES_NARROW_HI,
                                                      check_self, k2, lane);
            else if (tmax < 1.0)
                v = leaf_item_tb<KIND, FAR, SERIES_MID>(A, W, tl, t0, nt, own, ns, l, cx, cy, dn, SERIES_MID_HI, check_self,
                                                   k2, lane);
            else if (tmax < 4.0)
                v = leaf_item_tb<KIND, FAR, SERIES_WIDE>(A, W, tl, t0, nt, own, ns, l, cx, cy, dn, SERIES_WIDE_HI,
                                                    check_self, k2, lane);
            else
                v = leaf_item_tb<KIND, FAR, SERIES_WIDE, true>(A, W, tl, t0, nt, own, ns, l, cx, cy, dn, SERIES_WIDE_HI,
                                                          check_self, k2, lane);
            if (lane < nt) A.pots[t0 + lane] = FAR ? A.pots[t0 + lane] + v : v;
        }
    }
}

// the equivalent densities of the leaf list
static const double *launch_leaf_density(kifmm_plan *P, const PassArgs &A) {
    DenArgs D{};
    D.A = A;
    D.list = P->leaf_list.p;
    P->leaf_den.alloc((size_t)P->n_leaf_list * P->Q);
    D.den = P->leaf_den.p;
    D.lmin = 2;
    D.lmax = P->L - 1;
    int64_t tiles = 0;
    for (int l = 0; l <= MAX_LEVELS; l++) {
        D.loff[l] = P->leaf_loff[l];
        D.toff[l] = tiles;
        if (l >= D.lmin && l <= D.lmax && l < MAX_LEVELS) tiles += (P->leaf_loff[l + 1] - P->leaf_loff[l] + 31) / 32;
    }
    if (tiles) {
        const size_t smem = den_smem(P->Q);
        ensure_dyn_smem(k_leaf_density, smem);
        launch_pdl(k_leaf_density, dim3((unsigned)tiles), dim3(DEN_THREADS), smem, P->stream, D);
    }
    return D.den;
}

// Warps per block and blocks for `items` items of one warp each.  A block's
// table is shared by its warps; fewer items than resident warps: smaller
// blocks, down to two warps, spread them over the SMs.
static void pair_grid(const kifmm_plan *P, int64_t items, int *warps, unsigned *grid, size_t *smem) {
    const int64_t resident = (int64_t)P->num_sms * L64_BLOCKS_PER_SM * L64_MAX_WARPS;
    int w = L64_MAX_WARPS;
    while (w > 2 && items < (int64_t)P->num_sms * w * 2) w >>= 1;
    *warps = w;
    *grid = (unsigned)std::min<int64_t>((items + w - 1) / w, resident / w);
    *smem = LOGTAB_N * LOGTAB_COPIES * sizeof(double2) + (size_t)w * sizeof(Leaf64Warp);
}

template <int KIND, bool FAR>
static void launch_leaf_eval(kifmm_plan *P, const PassArgs &A, int check_self) {
    const int64_t nl = P->n_leaf_list;
    const double *den = launch_leaf_density(P, A);
    // Items: whole 32-target tiles once they fill the GPU's resident warps (16
    // per SM); smaller tiles for fewer leaves, down to 8 targets, where a
    // warp's run over its sources is the kernel's length.
    const int64_t resident = (int64_t)P->num_sms * L64_BLOCKS_PER_SM * L64_MAX_WARPS;
    int ts = 32;
    while (ts > 8 && nl * ((P->ppl + ts - 1) / ts) < resident) ts >>= 1;
    const int ntile = (int)std::min<int64_t>((P->ppl + ts - 1) / ts, 64);
    const int64_t items = nl * ntile;
    KIFMM_REQUIRE(items + resident < (1ll << 32), KIFMM_ERR_ARG, "leaf pass: too many leaves");
    int warps;
    unsigned grid;
    size_t smem;
    pair_grid(P, items, &warps, &grid, &smem);
    ensure_dyn_smem(k_leaf_eval_d<KIND, FAR>, smem);
    launch_pdl(k_leaf_eval_d<KIND, FAR>, dim3(grid), dim3(32 * warps), smem, P->stream, A, log_table(P->device), den,
               (unsigned)items, ntile, ts, check_self, (unsigned *)(P->scal.p + KIFMM_SCAL_TICKET));
}
void launch_leaf_eval_d(kifmm_plan *P, const PassArgs &A, int check_self) {
    if (P->kern.kind == KIFMM_KERNEL_LAPLACE) launch_leaf_eval<KIFMM_KERNEL_LAPLACE, false>(P, A, check_self);
    else launch_leaf_eval<KIFMM_KERNEL_MOD_HELMHOLTZ, false>(P, A, check_self);
}
// the K0 far field, added to the near field in pots
void launch_leaf_far_d(kifmm_plan *P, const PassArgs &A) {
    launch_leaf_eval<KIFMM_KERNEL_MOD_HELMHOLTZ, true>(P, A, 0);
}

// P2M, one warp per node: the Q check points are the targets of the pair loop,
// TB of them per lane on eight lanes, and four groups of lanes share the
// node's sources (all 32 lanes busy for every Nequiv that is a multiple of 8;
// one check point per lane left 24 of 64 lane slots idle at Nequiv 40).
// Bound by issue like the leaf pass.
template <int KIND, int NT, int TB, bool BEYOND = false>
__device__ __forceinline__ void p2m_node(const PassArgs &A, Leaf64Warp &W, const double2 *tl, int g, int b, int e,
                                         const double *lg, double cx, double cy, unsigned hi_end, double k2, int lane) {
    const int gi = lane & 7, j = lane >> 3, Q = A.Q;
    double tx[TB], ty[TB], acc[TB];
#pragma unroll
    for (int a = 0; a < TB; a++) {
        const int q = gi + 8 * a < Q ? gi + 8 * a : 0;  // unused slots repeat the first
        tx[a] = lg[q] + cx;
        ty[a] = lg[Q + q] + cy;
        acc[a] = 0.0;
    }
    for (int s0 = b; s0 < e; s0 += L64_CHUNK) {
        const int cn = min(L64_CHUNK, e - s0);
        __syncwarp();
#pragma unroll
        for (int h = 0; h < L64_CHUNK; h += 32) {
            const int q = h + lane;
            if (q < cn) {
                W.xy[q] = make_double2(A.xs[s0 + q], A.ys[s0 + q]);
                W.z[q] = A.taus[s0 + q];
            }
        }
        __syncwarp();
        pair_chunk<KIND, NT, TB, BEYOND>(W, tl, j, 4, 0, cn, tx, ty, A.k, k2, hi_end, false, acc);
    }
#pragma unroll
    for (int a = 0; a < TB; a++) {
        double v = acc[a];
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if (j == 0 && gi + 8 * a < Q) A.uup[(size_t)g * Q + gi + 8 * a] = v * pair_scale<KIND>();
    }
}
template <int KIND, int TB>
__global__ void __launch_bounds__(32 * L64_MAX_WARPS, L64_BLOCKS_PER_SM)
    k_p2m_d(PassArgs A, const double2 *__restrict__ logtab, const int32_t *__restrict__ list, int64_t nlist) {
    extern __shared__ __align__(16) unsigned char sm_p2m[];
    double2 *tab = (double2 *)sm_p2m;
    Leaf64Warp &W = ((Leaf64Warp *)(tab + LOGTAB_N * LOGTAB_COPIES))[threadIdx.x >> 5];
    stage_log_table(tab, logtab);
    __syncthreads();
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const double2 *tl = tab + (lane & (LOGTAB_COPIES - 1));
    const double k2 = A.k * A.k;
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t w = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); w < nlist; w += nw) {
        const int g = list[w], l = A.nlev[g], b = A.nbot[g], e = A.ntop[g];
        double cx, cy;
        node_center(A, g, l, cx, cy);
        const double *lg = A.ops + (size_t)l * A.stride + A.off_large;
        if (KIND == KIFMM_KERNEL_LAPLACE) {
            p2m_node<KIND, 1, TB>(A, W, tl, g, b, e, lg, cx, cy, LOG_HI_END, k2, lane);
            continue;
        }
        const double wl = ldexp(A.W, -l), tmax = 4.0 * wl * wl * k2;  // r < 2 w to the check circle
        if (tmax < 0.0625) p2m_node<KIND, SERIES_NARROW, TB>(A, W, tl, g, b, e, lg, cx, cy, SERIES_NARROW_HI, k2, lane);
        else if (tmax < 1.0) p2m_node<KIND, SERIES_MID, TB>(A, W, tl, g, b, e, lg, cx, cy, SERIES_MID_HI, k2, lane);
        else if (tmax < 4.0) p2m_node<KIND, SERIES_WIDE, TB>(A, W, tl, g, b, e, lg, cx, cy, SERIES_WIDE_HI, k2, lane);
        else p2m_node<KIND, SERIES_WIDE, TB, true>(A, W, tl, g, b, e, lg, cx, cy, SERIES_WIDE_HI, k2, lane);
    }
}
template <int KIND, int TB>
static void launch_p2m_tb(kifmm_plan *P, const PassArgs &A) {
    int warps;
    unsigned grid;
    size_t smem;
    pair_grid(P, P->n_p2m_list, &warps, &grid, &smem);
    ensure_dyn_smem(k_p2m_d<KIND, TB>, smem);
    launch_pdl(k_p2m_d<KIND, TB>, dim3(grid), dim3(32 * warps), smem, P->stream, A, log_table(P->device),
               (const int32_t *)P->p2m_list.p, P->n_p2m_list);
}
template <int KIND>
static void launch_p2m_kind(kifmm_plan *P, const PassArgs &A) {
    const int tb = (P->Q + 7) / 8;  // Nequiv <= 64
    if (tb <= 2) launch_p2m_tb<KIND, 2>(P, A);
    else if (tb == 3) launch_p2m_tb<KIND, 3>(P, A);
    else if (tb == 4) launch_p2m_tb<KIND, 4>(P, A);
    else if (tb == 5) launch_p2m_tb<KIND, 5>(P, A);
    else if (tb == 6) launch_p2m_tb<KIND, 6>(P, A);
    else launch_p2m_tb<KIND, 8>(P, A);
}
void launch_p2m_d(kifmm_plan *P, const PassArgs &A) {
    if (P->kern.kind == KIFMM_KERNEL_LAPLACE) launch_p2m_kind<KIFMM_KERNEL_LAPLACE>(P, A);
    else launch_p2m_kind<KIFMM_KERNEL_MOD_HELMHOLTZ>(P, A);
}

}  // namespace kifmm
