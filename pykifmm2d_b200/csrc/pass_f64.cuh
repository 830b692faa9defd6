// pass_f64.cuh -- the pair-loop kernels of pass_f64.cu (real densities) and
// pass_f64_complex.cu (complex ones), with their launchers.
#pragma once
#include <algorithm>
#include <type_traits>

#include "pair_f64.cuh"
#include "passes.cuh"

namespace kifmm {

// equivalent densities of every node (pass_f64.cu)
const double *launch_node_density(kifmm_plan *P, const PassArgs &A);

// L2P + P2P of the leaves, one warp per item: an item is up to ts (<= 32)
// targets of one leaf.  The warp's targets form ng groups of TB targets; sp =
// 32 / ng lanes share a group, lane (gi, j) taking sources j, j + sp, ..., so
// that a leaf of 28 points (the mean on the 1M mixture) keeps 28 lanes busy and
// each source read from shared memory serves TB pairs.  The leaf's sources
// (its own points, then its colleagues') are staged in chunks; the L2P is the
// same loop over the Q equivalent points of the leaf's local expansion, in
// box-relative coordinates.  Bound by issue: 12 FP64 instructions (two slots
// each) and about 10 others per Laplace pair.  Warps draw items from a ticket
// (the leaves differ in work by more than 10x); each warp draws one ticket past
// the end, so atomicInc's wrap leaves the counter at zero for the next launch.
constexpr int L64_CHUNK = 64;  // sources staged per pass, two per lane
// One warp's staged sources: positions, charges z (complex: a double2), and
// for the Helmholtz kernel pz = (pi Im z, -pi Re z), so that G z = re z + a pz.
template <int KIND, bool CPLX>
struct PairWarp {
    using Z = std::conditional_t<CPLX, double2, double>;
    static constexpr bool H0 = KIND == KIFMM_KERNEL_HELMHOLTZ;
    static constexpr int NC = CPLX ? 2 : 1;  // components of a sum
    double2 xy[L64_CHUNK];
    Z z[L64_CHUNK];
    double2 pz[H0 ? L64_CHUNK : 1];
    double red[NC][8][32];
    int rng[18];
    int pad[2];
    __device__ void stage(int q, double x, double y, Z v) {
        xy[q] = make_double2(x, y);
        z[q] = v;
        if constexpr (H0) pz[q] = make_double2(M_PI * v.y, -M_PI * v.x);
    }
};

// sum of a lane's target, and its update by value v of a pair with source u
template <int KIND, bool CPLX>
struct PairSum {
    double c[CPLX ? 2 : 1];
    using W = PairWarp<KIND, CPLX>;
    __device__ __forceinline__ void add(const PairValue &v, const typename W::Z &z, const double2 &pz) {
        if constexpr (!CPLX) {
            c[0] = fma(v.re, z, c[0]);
        } else if constexpr (!W::H0) {
            c[0] = fma(v.re, z.x, c[0]);
            c[1] = fma(v.re, z.y, c[1]);
        } else {
            c[0] = fma(v.re, z.x, fma(v.a, pz.x, c[0]));
            c[1] = fma(v.re, z.y, fma(v.a, pz.y, c[1]));
        }
    }
};

// Whether a target's r^2 to a source may be infinite or not a number.  The
// unchecked Laplace loop, which looks for small r^2 only, would take such a pair
// for an ordinary one.  Sources are checked when the tree is built; separate
// targets are anything (targets.cu).
__device__ __forceinline__ bool out_of_reach(double x, double y) {
    constexpr double REACH = 0x1p500;  // r^2 stays below 2^1002
    return !(fabs(x) < REACH && fabs(y) < REACH);
}

// Sums of the lane's TB targets over sources u, u + sp, ... below n.  CHECKED
// tests each pair and gives those that the fast value is not for to the math
// library (coincident pairs are left out with skip_equal); without it the
// return value tells afterwards whether there was such a pair (one instruction
// a pair instead of five), and the caller runs the sources again, checked.
template <int KIND, bool CPLX, int NT, int TB, bool CHECKED>
__device__ __forceinline__ bool pair_loop(const PairWarp<KIND, CPLX> &W, const double2 *tl, int &u, int sp, int n,
                                          const double *tx, const double *ty, double k, double k2, unsigned hi_end,
                                          bool skip_equal, PairSum<KIND, CPLX> *acc) {
    unsigned worst = 0;      // largest rank (K0, H0)
    int least = 0x7fffffff;  // smallest high word (Laplace: r^2 is finite, see out_of_reach)
#pragma unroll 1
    for (; u < n; u += sp) {
        const double2 s = W.xy[u];
        const auto z = W.z[u];
        const double2 pz = W.pz[PairWarp<KIND, CPLX>::H0 ? u : 0];
        bool all = true;
#pragma unroll
        for (int a = 0; a < TB; a++) {
            const double dx = tx[a] - s.x, dy = ty[a] - s.y;
            const double r2 = fma(dx, dx, dy * dy);
            const double t = KIND == KIFMM_KERNEL_LAPLACE ? r2 : r2 * k2;
            const PairValue v = pair_value<KIND, NT>(t, tl);
            if (CHECKED) {
                const bool ok = pair_ordinary(t, hi_end);
                if (ok) acc[a].add(v, z, pz);
                all = all && ok;
            } else {
                acc[a].add(v, z, pz);
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
                    acc[a].add(pair_value_any<KIND>(r2, k), z, pz);
            }
        }
    }
    return KIND == KIFMM_KERNEL_LAPLACE ? least < 0x00100000 : worst >= hi_end - 0x00100000u;
}
// ... where many pairs are past the series (leaves several 1/k wide): both
// values for all of the lane's targets where any of them needs it, so that the
// targets' chains overlap (a call per pair was bound by its latency: 2.5 times
// its instructions)
template <int KIND, bool CPLX, int NT, int TB>
__device__ __forceinline__ void pair_loop_beyond(const PairWarp<KIND, CPLX> &W, const double2 *tl, int u, int sp,
                                                 int n, const double *tx, const double *ty, double k, double k2,
                                                 unsigned hi_end, bool skip_equal, PairSum<KIND, CPLX> *acc) {
#pragma unroll 1
    for (; u < n; u += sp) {
        const double2 s = W.xy[u];
        const auto z = W.z[u];
        const double2 pz = W.pz[PairWarp<KIND, CPLX>::H0 ? u : 0];
        double t[TB];
        bool some_near = false, some_far = false, some_other = false;
#pragma unroll
        for (int a = 0; a < TB; a++) {
            const double dx = tx[a] - s.x, dy = ty[a] - s.y;
            t[a] = fma(dx, dx, dy * dy) * k2;
            const bool ok = pair_ordinary(t[a], hi_end), far = pair_beyond<KIND>(t[a]);
            some_near = some_near || ok;
            some_far = some_far || far;
            some_other = some_other || !(ok || far);
        }
        if (some_near) {
#pragma unroll
            for (int a = 0; a < TB; a++) {
                const PairValue v = pair_value<KIND, NT>(t[a], tl);
                if (pair_ordinary(t[a], hi_end)) acc[a].add(v, z, pz);
            }
        }
        if (some_far) {
#pragma unroll
            for (int a = 0; a < TB; a++) {
                const PairValue v = pair_value_beyond<KIND>(t[a], tl);
                if (pair_beyond<KIND>(t[a])) acc[a].add(v, z, pz);
            }
        }
        if (some_other) {
#pragma unroll
            for (int a = 0; a < TB; a++) {
                const double dx = tx[a] - s.x, dy = ty[a] - s.y;
                if (!pair_ordinary(t[a], hi_end) && !pair_beyond<KIND>(t[a]) && !(skip_equal && dx == 0.0 && dy == 0.0))
                    acc[a].add(pair_value_any<KIND>(fma(dx, dx, dy * dy), k), z, pz);
            }
        }
    }
}
// the staged sources u, u + sp, ... below n, the first n_own of them checked
// (the leaf's own points, where the target meets itself)
template <int KIND, bool CPLX, int NT, int TB, bool BEYOND>
__device__ __forceinline__ void pair_chunk(PairWarp<KIND, CPLX> &W, const double2 *tl, int u, int sp, int n_own, int n,
                                           const double *tx, const double *ty, double k, double k2, unsigned hi_end,
                                           bool skip_equal, PairSum<KIND, CPLX> *acc) {
    constexpr int NC = PairWarp<KIND, CPLX>::NC;
    if (BEYOND) {
        pair_loop_beyond<KIND, CPLX, NT, TB>(W, tl, u, sp, n, tx, ty, k, k2, hi_end, skip_equal, acc);
        return;
    }
    pair_loop<KIND, CPLX, NT, TB, true>(W, tl, u, sp, n_own, tx, ty, k, k2, hi_end, skip_equal, acc);
    const int lane = threadIdx.x & 31, u0 = u;
#pragma unroll
    for (int a = 0; a < TB; a++)
#pragma unroll
        for (int c = 0; c < NC; c++) W.red[c][a][lane] = acc[a].c[c];
    if (pair_loop<KIND, CPLX, NT, TB, false>(W, tl, u, sp, n, tx, ty, k, k2, hi_end, skip_equal, acc)) {
#pragma unroll
        for (int a = 0; a < TB; a++)
#pragma unroll
            for (int c = 0; c < NC; c++) acc[a].c[c] = W.red[c][a][lane];
        u = u0;
        pair_loop<KIND, CPLX, NT, TB, true>(W, tl, u, sp, n, tx, ty, k, k2, hi_end, skip_equal, acc);
    }
}
template <bool CPLX>
__device__ __forceinline__ auto load_value(const double *v, int i) {
    if constexpr (CPLX) return ((const double2 *)v)[i];
    else return v[i];
}

// Up to 32 targets of one leaf
struct LeafItem {
    const double *tx, *ty;  // target coordinates, at idx[t0 .. t0 + nt) or, without idx, at t0 ..
    const int32_t *idx;
    int t0, nt, n_own, ns, l, lane;
    int lanes;              // targets that set the lanes' stride over the sources (>= nt): a sum's order depends on it
    double cx, cy;
    const double *den;
    bool check_self;
    double k2;
};
// the near sources of the leaf (n_own of its own first), then the equivalent
// points of its local expansion; the sums are returned to lanes < nt
template <int KIND, bool CPLX, bool FAR, int NT, bool BEYOND, int TB>
__device__ __forceinline__ PairSum<KIND, CPLX> leaf_item(const PassArgs &A, PairWarp<KIND, CPLX> &W, const double2 *tl,
                                                         const LeafItem &I, unsigned hi_end,
                                                         int ng) {
    constexpr int NC = PairWarp<KIND, CPLX>::NC;
    const int nt = I.nt, lane = I.lane;
    const int sp = 32 / ng, j = lane / ng, gi = lane - j * ng;
    double tx[TB], ty[TB];
    PairSum<KIND, CPLX> acc[TB];
#pragma unroll
    for (int a = 0; a < TB; a++) {
        int i = I.t0 + (gi + a * ng < nt ? gi + a * ng : min(gi, nt - 1));  // unused slots repeat another
        if (I.idx) i = I.idx[i];
        tx[a] = I.tx[i];
        ty[a] = I.ty[i];
#pragma unroll
        for (int c = 0; c < NC; c++) acc[a].c[c] = 0.0;
    }
    const int u0 = j < sp ? j : 1 << 20;  // lanes past the last group idle
    for (int c0 = 0; !FAR && c0 < I.ns; c0 += L64_CHUNK) {
        const int cn = min(L64_CHUNK, I.ns - c0);
        __syncwarp();
#pragma unroll
        for (int h = 0; h < L64_CHUNK; h += 32) {
            const int q = h + lane;
            if (q < cn) {
                const int p = range_point(W.rng, c0 + q);
                W.stage(q, A.xs[p], A.ys[p], load_value<CPLX>(A.taus, p));
            }
        }
        __syncwarp();
        pair_chunk<KIND, CPLX, NT, TB, BEYOND>(W, tl, u0, sp, min(I.n_own - c0, cn), cn, tx, ty, A.k, I.k2, hi_end,
                                               I.check_self, acc);
    }
    if (I.l >= 2) {
        const double *lg = A.ops + (size_t)I.l * A.stride + A.off_large;
        const int Qc = A.Qc;
        __syncwarp();
        for (int q = lane; q < Qc; q += 32) {
            if constexpr (CPLX) W.stage(q, lg[q], lg[Qc + q], make_double2(I.den[q], I.den[Qc + q]));
            else W.stage(q, lg[q], lg[Qc + q], I.den[q]);
        }
        __syncwarp();
#pragma unroll
        for (int a = 0; a < TB; a++) {
            tx[a] -= I.cx;
            ty[a] -= I.cy;
        }
        pair_chunk<KIND, CPLX, NT, TB, BEYOND>(W, tl, u0, sp, 0, Qc, tx, ty, A.k, I.k2, hi_end, false, acc);
    }
    __syncwarp();
#pragma unroll
    for (int a = 0; a < TB; a++)
#pragma unroll
        for (int c = 0; c < NC; c++) W.red[c][a][lane] = acc[a].c[c];
    __syncwarp();
    PairSum<KIND, CPLX> v;
#pragma unroll
    for (int c = 0; c < NC; c++) v.c[c] = 0.0;
    if (lane < nt) {
        const int slot = lane / ng, grp = lane - slot * ng;
        for (int m = 0; m < sp; m++)
#pragma unroll
            for (int c = 0; c < NC; c++) v.c[c] += W.red[c][slot][grp + m * ng];
    }
#pragma unroll
    for (int c = 0; c < NC; c++) v.c[c] *= pair_scale<KIND>();
    return v;
}
// REST: a tile may hold fewer targets than its layout is for (separate targets)
template <int KIND, bool CPLX, bool FAR, bool REST, int NT, bool BEYOND = false>
__device__ __forceinline__ PairSum<KIND, CPLX> leaf_item_tb(const PassArgs &A, PairWarp<KIND, CPLX> &W,
                                                            const double2 *tl, const LeafItem &I, unsigned hi_end) {
    // the number of targets per lane that leaves the fewest lanes idle: pair
    // slots per source TB / (32 / ceil(lanes / TB)), compared by cross products
    const int g2 = (I.lanes + 1) >> 1;
    if constexpr (BEYOND) return leaf_item<KIND, CPLX, FAR, NT, true, 2>(A, W, tl, I, hi_end, g2);  // (a larger body)
    else {
        const int g3 = (I.lanes + 2) / 3, g4 = (I.lanes + 3) >> 2, s2 = 32 / g2, s3 = 32 / g3, s4 = 32 / g4;
        const bool four = s4 * 3 >= s3 * 4 && s4 * 2 >= s2 * 4, three = s3 * 2 >= s2 * 3;
        if constexpr (!REST) {
            if (four) return leaf_item<KIND, CPLX, FAR, NT, BEYOND, 4>(A, W, tl, I, hi_end, g4);
            if (three) return leaf_item<KIND, CPLX, FAR, NT, BEYOND, 3>(A, W, tl, I, hi_end, g3);
            return leaf_item<KIND, CPLX, FAR, NT, BEYOND, 2>(A, W, tl, I, hi_end, g2);
        }
        // fewer targets than the layout is for: as many per lane as they need
        const int ng = four ? g4 : three ? g3 : g2;
        if (I.nt > 3 * ng) return leaf_item<KIND, CPLX, FAR, NT, BEYOND, 4>(A, W, tl, I, hi_end, ng);
        if (I.nt > 2 * ng) return leaf_item<KIND, CPLX, FAR, NT, BEYOND, 3>(A, W, tl, I, hi_end, ng);
        if (I.nt <= ng) return leaf_item<KIND, CPLX, FAR, NT, BEYOND, 1>(A, W, tl, I, hi_end, ng);
        return leaf_item<KIND, CPLX, FAR, NT, BEYOND, 2>(A, W, tl, I, hi_end, ng);
    }
}

// ... with the series that reaches to tmax, the largest (k r)^2 inside the boxes
template <int KIND, bool CPLX, bool FAR, bool REST = false>
__device__ __forceinline__ PairSum<KIND, CPLX> leaf_item_series(const PassArgs &A, PairWarp<KIND, CPLX> &W,
                                                                const double2 *tl, const LeafItem &I, double tmax) {
    if (KIND == KIFMM_KERNEL_LAPLACE) return leaf_item_tb<KIND, CPLX, FAR, REST, 1>(A, W, tl, I, LOG_HI_END);
    if (tmax < 0.0625) return leaf_item_tb<KIND, CPLX, FAR, REST, SERIES_NARROW>(A, W, tl, I, SERIES_NARROW_HI);
    if (tmax < 1.0) return leaf_item_tb<KIND, CPLX, FAR, REST, SERIES_MID>(A, W, tl, I, SERIES_MID_HI);
    if (tmax < 4.0) return leaf_item_tb<KIND, CPLX, FAR, REST, SERIES_WIDE>(A, W, tl, I, SERIES_WIDE_HI);
    return leaf_item_tb<KIND, CPLX, FAR, REST, SERIES_WIDE, true>(A, W, tl, I, SERIES_WIDE_HI);
}

// 16 warps per SM at 128 registers measured 1-5% faster than 24 at 80 (the K0
// series spill there), and 64-source chunks the same as 96 or 128
constexpr int L64_MAX_WARPS = 8, L64_BLOCKS_PER_SM = 2;
// FAR: the L2P alone, added to the near field that pots already holds
template <int KIND, bool CPLX, bool FAR>
__global__ void __launch_bounds__(32 * L64_MAX_WARPS, L64_BLOCKS_PER_SM)
    k_leaf_eval_d(PassArgs A, const double2 *__restrict__ logtab, const double *__restrict__ den, unsigned nitems,
                  int ntile, int ts, int check_self, unsigned *__restrict__ ticket) {
    extern __shared__ __align__(16) unsigned char sm_l64[];
    double2 *tab = (double2 *)sm_l64;
    auto &W = ((PairWarp<KIND, CPLX> *)(tab + LOGTAB_N * LOGTAB_COPIES))[threadIdx.x >> 5];
    stage_log_table(tab, logtab);
    __syncthreads();
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const double2 *tl = tab + (lane & (LOGTAB_COPIES - 1));
    LeafItem I;
    I.tx = A.xs;
    I.ty = A.ys;
    I.idx = nullptr;
    I.lane = lane;
    I.check_self = check_self;
    I.k2 = pair_k2(A.k);
    const unsigned last = nitems + gridDim.x * (blockDim.x >> 5) - 1;
    for (;;) {
        unsigned it = 0;
        if (lane == 0) it = atomicInc(ticket, last);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= nitems) return;
        const unsigned w = it / ntile;
        const int rv = A.leaf_rec[(size_t)w * LEAF_REC_WORDS + lane];
        const int l = __shfl_sync(0xffffffffu, rv, LR_LEVEL), b = __shfl_sync(0xffffffffu, rv, LR_BOT),
                  e = __shfl_sync(0xffffffffu, rv, LR_TOP);
        const uint64_t key = (uint64_t)(uint32_t)__shfl_sync(0xffffffffu, rv, LR_KEY_LO) |
                             ((uint64_t)(uint32_t)__shfl_sync(0xffffffffu, rv, LR_KEY_HI) << 32);
        I.ns = __shfl_sync(0xffffffffu, rv, LR_NSRC);
        if (FAR && l < 2) continue;
        __syncwarp();
        if (lane >= LR_RNG && lane < LR_RNG + 18) W.rng[lane - LR_RNG] = rv;
        __syncwarp();
        const double wl = ldexp(A.W, -l);
        I.l = l;
        I.cx = A.root + ((double)compact2(key >> 1) + 0.5) * wl;
        I.cy = A.root + ((double)compact2(key) + 0.5) * wl;
        I.n_own = e - b;
        I.den = den + (size_t)w * A.Q;
        // r^2 <= 8 w^2 over the 3x3 cells; to the equivalent points r < 2 w
        const double tmax = KIND == KIFMM_KERNEL_LAPLACE ? 0.0 : (FAR ? 4.0 : 8.0) * wl * wl * I.k2;
        for (int t0 = b + (int)(it - w * ntile) * ts; t0 < e; t0 += ntile * ts) {
            I.t0 = t0;
            I.lanes = I.nt = min(ts, e - t0);
            const PairSum<KIND, CPLX> v = leaf_item_series<KIND, CPLX, FAR>(A, W, tl, I, tmax);
            if (lane >= I.nt) continue;
            const int o = A.out ? A.perm[t0 + lane] : t0 + lane;
            if constexpr (CPLX) ((double2 *)(A.out ? A.out : A.pots))[o] = make_double2(v.c[0], v.c[1]);
            else (A.out ? A.out : A.pots)[o] = FAR ? A.pots[t0 + lane] + v.c[0] : v.c[0];
        }
    }
}

// Warps per block and blocks for `items` items of one warp each.  A block's
// table is shared by its warps; fewer items than resident warps: smaller
// blocks, down to two warps, spread them over the SMs.
static void pair_grid(const kifmm_plan *P, int64_t items, size_t warp_bytes, int *warps, unsigned *grid,
                      size_t *smem) {
    const int64_t resident = (int64_t)P->num_sms * L64_BLOCKS_PER_SM * L64_MAX_WARPS;
    int w = L64_MAX_WARPS;
    while (w > 2 && items < (int64_t)P->num_sms * w * 2) w >>= 1;
    *warps = w;
    *grid = (unsigned)std::min<int64_t>((items + w - 1) / w, resident / w);
    *smem = LOGTAB_N * LOGTAB_COPIES * sizeof(double2) + (size_t)w * warp_bytes;
}

// (near_done: an event that the leaf pass, but not the densities, comes after)
template <int KIND, bool CPLX, bool FAR>
static void launch_leaf_eval(kifmm_plan *P, const PassArgs &A, int check_self, cudaEvent_t near_done = nullptr) {
    const int64_t nl = P->n_leaf_list;
    const double *den = launch_leaf_density(P, A);
    if (near_done) KIFMM_CUDA(cudaStreamWaitEvent(P->stream, near_done, 0));
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
    pair_grid(P, items, sizeof(PairWarp<KIND, CPLX>), &warps, &grid, &smem);
    ensure_dyn_smem(k_leaf_eval_d<KIND, CPLX, FAR>, smem);
    launch_pdl(k_leaf_eval_d<KIND, CPLX, FAR>, dim3(grid), dim3(32 * warps), smem, P->stream, A, log_table(P->device), den,
               (unsigned)items, ntile, ts, check_self, (unsigned *)(P->scal.p + KIFMM_SCAL_TICKET));
}
// P2M, one warp per node: the check points are the targets of the pair loop,
// TB of them per lane on eight lanes, and four groups of lanes share the
// node's sources (all 32 lanes busy for every Nequiv that is a multiple of 8;
// one check point per lane left 24 of 64 lane slots idle at Nequiv 40).
// Bound by issue like the leaf pass.
template <int KIND, bool CPLX, int TB, int NT, bool BEYOND = false>
__device__ __forceinline__ void p2m_node(const PassArgs &A, PairWarp<KIND, CPLX> &W, const double2 *tl, int g, int b,
                                         int e, const double *lg, double cx, double cy, unsigned hi_end, double k2,
                                         int lane) {
    constexpr int NC = PairWarp<KIND, CPLX>::NC;
    const int gi = lane & 7, j = lane >> 3, Qc = A.Qc;
    double tx[TB], ty[TB];
    PairSum<KIND, CPLX> acc[TB];
#pragma unroll
    for (int a = 0; a < TB; a++) {
        const int q = gi + 8 * a < Qc ? gi + 8 * a : 0;  // unused slots repeat the first
        tx[a] = lg[q] + cx;
        ty[a] = lg[Qc + q] + cy;
#pragma unroll
        for (int c = 0; c < NC; c++) acc[a].c[c] = 0.0;
    }
    for (int s0 = b; s0 < e; s0 += L64_CHUNK) {
        const int cn = min(L64_CHUNK, e - s0);
        __syncwarp();
#pragma unroll
        for (int h = 0; h < L64_CHUNK; h += 32) {
            const int q = h + lane;
            if (q < cn) W.stage(q, A.xs[s0 + q], A.ys[s0 + q], load_value<CPLX>(A.taus, s0 + q));
        }
        __syncwarp();
        pair_chunk<KIND, CPLX, NT, TB, BEYOND>(W, tl, j, 4, 0, cn, tx, ty, A.k, k2, hi_end, false, acc);
    }
#pragma unroll
    for (int a = 0; a < TB; a++)
#pragma unroll
        for (int c = 0; c < NC; c++) {
            double v = acc[a].c[c];
            v += __shfl_xor_sync(0xffffffffu, v, 8);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            if (j == 0 && gi + 8 * a < Qc) A.uup[(size_t)g * A.Q + c * Qc + gi + 8 * a] = v * pair_scale<KIND>();
        }
}
template <int KIND, bool CPLX, int TB>
__global__ void __launch_bounds__(32 * L64_MAX_WARPS, L64_BLOCKS_PER_SM)
    k_p2m_d(PassArgs A, const double2 *__restrict__ logtab, const int32_t *__restrict__ list, int64_t nlist) {
    extern __shared__ __align__(16) unsigned char sm_p2m[];
    double2 *tab = (double2 *)sm_p2m;
    auto &W = ((PairWarp<KIND, CPLX> *)(tab + LOGTAB_N * LOGTAB_COPIES))[threadIdx.x >> 5];
    stage_log_table(tab, logtab);
    __syncthreads();
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const double2 *tl = tab + (lane & (LOGTAB_COPIES - 1));
    const double k2 = pair_k2(A.k);
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t w = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); w < nlist; w += nw) {
        const int g = list[w], l = A.nlev[g], b = A.nbot[g], e = A.ntop[g];
        double cx, cy;
        node_center(A, g, l, cx, cy);
        const double *lg = A.ops + (size_t)l * A.stride + A.off_large;
        const double wl = ldexp(A.W, -l), tmax = 4.0 * wl * wl * k2;  // r < 2 w to the check circle
        if (KIND == KIFMM_KERNEL_LAPLACE)
            p2m_node<KIND, CPLX, TB, 1>(A, W, tl, g, b, e, lg, cx, cy, LOG_HI_END, k2, lane);
        else if (tmax < 0.0625)
            p2m_node<KIND, CPLX, TB, SERIES_NARROW>(A, W, tl, g, b, e, lg, cx, cy, SERIES_NARROW_HI, k2, lane);
        else if (tmax < 1.0)
            p2m_node<KIND, CPLX, TB, SERIES_MID>(A, W, tl, g, b, e, lg, cx, cy, SERIES_MID_HI, k2, lane);
        else if (tmax < 4.0)
            p2m_node<KIND, CPLX, TB, SERIES_WIDE>(A, W, tl, g, b, e, lg, cx, cy, SERIES_WIDE_HI, k2, lane);
        else p2m_node<KIND, CPLX, TB, SERIES_WIDE, true>(A, W, tl, g, b, e, lg, cx, cy, SERIES_WIDE_HI, k2, lane);
    }
}
template <int KIND, bool CPLX, int TB>
static void launch_p2m_tb(kifmm_plan *P, const PassArgs &A) {
    int warps;
    unsigned grid;
    size_t smem;
    pair_grid(P, P->n_p2m_list, sizeof(PairWarp<KIND, CPLX>), &warps, &grid, &smem);
    ensure_dyn_smem(k_p2m_d<KIND, CPLX, TB>, smem);
    launch_pdl(k_p2m_d<KIND, CPLX, TB>, dim3(grid), dim3(32 * warps), smem, P->stream, A, log_table(P->device),
               (const int32_t *)P->p2m_list.p, P->n_p2m_list);
}
template <int KIND, bool CPLX>
static void launch_p2m_kind(kifmm_plan *P, const PassArgs &A) {
    const int tb = (P->Qc + 7) / 8;  // Nequiv <= 64, complex <= 32
    if (tb <= 2) launch_p2m_tb<KIND, CPLX, 2>(P, A);
    else if (tb == 3) launch_p2m_tb<KIND, CPLX, 3>(P, A);
    else if (CPLX || tb == 4) launch_p2m_tb<KIND, CPLX, 4>(P, A);
    else if constexpr (!CPLX) {
        if (tb == 5) launch_p2m_tb<KIND, CPLX, 5>(P, A);
        else if (tb == 6) launch_p2m_tb<KIND, CPLX, 6>(P, A);
        else launch_p2m_tb<KIND, CPLX, 8>(P, A);
    }
}
}  // namespace kifmm
