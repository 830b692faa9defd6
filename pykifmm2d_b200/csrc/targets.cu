// targets.cu -- evaluation at separate targets (class_fmm.py:379-399 with
// targets other than the sources): locate (numba_locate_points,
// tree.py:712-727), L2P and P2P, in FP64 (real and complex values) and in the
// mixed form's FP32 near field.
//
// Targets are grouped by the leaf that holds them, so that a warp's targets
// share one leaf: its source ranges, its sources staged once in shared memory,
// and the equivalent density of its local expansion.  Grouping is one descent
// per target with a rank among its leaf's targets (counted per block in a
// shared-memory hash table, then one global atomic per block and leaf), one pass
// over the nodes that lays out the groups and their work items, and one pass
// that writes the targets' indices in group order; a Morton sort of the targets
// took ten passes over them (0.32 of 1.26 ms at 3M targets).  The order within a
// group is whatever the atomics give, and with it the targets that share an item;
// no target's sum depends on it, so that equal calls give equal bits: the FP32 form
// sums a target on one lane, the others split the sources over lanes in the same
// way for all of a leaf's targets (TargetItem::lanes).
#include "leaf_f32.cuh"
#include "pass_f64.cuh"

namespace kifmm {

struct TargetItem {
    int g, start;    // leaf, first grouped target
    short n, lanes;  // targets (<= TI_MAX); those of the leaf's largest 32-target tile
    int level;
};
constexpr int TI_MAX = 64;  // most targets of an item: two per lane in the packed FP32 loop

// counters of a call (P->tcount): targets laid out, items, ticket; targets left out of
// the groups
enum { TC_TARGETS, TC_ITEMS, TC_TICKET, TC_APART, TC_WORDS };

constexpr int TL_THREADS = 256, TL_PER = 8, TL_TILE = TL_THREADS * TL_PER, TL_SLOTS = 2 * TL_TILE;
// the leaf of every target and its rank among the leaf's targets; cnt[node]:
// targets of the node.  The strict '>' descent takes, level by level, the bits of
// the target's cell on the key grid (whose lines are the cells' midlines at
// every level): the coordinates clamped into the box, NaN in cell 0.  order (or
// null): targets out of reach are left out of the groups, leaf ~g, and listed from its
// end.
__global__ void __launch_bounds__(TL_THREADS) k_target_leaf(PassArgs A, const double *__restrict__ tx,
                                                            const double *__restrict__ ty, int64_t n, double h,
                                                            unsigned *__restrict__ cnt, int32_t *__restrict__ leaf,
                                                            unsigned *__restrict__ rank, unsigned *__restrict__ tcount,
                                                            int32_t *__restrict__ order) {
    __shared__ int key[TL_SLOTS];
    __shared__ unsigned num[TL_SLOTS];
    for (int i = threadIdx.x; i < TL_SLOTS; i += TL_THREADS) {
        key[i] = -1;
        num[i] = 0;
    }
    __syncthreads();
    const int64_t i0 = (int64_t)blockIdx.x * TL_TILE;
    int slot[TL_PER], lf[TL_PER];
    unsigned rk[TL_PER], cx[TL_PER], cy[TL_PER], apart = 0;
    // the thread's descents side by side, a level of all of them per pass: their
    // node loads overlap
#pragma unroll
    for (int k = 0; k < TL_PER; k++) {
        const int64_t i = i0 + k * TL_THREADS + threadIdx.x;
        const double px = i < n ? tx[i] : 0.0, py = i < n ? ty[i] : 0.0;
        if (order && out_of_reach(px, py)) apart |= 1u << k;
        cx[k] = h > 0 && px == px ? (unsigned)grid_cell(px, A.root, h) << (32 - KEY_DEPTH) : 0u;
        cy[k] = h > 0 && py == py ? (unsigned)grid_cell(py, A.root, h) << (32 - KEY_DEPTH) : 0u;
        lf[k] = 0;
    }
    for (bool more = true; more;) {
        bool split[TL_PER];
        int child[TL_PER];
#pragma unroll
        for (int k = 0; k < TL_PER; k++) {
            split[k] = A.nflag[lf[k]] & NF_SPLIT;
            child[k] = A.nchild[lf[k]];
        }
        more = false;
#pragma unroll
        for (int k = 0; k < TL_PER; k++)
            if (split[k]) {
                lf[k] = child[k] + (int)(2 * (cx[k] >> 31) + (cy[k] >> 31));
                cx[k] <<= 1;
                cy[k] <<= 1;
                more = true;
            }
    }
#pragma unroll
    for (int k = 0; k < TL_PER; k++) {
        const int64_t i = i0 + k * TL_THREADS + threadIdx.x;
        slot[k] = -1;
        if (i >= n) continue;
        if ((apart >> k) & 1u) {
            leaf[i] = ~lf[k];
            order[n - 1 - atomicAdd(&tcount[TC_APART], 1u)] = (int32_t)i;
            continue;
        }
        int s = (int)((unsigned)lf[k] * 2654435761u >> 20) & (TL_SLOTS - 1);
        for (;;) {  // at most TL_TILE distinct leaves in twice as many slots
            const int was = atomicCAS(&key[s], -1, lf[k]);
            if (was == -1 || was == lf[k]) break;
            s = (s + 1) & (TL_SLOTS - 1);
        }
        slot[k] = s;
        rk[k] = atomicAdd(&num[s], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < TL_SLOTS; i += TL_THREADS)
        if (key[i] >= 0) num[i] = atomicAdd(&cnt[key[i]], num[i]);  // count -> base rank of the block's targets
    __syncthreads();
#pragma unroll
    for (int k = 0; k < TL_PER; k++) {
        const int64_t i = i0 + k * TL_THREADS + threadIdx.x;
        if (slot[k] < 0) continue;
        leaf[i] = lf[k];
        rank[i] = num[slot[k]] + rk[k];
    }
}

// first position of each node's targets, and the work items of `per` targets
__global__ void k_target_items(PassArgs A, int64_t nn, int per, const unsigned *__restrict__ cnt,
                               unsigned *__restrict__ off, TargetItem *__restrict__ items,
                               unsigned *__restrict__ tcount) {
    const int lane = threadIdx.x & 31;
    const int64_t g0 = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * 32, g = g0 + lane;
    if (g0 >= nn) return;
    const unsigned c = g < nn ? cnt[g] : 0u, it = (c + per - 1) / per;
    unsigned sc = c, si = it;  // inclusive scans within the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned a = __shfl_up_sync(0xffffffffu, sc, o), b = __shfl_up_sync(0xffffffffu, si, o);
        if (lane >= o) sc += a, si += b;
    }
    unsigned bc = 0, bi = 0;
    if (lane == 31 && sc) {
        bc = atomicAdd(&tcount[TC_TARGETS], sc);
        bi = atomicAdd(&tcount[TC_ITEMS], si);
    }
    bc = __shfl_sync(0xffffffffu, bc, 31) + sc - c;
    bi = __shfl_sync(0xffffffffu, bi, 31) + si - it;
    if (c) off[g] = bc;
    for (unsigned m = __ballot_sync(0xffffffffu, c != 0); m; m &= m - 1) {  // the warp writes one node's items
        const int j = __ffs(m) - 1;
        const unsigned cj = __shfl_sync(0xffffffffu, c, j), oj = __shfl_sync(0xffffffffu, bc, j),
                       fj = __shfl_sync(0xffffffffu, bi, j), nj = __shfl_sync(0xffffffffu, it, j);
        const int lv = A.nlev[g0 + j];
        const short lanes = (short)min(min(cj, (unsigned)per), 32u);
        for (unsigned q = lane; q < nj; q += 32)
            items[fj + q] =
                TargetItem{(int)(g0 + j), (int)(oj + q * per), (short)min((unsigned)per, cj - q * per), lanes, lv};
    }
}

__global__ void k_target_place(int64_t n, const int32_t *__restrict__ leaf, const unsigned *__restrict__ rank,
                               const unsigned *__restrict__ off, int32_t *__restrict__ order) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        if (leaf[i] >= 0) order[off[leaf[i]] + rank[i]] = (int32_t)i;
}

struct TargetArgs {
    const double *tx, *ty;     // targets in the caller's order
    int64_t n;
    const int32_t *leaf;       // their leaves (~leaf: not in a group)
    const int32_t *order;      // their indices in group order, then those not in a group
    const double *den;         // [n_nodes][Q] equivalent densities
    const TargetItem *items;
    unsigned *tcount;
    double *pot;
    int check_self;
};

// source ranges of leaf g by the whole warp, in the order of A's direction
// table (own_first: the leaf itself before its colleagues); returns their total
__device__ __forceinline__ int warp_ranges(const PassArgs &A, int g, bool own_first, int *rng, int lane) {
    const int d = own_first ? (lane == 0 ? 4 : lane <= 4 ? lane - 1 : lane) : lane;
    int rb = 0, rn = 0;
    if (lane < 9) {
        const int c = A.ncoll[9 * (size_t)g + d];
        if (c >= 0) rb = A.nbot[c], rn = A.ntop[c] - rb;
    }
    int s = rn;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += u;
    }
    const int total = __shfl_sync(0xffffffffu, s, 8);
    __syncwarp();
    if (lane < 9) {
        rng[lane] = s - rn;
        rng[9 + lane] = rb - (s - rn);
    }
    __syncwarp();
    return total;
}

__device__ __forceinline__ unsigned next_item(const TargetArgs &T, int lane) {
    unsigned it = 0;
    if (lane == 0) it = atomicAdd(&T.tcount[TC_TICKET], 1u);
    return __shfl_sync(0xffffffffu, it, 0);
}

// Laplace sum of a target out of reach over n equivalent points at x[q], x[n + q]:
// whatever log() gives
template <bool CPLX>
__device__ __noinline__ PairSum<KIFMM_KERNEL_LAPLACE, CPLX> far_apart(const double *x, const double *den, int n,
                                                                      double px, double py) {
    constexpr int LAP = KIFMM_KERNEL_LAPLACE;
    PairSum<LAP, CPLX> v{};
    for (int q = 0; q < n; q++) {
        const double dx = px - x[q], dy = py - x[n + q];
        const PairValue g = pair_value_any<LAP>(fma(dx, dx, dy * dy), 0.0);
        if constexpr (CPLX) v.add(g, make_double2(den[q], den[n + q]), double2{});
        else v.add(g, den[q], double2{});
    }
    return v;
}
// ... its potential at leaf g, near sources first
template <bool CPLX>
__device__ __noinline__ void target_apart(const PassArgs &A, const TargetArgs &T, int64_t i) {
    constexpr int LAP = KIFMM_KERNEL_LAPLACE;
    const int g = ~T.leaf[i];
    const double px = T.tx[i], py = T.ty[i];
    PairSum<LAP, CPLX> v{}, far{};
    for (int d = 0; d < 9; d++) {
        const int c = A.ncoll[9 * (size_t)g + d];
        for (int s = c >= 0 ? A.nbot[c] : 0, e = c >= 0 ? A.ntop[c] : 0; s < e; s++) {
            const double dx = px - A.xs[s], dy = py - A.ys[s];
            v.add(pair_value_any<LAP>(fma(dx, dx, dy * dy), 0.0), load_value<CPLX>(A.taus, s), double2{});
        }
    }
    const int l = A.nlev[g];
    if (l >= 2) {
        double cx, cy;
        node_center(A, g, l, cx, cy);
        far = far_apart<CPLX>(A.ops + (size_t)l * A.stride + A.off_large, T.den + (size_t)g * A.Q, A.Qc, px - cx, py - cy);
    }
    for (int c = 0; c < PairWarp<LAP, CPLX>::NC; c++)
        T.pot[PairWarp<LAP, CPLX>::NC * i + c] = (v.c[c] + far.c[c]) * pair_scale<LAP>();
}

// FP64, real or complex: the leaf pass's pair loops on the item's targets
template <int KIND, bool CPLX>
__global__ void __launch_bounds__(32 * L64_MAX_WARPS, L64_BLOCKS_PER_SM)
    k_eval_targets_d(const __grid_constant__ PassArgs A, const double2 *__restrict__ logtab,
                     const __grid_constant__ TargetArgs T) {
    extern __shared__ __align__(16) unsigned char sm_tgd[];
    double2 *tab = (double2 *)sm_tgd;
    auto &W = ((PairWarp<KIND, CPLX> *)(tab + LOGTAB_N * LOGTAB_COPIES))[threadIdx.x >> 5];
    stage_log_table(tab, logtab);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const double2 *tl = tab + (lane & (LOGTAB_COPIES - 1));
    LeafItem I;
    I.tx = T.tx;
    I.ty = T.ty;
    I.idx = T.order;
    I.lane = lane;
    I.check_self = T.check_self;
    I.k2 = pair_k2(A.k);
    I.n_own = 0;  // a coincidence with a source is the exception here
    const unsigned nitems = T.tcount[TC_ITEMS];
    for (unsigned it = next_item(T, lane); it < nitems; it = next_item(T, lane)) {
        const TargetItem J = T.items[it];
        I.ns = warp_ranges(A, J.g, true, W.rng, lane);
        I.l = J.level;
        node_center(A, J.g, J.level, I.cx, I.cy);
        I.den = T.den + (size_t)J.g * A.Q;
        const double wl = ldexp(A.W, -J.level);
        I.lanes = J.lanes;
        for (int t0 = 0; t0 < J.n; t0 += 32) {
            I.t0 = J.start + t0;
            I.nt = min(32, J.n - t0);
            const PairSum<KIND, CPLX> v = leaf_item_series<KIND, CPLX, false, true>(A, W, tl, I, 8.0 * wl * wl * I.k2);
            if (lane >= I.nt) continue;
            const int o = T.order[I.t0 + lane];
            if constexpr (CPLX) ((double2 *)T.pot)[o] = make_double2(v.c[0], v.c[1]);
            else T.pot[o] = v.c[0];
        }
    }
    if constexpr (KIND == KIFMM_KERNEL_LAPLACE) {
        const unsigned na = T.tcount[TC_APART];
        for (unsigned w = blockIdx.x * blockDim.x + threadIdx.x; w < na; w += gridDim.x * blockDim.x)
            target_apart<CPLX>(A, T, T.order[T.n - 1 - w]);
    }
}

// Mixed form: P2P in FP32 on coordinates relative to the leaf's centre, one
// running sum per target over the leaf's colleagues' sources in direction
// order (pairs at distance 0 skipped); L2P in FP64 on the pair loops.  An item
// of more than 32 targets puts two on a lane and runs packed FP32 pairs:
// offsets, squared distances and products of both in one instruction, the same
// operations as the single form.  Bound by the 16/clk/SM lg2 unit (Laplace):
// 3M targets, 8e8 pairs, 0.17 ms.
// Two blocks of twelve warps to an SM: the logarithm table takes 32 KB a block, and
// three blocks of eight warps left the gathers 28 KB of L1 (3M targets: 509 us, now
// 479).
constexpr int TF_WARPS = 12, TF_BLOCKS_PER_SM = 2;
struct NearWarp {
    ulonglong2 xy[L64_CHUNK];  // (x, x | y, y)
    f32x2 z[L64_CHUNK];        // (z, z)
};
template <int KIND>
__device__ __forceinline__ float near_term(float r2, float k) {
    return KIND == KIFMM_KERNEL_LAPLACE ? __log2f(r2) : k0_f(k * sqrtf(r2));
}
template <int KIND, int TB>
__device__ __forceinline__ void target_near(const PassArgs &A, NearWarp &N, const int *rng, int ns, double cx, double cy,
                                            const float (&rx)[TB], const float (&ry)[TB], float (&acc)[TB], int lane) {
    constexpr float MIN_NORMAL = 1.17549435e-38f;
    const float kk = (float)A.k;
    f32x2 tx2 = 0, ty2 = 0, acc2 = 0;
    if (TB == 2) tx2 = f2_pack(rx[0], rx[TB - 1]), ty2 = f2_pack(ry[0], ry[TB - 1]);
    for (int c0 = 0; c0 < ns; c0 += L64_CHUNK) {
        const int cn = min(L64_CHUNK, ns - c0);
        __syncwarp();
#pragma unroll
        for (int h = 0; h < L64_CHUNK; h += 32) {
            const int q = h + lane;
            if (q < cn) {
                const int s = range_point(rng, c0 + q);
                const float x = (float)(A.xs[s] - cx), y = (float)(A.ys[s] - cy), z = (float)A.taus[s];
                N.xy[q] = make_ulonglong2(f2_pack(x, x), f2_pack(y, y));
                N.z[q] = f2_pack(z, z);
            }
        }
        __syncwarp();
        if (KIND == KIFMM_KERNEL_LAPLACE && TB == 2) {
#pragma unroll 2
            for (int u = 0; u < cn; u++) {
                const ulonglong2 s = N.xy[u];
                const f32x2 z = N.z[u], dx = f2_sub(tx2, s.x), dy = f2_sub(ty2, s.y);
                const f32x2 r = f2_fma(dx, dx, f2_mul(dy, dy));
                float ra, rb;
                f2_unpack(r, ra, rb);
                if (ra >= MIN_NORMAL && rb >= MIN_NORMAL) {  // lg2 of normal numbers: no scaling needed
                    acc2 = f2_fma(z, lg2_pair(r), acc2);
                } else {
                    float sa, sb, za, zb;
                    f2_unpack(acc2, sa, sb);
                    f2_unpack(z, za, zb);
                    if (ra > 0.f) sa = fmaf(za, __log2f(ra), sa);
                    if (rb > 0.f) sb = fmaf(za, __log2f(rb), sb);
                    acc2 = f2_pack(sa, sb);
                }
            }
        } else {
            for (int u = 0; u < cn; u++) {
                float x, y, z, unused;
                f2_unpack(N.xy[u].x, x, unused);
                f2_unpack(N.xy[u].y, y, unused);
                f2_unpack(N.z[u], z, unused);
#pragma unroll
                for (int a = 0; a < TB; a++) {
                    const float dx = rx[a] - x, dy = ry[a] - y;
                    const float r2 = fmaf(dx, dx, dy * dy);
                    if (r2 > 0.f) acc[a] = fmaf(z, near_term<KIND>(r2, kk), acc[a]);
                }
            }
        }
    }
    if (KIND == KIFMM_KERNEL_LAPLACE && TB == 2) f2_unpack(acc2, acc[0], acc[TB - 1]);
}
template <int KIND, int TB>
__device__ __forceinline__ void target_item_f(const PassArgs &A, const TargetArgs &T, const TargetItem &J,
                                              PairWarp<KIND, false> &W, NearWarp &N, const double2 *tl, int lane) {
    constexpr float SCALE = KIND == KIFMM_KERNEL_LAPLACE ? -0.05515890934390497f : 0.15915494309189535f;  // -ln 2/(4 pi)
    double cx, cy;
    node_center(A, J.g, J.level, cx, cy);
    const int ns = warp_ranges(A, J.g, false, W.rng, lane);
    double tx[TB], ty[TB];
    float rx[TB], ry[TB], acc[TB];
#pragma unroll
    for (int a = 0; a < TB; a++) {
        const int i = T.order[J.start + min(lane + 32 * a, J.n - 1)];  // lanes past the end repeat the last target
        tx[a] = T.tx[i] - cx;
        ty[a] = T.ty[i] - cy;
        rx[a] = (float)tx[a];
        ry[a] = (float)ty[a];
        acc[a] = 0.f;
    }
    target_near<KIND, TB>(A, N, W.rng, ns, cx, cy, rx, ry, acc, lane);
    PairSum<KIND, false> far[TB];
#pragma unroll
    for (int a = 0; a < TB; a++) far[a].c[0] = 0.0;
    if (J.level >= 2) {
        const double *lg = A.ops + (size_t)J.level * A.stride + A.off_large, *den = T.den + (size_t)J.g * A.Q;
        __syncwarp();
        for (int q = lane; q < A.Q; q += 32) W.stage(q, lg[q], lg[A.Q + q], den[q]);
        __syncwarp();
        const double wl = ldexp(A.W, -J.level), k2 = pair_k2(A.k), tmax = 4.0 * wl * wl * k2;  // r < 2 w inside the box
        if (KIND == KIFMM_KERNEL_LAPLACE)
            pair_chunk<KIND, false, 1, TB, false>(W, tl, 0, 1, 0, A.Q, tx, ty, A.k, k2, LOG_HI_END, false, far);
        else if (tmax < 0.0625)
            pair_chunk<KIND, false, SERIES_NARROW, TB, false>(W, tl, 0, 1, 0, A.Q, tx, ty, A.k, k2, SERIES_NARROW_HI,
                                                              false, far);
        else if (tmax < 1.0)
            pair_chunk<KIND, false, SERIES_MID, TB, false>(W, tl, 0, 1, 0, A.Q, tx, ty, A.k, k2, SERIES_MID_HI, false,
                                                           far);
        else if (tmax < 4.0)
            pair_chunk<KIND, false, SERIES_WIDE, TB, false>(W, tl, 0, 1, 0, A.Q, tx, ty, A.k, k2, SERIES_WIDE_HI, false,
                                                            far);
        else
            pair_chunk<KIND, false, SERIES_WIDE, TB, true>(W, tl, 0, 1, 0, A.Q, tx, ty, A.k, k2, SERIES_WIDE_HI, false,
                                                           far);
        if constexpr (KIND == KIFMM_KERNEL_LAPLACE) {
#pragma unroll
            for (int a = 0; a < TB; a++)
                if (out_of_reach(tx[a], ty[a])) far[a] = far_apart<false>(lg, den, A.Q, tx[a], ty[a]);
        }
    }
#pragma unroll
    for (int a = 0; a < TB; a++)
        if (lane + 32 * a < J.n)
            T.pot[T.order[J.start + lane + 32 * a]] = (double)(acc[a] * SCALE) + far[a].c[0] * pair_scale<KIND>();
}
template <int KIND>
__global__ void __launch_bounds__(32 * TF_WARPS, TF_BLOCKS_PER_SM)
    k_eval_targets_f(PassArgs A, const double2 *__restrict__ logtab, TargetArgs T) {
    extern __shared__ __align__(16) unsigned char sm_tgf[];
    double2 *tab = (double2 *)sm_tgf;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    PairWarp<KIND, false> &W = ((PairWarp<KIND, false> *)(tab + LOGTAB_N * LOGTAB_COPIES))[warp];
    NearWarp &N = ((NearWarp *)((PairWarp<KIND, false> *)(tab + LOGTAB_N * LOGTAB_COPIES) + nw))[warp];
    stage_log_table(tab, logtab);
    __syncthreads();
    const double2 *tl = tab + (lane & (LOGTAB_COPIES - 1));
    const unsigned nitems = T.tcount[TC_ITEMS];
    for (unsigned it = next_item(T, lane); it < nitems; it = next_item(T, lane)) {
        const TargetItem J = T.items[it];
        if (J.n > 32) target_item_f<KIND, 2>(A, T, J, W, N, tl, lane);
        else target_item_f<KIND, 1>(A, T, J, W, N, tl, lane);
    }
}

// groups the targets and evaluates the leaves' equivalent densities
static TargetArgs group_targets(kifmm_plan *P, const PassArgs &A, const double *tx, const double *ty, int64_t n,
                                int check_self, bool fp32, double *pot) {
    cudaStream_t s = P->stream;
    // Targets per item: 64, fewer where that leaves the resident warps less than
    // four items each (a launch of 1.3 rounds of items lasts two); down to 32 for
    // the FP32 form, which keeps a target on one lane, and to 8 for the others.
    const int64_t nn = P->n_nodes, want = 4 * (int64_t)P->num_sms * L64_BLOCKS_PER_SM * L64_MAX_WARPS;
    int per = TI_MAX;
    while (per > (fp32 ? 32 : 8) && n / per < want) per >>= 1;
    const int64_t max_items = (n + per - 1) / per + std::min(n, nn);
    P->tleaf.alloc(n);
    P->trank.alloc(n);
    P->tperm.alloc(n);
    P->tcount.alloc(TC_WORDS + 2 * nn);  // counters, targets per node, first target of each node
    P->titems.alloc(4 * max_items);
    unsigned *cnt = P->tcount.p + TC_WORDS, *off = cnt + nn;
    KIFMM_CUDA(cudaMemsetAsync(P->tcount.p, 0, (TC_WORDS + nn) * sizeof(unsigned), s));
    k_target_leaf<<<(unsigned)((n + TL_TILE - 1) / TL_TILE), TL_THREADS, 0, s>>>(
        A, tx, ty, n, std::ldexp(P->W, -KEY_DEPTH), cnt, P->tleaf.p, P->trank.p, P->tcount.p,
        P->kern.kind == KIFMM_KERNEL_LAPLACE && !fp32 ? P->tperm.p : nullptr);
    KIFMM_LAUNCHED();
    k_target_items<<<(unsigned)((nn + 255) / 256), 256, 0, s>>>(A, nn, per, cnt, off, (TargetItem *)P->titems.p,
                                                                P->tcount.p);
    KIFMM_LAUNCHED();
    k_target_place<<<grid_for(n, 256, P->num_sms * 16), 256, 0, s>>>(n, P->tleaf.p, P->trank.p, off, P->tperm.p);
    KIFMM_LAUNCHED();
    TargetArgs T{};
    T.n = n;
    T.leaf = P->tleaf.p;
    T.tx = tx;
    T.ty = ty;
    T.order = P->tperm.p;
    T.den = launch_node_density(P, A);
    T.items = (const TargetItem *)P->titems.p;
    T.tcount = P->tcount.p;
    T.pot = pot;
    T.check_self = check_self;
    return T;
}
// at most one warp per item; the items are counted on the device
static unsigned target_grid(const kifmm_plan *P, int64_t n, int warps, int blocks_per_sm) {
    const int64_t items = std::min<int64_t>(n, n / 8 + P->n_nodes);
    return (unsigned)std::min<int64_t>((items + warps - 1) / warps, (int64_t)P->num_sms * blocks_per_sm);
}
template <int KIND, bool CPLX>
static void eval_targets_d(kifmm_plan *P, const PassArgs &A, const TargetArgs &T, int64_t n) {
    const size_t smem = LOGTAB_N * LOGTAB_COPIES * sizeof(double2) + L64_MAX_WARPS * sizeof(PairWarp<KIND, CPLX>);
    ensure_dyn_smem(k_eval_targets_d<KIND, CPLX>, smem);
    k_eval_targets_d<KIND, CPLX><<<target_grid(P, n, L64_MAX_WARPS, L64_BLOCKS_PER_SM), 32 * L64_MAX_WARPS, smem,
                                   P->stream>>>(A, log_table(P->device), T);
    KIFMM_LAUNCHED();
}
template <int KIND>
static void eval_targets_f(kifmm_plan *P, const PassArgs &A, const TargetArgs &T, int64_t n) {
    const size_t smem = LOGTAB_N * LOGTAB_COPIES * sizeof(double2) +
                        TF_WARPS * (sizeof(PairWarp<KIND, false>) + sizeof(NearWarp));
    ensure_dyn_smem(k_eval_targets_f<KIND>, smem);
    k_eval_targets_f<KIND><<<target_grid(P, n, TF_WARPS, TF_BLOCKS_PER_SM), 32 * TF_WARPS, smem, P->stream>>>(
        A, log_table(P->device), T);
    KIFMM_LAUNCHED();
}

// the targets of one grouping: their indices are 32-bit
static void eval_targets(kifmm_plan *P, const double *tx, const double *ty, int64_t n, int check_self, double *pot) {
    constexpr int LAP = KIFMM_KERNEL_LAPLACE, K0 = KIFMM_KERNEL_MOD_HELMHOLTZ, H0 = KIFMM_KERNEL_HELMHOLTZ;
    const PassArgs A = make_pass_args(P);
    const bool fp32 = P->opt.precision == KIFMM_PREC_MIXED && !P->opt.near_fp64 && !P->cplx;
    const TargetArgs T = group_targets(P, A, tx, ty, n, check_self, fp32, pot);
    const int kind = P->kern.kind;
    if (P->cplx) {
        if (kind == LAP) eval_targets_d<LAP, true>(P, A, T, n);
        else if (kind == K0) eval_targets_d<K0, true>(P, A, T, n);
        else eval_targets_d<H0, true>(P, A, T, n);
    } else if (fp32) {
        if (kind == LAP) eval_targets_f<LAP>(P, A, T, n);
        else eval_targets_f<K0>(P, A, T, n);
    } else if (kind == LAP) eval_targets_d<LAP, false>(P, A, T, n);
    else eval_targets_d<K0, false>(P, A, T, n);
}

// The real forms refuse more than 2^31 - 1 targets; the complex one takes any number,
// in runs.
void run_eval_targets(kifmm_plan *P, const double *tx, const double *ty, int64_t n, int check_self, double *pot) {
    constexpr int64_t RUN = 1ll << 27;
    KIFMM_REQUIRE(P->cplx || n < (1ll << 31), KIFMM_ERR_ARG, "evaluate_to_points: more than 2^31 - 1 targets");
    if (!P->cplx) return eval_targets(P, tx, ty, n, check_self, pot);
    for (int64_t i = 0; i < n; i += RUN) eval_targets(P, tx + i, ty + i, std::min(RUN, n - i), check_self, pot + 2 * i);
}

}  // namespace kifmm
