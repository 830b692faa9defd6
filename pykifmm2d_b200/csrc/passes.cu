// passes.cu -- FMM passes in FP64 (the "plain" form) and their drivers.
//
// Reference: FMM.build_expansions (pykifmm2d/class_fmm.py:299-352) and
// FMM.evaluate_to_points (:379-399).  State is kept as check potentials:
//   u_up   (reference Check_Us)        -- upward check potential of a node;
//   u_down (reference Local_Solutions) -- downward check potential of a node.
// Nodes of a level are stored sibling-group contiguous, so the four children
// of an entry (split or X-list cell) form one 4Q vector.
#include <algorithm>

#include "kifmm_internal.cuh"
#include "passes.cuh"
#include "async_copy.cuh"

namespace kifmm {

// Densities to tree order.  The apply's first kernel: it also clears the
// scalars that an apply starts from (error flags, ticket), flags[0 .. nflag).
__global__ void k_gather_tau(const double *__restrict__ tau, const int32_t *__restrict__ perm, int64_t n,
                             double *__restrict__ taus, unsigned long long *__restrict__ flags, int nflag) {
    pdl_wait();
    pdl_trigger();  // the P2M's blocks fill every SM: not before this kernel runs
    if (blockIdx.x == 0 && threadIdx.x < nflag) flags[threadIdx.x] = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        taus[i] = tau[perm[i]];
}

__global__ void k_scatter_pot(const double *__restrict__ pots, const int32_t *__restrict__ perm, int64_t n,
                              double *__restrict__ pot) {
    pdl_trigger();
    pdl_wait();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        pot[perm[i]] = pots[i];
}

// M2L + L2L into the children of the split entries of level l (targets on
// level l+1): class_fmm.py:324-343.  A block owns M2L_TE entries and 4Q rows;
// for each parent direction the source groups are staged in shared memory
// and the column-major operator is streamed once per block.
constexpr int M2L_TE = 16;
__global__ void k_m2l_d(PassArgs A, int l) {
    extern __shared__ double sm[];
    const int Q = A.Q, Q4 = 4 * Q, r = threadIdx.x;
    double *src = sm;                         // [TE][4Q]
    __shared__ int64_t sgrp[M2L_TE];
    __shared__ int spar[M2L_TE];
    __shared__ int64_t schild[M2L_TE];
    const int64_t e0 = (int64_t)blockIdx.x * M2L_TE;
    const int64_t ne = A.T.ne[l];
    if (r < M2L_TE) {
        int64_t e = e0 + r;
        bool act = e < ne && !(A.ent[A.T.eoff[l] + e] & 1);
        spar[r] = act ? A.ent_node[A.T.eoff[l] + e] : -1;
        schild[r] = act ? A.T.off[l + 1] + 4 * e : -1;
    }
    __syncthreads();
    double acc[M2L_TE];
#pragma unroll
    for (int t = 0; t < M2L_TE; t++) acc[t] = 0.0;
    const double *opl = A.ops + (size_t)(l + 1) * A.stride + A.off_m2l;
    for (int d = 0; d < 9; d++) {
        if (d == 4) continue;
        if (r < M2L_TE) {
            int p = spar[r];
            int64_t grp = -1;
            if (p >= 0) {
                const int je = m2l_source_entry(A.ncoll, A.nent, A.nbot, A.ntop, p, d);
                if (je >= 0) grp = A.T.off[l + 1] + 4 * (je - A.T.eoff[l]);
            }
            sgrp[r] = grp;
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < M2L_TE * Q4; idx += blockDim.x) {
            int t = idx / Q4, c = idx % Q4;
            int64_t grp = sgrp[t];
            src[idx] = grp >= 0 ? A.uup[(size_t)grp * Q + c] : 0.0;
        }
        __syncthreads();
        const double *op = opl + (size_t)d * Q4 * Q4;
        if (r < Q4)
            for (int c = 0; c < Q4; c++) {
                double a = op[(size_t)c * Q4 + r];
#pragma unroll
                for (int t = 0; t < M2L_TE; t++) acc[t] = fma(a, src[t * Q4 + c], acc[t]);
            }
        __syncthreads();
    }
    if (l >= 2) {  // L2L from the parents' downward check potentials
        for (int idx = threadIdx.x; idx < M2L_TE * Q; idx += blockDim.x) {
            int t = idx / Q, c = idx % Q;
            int p = spar[t];
            src[idx] = p >= 0 ? A.udown[(size_t)p * Q + c] : 0.0;
        }
        __syncthreads();
        const double *op = A.ops + (size_t)l * A.stride + A.off_l2l;  // [Q][4Q]
        if (r < Q4)
            for (int c = 0; c < Q; c++) {
                double a = op[(size_t)c * Q4 + r];
#pragma unroll
                for (int t = 0; t < M2L_TE; t++) acc[t] = fma(a, src[t * Q + c], acc[t]);
            }
    }
    if (r < Q4)
#pragma unroll
        for (int t = 0; t < M2L_TE; t++)
            if (schild[t] >= 0) A.udown[(size_t)schild[t] * Q + r] = acc[t];
}

// M2L of every level in one launch on the FP64 tensor path (mma.sync
// m8n8k4 .f64), class_fmm.py:336-343 recast target-centric: for the children
// ta of a target group and the children sb of its source group in direction d,
//   u_down(ta) = sum_{d, sb} P_o . u_up(sb),  o = 2 d - ta + sb,
// P_o one of the level's 40 far offset blocks (Q x Q; near offsets are left
// out).  A block owns 8 NCT consecutive entries of one level (its target
// groups) and cp of their four children, 4 / cp of its four compute warps to
// each, NR row tiles (8 rows) to a warp.  A stage is a pair (d, sb) and a run of
// kc of the Q columns: the columns of the children's offset blocks, one bulk
// copy each, and that part of the targets' source vectors (zeros where a
// target has no source), copied by 16-byte cp.async.  Stages run through a ring
// of shared-memory slots, warp-specialised: two copy warps fill a slot on its
// full barriers as soon as the compute warps have arrived on its empty
// barrier, so the copies of the next stages land while one computes and no
// block-wide barrier stands in the loop.  A warp whose child has a near offset
// passes the stage over, and every warp an 8-target column tile without a
// source.  The result is assigned to the children's u_down (the L2L chain adds
// afterwards).  Needs Q even.
//
// Bound by the FP64 tensor path for large trees (256 multiply-adds in 16 clocks
// of a scheduler, the vector pipe's rate; 87 us of products in 187 us at 1M
// points, 234 before) and by the stages' latency for small ones.  What the
// shape answers to, as measured: two compute warps per scheduler keep the pipe within 2% of its rate from shared memory, one 75-80%;
// a number of compute warps that is no multiple of four leaves three
// schedulers waiting for the fourth; one warp issues a bulk copy, or a 512-byte
// cp.async instruction, about every 86 clocks (64 row copies a stage were 2400
// of 3300 clocks a stage on a 1k-point tree); a run-time test per column tile
// took 14 instructions a multiply-add.  Reading the offset blocks instead of
// assembled 4Q x 4Q ones leaves out the near blocks' products (16% on a full V
// list) and 1 MB of operator per level.
constexpr int MD_MAX_NBUF = 8;   // most ring slots
constexpr int MD_CWARPS = 4;     // compute warps of a block
constexpr int MD_PWARPS = 2;     // copy warps
constexpr int MD_BLOCK = 32 * (MD_CWARPS + MD_PWARPS);
struct M2lDmmaArgs {
    PassArgs A;
    const double *blocks;           // [L][49] offset blocks
    M2lBlocks B;
    int lmin, lmax;
    int cp;                         // children per block (1, 2 or 4)
    int kc;                         // columns of a stage (a multiple of 4)
    int nbuf;                       // ring slots
    int64_t tile_off[MAX_LEVELS + 1];  // first tile of each parent level
    long long wait_limit;
    unsigned long long *err;
};
// warp-uniform bounded wait on an mbarrier phase (every lane polls; true
// once the phase has completed, false after `limit` polls)
__device__ __forceinline__ bool warp_wait_all(uint32_t bar, uint32_t parity, long long limit) {
    return __any_sync(0xffffffffu, mbar_wait(bar, parity, limit));
}
// ... on two mbarriers at the same phase, odd lanes polling the second
__device__ __forceinline__ bool warp_wait_both(uint32_t bar0, uint32_t bar1, uint32_t parity, long long limit) {
    return __all_sync(0xffffffffu, mbar_wait(threadIdx.x & 1 ? bar1 : bar0, parity, limit));
}
__host__ __device__ __forceinline__ int pad4mod8(int m) { return m + (12 - m % 8) % 8; }
static size_t m2l_stage_bytes(const M2lBlocks &B, int cp, int te, int kc) {
    return ((size_t)cp * kc * B.ldq + (size_t)te * pad4mod8(kc)) * sizeof(double);
}
static size_t m2l_dmma_smem(const M2lBlocks &B, int cp, int te, int kc, int nbuf) {
    return std::max(nbuf * m2l_stage_bytes(B, cp, te, kc), (size_t)te * (cp * B.qp + 1) * sizeof(double)) +
           te * 8 * sizeof(int) + 64;
}
// slot of the offset between source child sb in direction dd (0..7, centre
// left out) and target child ta; -1: near
__device__ __forceinline__ int m2l_slot(int dd, int ta, int sb) {
    const int d = dd < 4 ? dd : dd + 1, dx = d / 3 - 1, dy = d - 3 * (dx + 1) - 1;
    const int ox = 2 * dx - (ta >> 1) + (sb >> 1), oy = 2 * dy - (ta & 1) + (sb & 1);
    return ox >= -1 && ox <= 1 && oy >= -1 && oy <= 1 ? -1 : (ox + 3) * 7 + oy + 3;
}
// a stage's products for the column tiles of mask CM
template <int NR, int NCT, int CM>
__device__ __forceinline__ void m2l_ksteps(double (&acc)[NR][NCT][2], const double *o, int ldq, const double *xs,
                                           int ldx, int kn) {
#pragma unroll 2
    for (int k = 0; k < kn; k += 4) {
        double a[NR], bv[NCT];
#pragma unroll
        for (int i = 0; i < NR; i++) a[i] = o[k * ldq + 8 * i];
#pragma unroll
        for (int c = 0; c < NCT; c++)
            if ((CM >> c) & 1) bv[c] = xs[8 * c * ldx + k];
#pragma unroll
        for (int c = 0; c < NCT; c++)
            if ((CM >> c) & 1)
#pragma unroll
                for (int i = 0; i < NR; i++) dmma_8x8x4(acc[i][c][0], acc[i][c][1], a[i], bv[c]);
    }
}
template <int NR, int NCT, int CM>
__device__ __forceinline__ void m2l_masked(int cm, double (&acc)[NR][NCT][2], const double *o, int ldq,
                                           const double *xs, int ldx, int kn) {
    if (cm == CM) m2l_ksteps<NR, NCT, CM>(acc, o, ldq, xs, ldx, kn);
    else if constexpr (CM > 1) m2l_masked<NR, NCT, CM - 1>(cm, acc, o, ldq, xs, ldx, kn);
}
template <int NR, int NCT>
__global__ void __launch_bounds__(MD_BLOCK, NR <= 6 ? 3 : 2) k_m2l_dmma(M2lDmmaArgs M) {
    constexpr int TE = 8 * NCT;
    extern __shared__ __align__(128) double sm_md[];
    const PassArgs &A = M.A;
    const int Q = A.Q, qp = M.B.qp, kp = M.B.kp, ldq = M.B.ldq, cp = M.cp, kc = M.kc, nbuf = M.nbuf;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ldx = pad4mod8(kc), RB = cp * qp, oblk = kc * ldq;  // doubles per child of a slot
    const size_t stage_d = (size_t)cp * oblk + (size_t)TE * ldx;
    int *ssrc = (int *)(sm_md + (nbuf * stage_d > (size_t)TE * (RB + 1) ? nbuf * stage_d : (size_t)TE * (RB + 1)));
    __shared__ __align__(8) uint64_t bars[MD_MAX_NBUF], obar[MD_MAX_NBUF], empty[MD_MAX_NBUF];
    __shared__ int sabort, snst;
    __shared__ int sact[TE];
    __shared__ int scm[8], sst[32];  // column tiles with a source; pairs: 4 dd + sb, children mask << 8
    pdl_trigger();
    const int parts = 4 / cp;
    const int64_t b = blockIdx.x / parts;
    const int ta0 = (int)(blockIdx.x - b * parts) * cp;  // this block's children
    int l = M.lmin;
    while (l < M.lmax && M.tile_off[l + 1] <= b) l++;
    const int64_t e0 = (b - M.tile_off[l]) * TE, ne = A.T.ne[l], eoff = A.T.eoff[l];
    const double *opl = M.blocks + (size_t)(l + 1) * 49 * M.B.block;  // target level's operators
    if (tid == 0) {
        for (int i = 0; i < nbuf; i++) {
            mbar_init(smem_u32(&bars[i]), 32 * MD_PWARPS);  // full: every copy lane's copies
            mbar_init(smem_u32(&obar[i]));                  // ... and the offset blocks (transaction bytes)
            mbar_init(smem_u32(&empty[i]), MD_CWARPS);      // empty: each compute warp is done with it
        }
        sabort = 0;
    }
    // the source vectors' padding (columns Q .. kp of the last run; kp - Q is 0
    // or 2) meets zero columns of the operator: it must only be finite to begin
    // with (later it holds values of the same target's earlier sources)
    if (kp > Q)
        for (int i = tid; i < nbuf * TE; i += MD_BLOCK) {
            const int slot = i / TE, n = i - slot * TE, k = Q - (kp - 1) / kc * kc;
            double *x = sm_md + slot * stage_d + (size_t)cp * oblk + (size_t)n * ldx;
            for (int c = k; c < kc; c++) x[c] = 0.0;
        }
    pdl_wait();  // u_up comes from the M2M chain
    for (int i = tid; i < TE * 8; i += MD_BLOCK) {  // the tile's targets in M2L target order
        const int64_t e = e0 + (i >> 3), ej = e < ne ? (int64_t)A.m2l_perm[eoff + e] : -1;
        const bool act = ej >= 0 && !(A.ent[ej] & 1);
        ssrc[i] = act ? A.m2l_src8[ej * 8 + (i & 7)] : -1;
        if ((i & 7) == 0) sact[i >> 3] = act ? (int)(ej - eoff) + 1 : 0;  // 1 + index in the level, 0: none
    }
    __syncthreads();
    for (int dd = warp; dd < 8; dd += MD_BLOCK / 32) {  // column tiles of direction dd with a source
        const unsigned m = __ballot_sync(0xffffffffu, lane < TE && ssrc[(lane < TE ? lane : 0) * 8 + dd] >= 0);
        int cm = 0;
#pragma unroll
        for (int c = 0; c < NCT; c++) cm |= ((m >> (8 * c)) & 0xff) ? 1 << c : 0;
        if (lane == 0) scm[dd] = cm;
    }
    __syncthreads();
    if (warp == 0) {  // the (direction, source child) pairs with a source and a far child
        int cm = 0;
        for (int c = 0; c < cp; c++) cm |= (m2l_slot(lane >> 2, ta0 + c, lane & 3) >= 0) << c;
        if (!scm[lane >> 2]) cm = 0;
        const unsigned m = __ballot_sync(0xffffffffu, cm);
        if (cm) sst[__popc(m & ((1u << lane) - 1))] = lane | cm << 8;
        if (lane == 0) snst = __popc(m);
    }
    __syncthreads();
    const int npair = snst;
    const int g = lane >> 2, t = lane & 3, wpc = MD_CWARPS / cp, ch = warp / wpc;  // the warp's child
    const int row0 = (warp - ch * wpc) * NR * 8;                                   // and its rows there
    double acc[NR][NCT][2];
#pragma unroll
    for (int i = 0; i < NR; i++)
#pragma unroll
        for (int c = 0; c < NCT; c++) acc[i][c][0] = acc[i][c][1] = 0.0;
    volatile int *abort_flag = &sabort;
    int slot = 0, round = 0;
    if (warp >= MD_CWARPS) {
        // copy warps: a stage goes into the next slot once the compute warps have
        // released the slot's previous stage.  A lane copies pieces q, q + LQ, ...
        // of the vectors of targets n0, n0 + rpp, ... (LQ lanes to a vector); the
        // source groups change with the direction only and are kept in registers.
        constexpr int LANES = 32 * MD_PWARPS, LQ = 8, RPP = LANES / LQ, MAXI = (TE + RPP - 1) / RPP;
        const int pl = tid - 32 * MD_CWARPS, n0 = pl / LQ, q0 = pl % LQ;
        const double *const src0 = A.uup + (int64_t)(A.T.off[l + 1] - 4 * eoff) * Q;
        int je[MAXI], dir = -1, issued = 0;
        auto copy_stages = [&] {  // ends at a wait that runs out, here or in another warp
            for (int pr = 0; pr < npair; pr++) {
                const int sv = sst[pr], dd = (sv >> 2) & 7, sb = sv & 3, ctile = scm[dd];
                if (dd != dir) {
                    dir = dd;
#pragma unroll
                    for (int i = 0; i < MAXI; i++) {
                        const int n = n0 + i * RPP;  // -2: no copy (no such target, or a column tile passed over)
                        je[i] = n < TE && ((ctile >> (n >> 3)) & 1) ? ssrc[n * 8 + dd] : -2;
                    }
                }
                for (int k0 = 0; k0 < kp; k0 += kc) {
                    if (round && !warp_wait_all(smem_u32(&empty[slot]), (uint32_t)(round - 1) & 1u, M.wait_limit)) {
                        if (lane == 0) {
                            *abort_flag = 1;
                            atomicOr(M.err, 1ull);
                        }
                        return;
                    }
                    if (*abort_flag) return;
                    const int kn = min(kc, kp - k0), kq = min(kc, Q - k0) >> 1;  // columns; 16-byte pieces of a vector
                    const uint32_t ob = smem_u32(&obar[slot]), od = smem_u32(sm_md + slot * stage_d);
                    if (pl == 0) mbar_expect_tx(ob, (uint32_t)(__popc(sv >> 8) * kn * ldq) * 8u);
                    __syncwarp();
                    if (pl < cp && ((sv >> (8 + pl)) & 1))
                        bulk_g2s(od + (uint32_t)(pl * oblk) * 8u,
                                 opl + (size_t)m2l_slot(dd, ta0 + pl, sb) * M.B.block + (size_t)k0 * ldq,
                                 (uint32_t)(kn * ldq) * 8u, ob);
                    issued++;
                    const uint32_t xd = od + (uint32_t)(cp * oblk + n0 * ldx) * 8u;
                    for (int q = q0; q < kq; q += LQ) {
#pragma unroll
                        for (int i = 0; i < MAXI; i++)
                            if (je[i] != -2)  // -1: zeros
                                cp_async16(xd + (uint32_t)(i * RPP * ldx + 2 * q) * 8u,
                                           src0 + (je[i] >= 0 ? (4 * (int64_t)je[i] + sb) * Q + k0 + 2 * q : 0),
                                           je[i] >= 0 ? 16 : 0);
                    }
                    cp_async_arrive(smem_u32(&bars[slot]));
                    if (++slot == nbuf) slot = 0, round++;
                }
            }
        };
        copy_stages();
        // every copy issued lands before the block goes on (consumed stages have
        // landed already; this matters after an abort)
        cp_async_wait_all();
        if (warp == MD_CWARPS)
            for (int st = issued > nbuf ? issued - nbuf : 0; st < issued; st++)
                mbar_wait(smem_u32(&obar[st % nbuf]), (uint32_t)(st / nbuf) & 1u, kDrainWaitPolls);
    } else {
        auto compute_stages = [&] {
            for (int pr = 0; pr < npair; pr++) {
                const int sv = sst[pr], cm = scm[(sv >> 2) & 7];
                const bool far = (sv >> (8 + ch)) & 1;
                for (int k0 = 0; k0 < kp; k0 += kc) {
                    if (!warp_wait_both(smem_u32(&obar[slot]), smem_u32(&bars[slot]), (uint32_t)round & 1u, M.wait_limit)) {
                        if (lane == 0) {
                            *abort_flag = 1;
                            atomicOr(M.err, 1ull);
                        }
                        return;
                    }
                    if (*abort_flag) return;
                    if (far) {
                        const double *os = sm_md + slot * stage_d;
                        m2l_masked<NR, NCT, (1 << NCT) - 1>(cm, acc, os + (size_t)ch * oblk + t * ldq + row0 + g, ldq,
                                                            os + (size_t)cp * oblk + (size_t)g * ldx + t, ldx,
                                                            min(kc, kp - k0));
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&empty[slot]));  // this warp is done with the slot
                    if (++slot == nbuf) slot = 0, round++;
                }
            }
        };
        compute_stages();
    }
    __syncthreads();
    if (*abort_flag) return;
    // D through shared memory (the stage buffers are free), then coalesced stores
    double *cs = sm_md;  // [TE targets][RB + 1]
    if (warp < MD_CWARPS)
#pragma unroll
        for (int i = 0; i < NR; i++)
#pragma unroll
            for (int c = 0; c < NCT; c++) {
                const int r = ch * qp + row0 + 8 * i + g;
                cs[(size_t)(8 * c + 2 * t) * (RB + 1) + r] = acc[i][c][0];
                cs[(size_t)(8 * c + 2 * t + 1) * (RB + 1) + r] = acc[i][c][1];
            }
    __syncthreads();
    for (int n = warp; n < TE * cp; n += MD_BLOCK / 32) {
        const int e = n / cp, c = n - e * cp;
        if (!sact[e]) continue;
        double *dst = A.udown + ((size_t)A.T.off[l + 1] + 4 * (size_t)(sact[e] - 1) + ta0 + c) * Q;
        for (int r = lane; r < Q; r += 32) dst[r] = cs[(size_t)e * (RB + 1) + c * qp + r];
    }
}
// Children per block and targets per tile.  Large trees: all four children (a
// warp each) and 16 targets, three blocks to an SM (32 targets, two blocks to
// an SM, measured 218 against 187 us at 1M points, 205 against 171 at 500k with
// Nequiv 40: their last wave costs more than the operator reads saved); while
// that makes fewer than two blocks per SM, 8 targets, then two children per
// block (where their row tiles split evenly over two warps): a block's time
// falls with its products.
struct M2lShape {
    int cp, nr, nct;
};
static int64_t m2l_tiles(const kifmm_plan *P, int lmin, int lmax, int te) {
    int64_t t = 0;
    for (int l = lmin; l <= lmax; l++) t += (P->lt.ne[l] + te - 1) / te;
    return t;
}
static M2lShape m2l_shape(const kifmm_plan *P, const M2lBlocks &B, int lmin, int lmax) {
    const int tpc = B.qp / 8;
    M2lShape S{4, tpc, 2};
    if (m2l_tiles(P, lmin, lmax, 16) < 2 * P->num_sms) S.nct = 1;
    if (S.nct == 1 && tpc % 2 == 0 && m2l_tiles(P, lmin, lmax, 8) < 2 * P->num_sms) S.cp = 2, S.nr = tpc / 2;
    return S;
}
template <int NR, int NCT>
static void launch_m2l_dmma(kifmm_plan *P, M2lDmmaArgs &M) {
    int64_t tiles = 0;
    for (int l = 0; l <= MAX_LEVELS; l++) {
        M.tile_off[l] = tiles;
        if (l >= M.lmin && l <= M.lmax) tiles += m2l_tiles(P, l, l, 8 * NCT);
    }
    if (!tiles) return;
    // A stage has about 24 columns, all of them where an SM gets one block (41 ->
    // 27 us at 1k points: half as many stages), and the ring as many slots as
    // leave room for the blocks that an SM gets, three at most.
    const int64_t blocks = tiles * (4 / M.cp), per_sm = std::min<int64_t>(3, (blocks + P->num_sms - 1) / P->num_sms);
    const int runs = per_sm == 1 ? 1 : (M.B.kp + 27) / 28;
    M.kc = ((M.B.kp + runs - 1) / runs + 3) & ~3;
    const size_t stage = m2l_stage_bytes(M.B, M.cp, 8 * NCT, M.kc);
    M.nbuf = (int)std::max<int64_t>(2, std::min<int64_t>(MD_MAX_NBUF, (int64_t)(((224 << 10) / per_sm - 4096) / stage)));
    const size_t smem = m2l_dmma_smem(M.B, M.cp, 8 * NCT, M.kc, M.nbuf);
    ensure_dyn_smem(k_m2l_dmma<NR, NCT>, smem);
    launch_pdl(k_m2l_dmma<NR, NCT>, dim3((unsigned)blocks), dim3(MD_BLOCK), smem, P->stream, M);
}
template <int NR>
static void launch_m2l_dmma_nr(kifmm_plan *P, int nct, M2lDmmaArgs &M) {
    if (nct == 2) launch_m2l_dmma<NR, 2>(P, M);
    else launch_m2l_dmma<NR, 1>(P, M);
}
static void launch_m2l_dmma(kifmm_plan *P, const PassArgs &A, int lmin, int lmax) {
    M2lDmmaArgs M{};
    M.A = A;
    M.blocks = P->ops_tmp.p;
    M.B = m2l_blocks(P->Q);
    M.lmin = lmin;
    M.lmax = lmax;
    M.wait_limit = plan_wait_polls(P);
    M.err = P->scal.p + KIFMM_SCAL_PASS_ERR;
    const M2lShape S = m2l_shape(P, M.B, lmin, lmax);
    M.cp = S.cp;
    switch (S.nr) {
        case 1: return launch_m2l_dmma_nr<1>(P, S.nct, M);
        case 2: return launch_m2l_dmma_nr<2>(P, S.nct, M);
        case 3: return launch_m2l_dmma_nr<3>(P, S.nct, M);
        case 4: return launch_m2l_dmma_nr<4>(P, S.nct, M);
        case 5: return launch_m2l_dmma_nr<5>(P, S.nct, M);
        case 6: return launch_m2l_dmma_nr<6>(P, S.nct, M);
        case 7: return launch_m2l_dmma_nr<7>(P, S.nct, M);
        default: return launch_m2l_dmma_nr<8>(P, S.nct, M);
    }
}

PassArgs make_pass_args(kifmm_plan *P) {
    PassArgs A{};
    A.T = P->lt;
    A.Q = P->Q;
    A.Qc = P->Qc;
    A.kind = P->kern.kind;
    A.k = P->kern.k;
    A.root = P->root_min;
    A.W = P->W;
    A.ops = P->ops.p;
    A.ops_f = P->ops_f.p;
    A.stride = P->ops_stride;
    A.off_inv = 0;
    A.off_m2m = (size_t)P->Q * P->Q;
    A.off_l2l = (size_t)5 * P->Q * P->Q;
    A.off_m2l = (size_t)9 * P->Q * P->Q;
    A.off_large = (size_t)153 * P->Q * P->Q;
    A.ent = P->ent.p;
    A.ent_node = P->ent_node.p;
    A.nkey = P->nkey.p;
    A.nlev = P->nlev.p;
    A.nflag = P->nflag.p;
    A.nbot = P->nbot.p;
    A.ntop = P->ntop.p;
    A.nchild = P->nchild.p;
    A.nent = P->nent.p;
    A.ncoll = P->ncoll.p;
    A.xs = P->xs.p;
    A.ys = P->ys.p;
    A.taus = P->taus.p;
    A.pots = P->pots.p;
    A.uup = P->uup.p;
    A.udown = P->udown.p;
    A.leaf_rec = P->leaf_rec.p;
    A.m2l_perm = P->m2l_perm.p;
    A.m2l_src8 = P->m2l_src8.p;
    A.taylor = P->l2p_taylor.p;
    A.leaf_coef = P->leaf_coef.p;
    return A;
}

__global__ void k_leaf_records(PassArgs A, const int32_t *__restrict__ leaves, int64_t n, int32_t *__restrict__ rec) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int g = leaves[i];
        int r[LEAF_REC_WORDS] = {};
        r[LR_NODE] = g;
        r[LR_LEVEL] = A.nlev[g];
        r[LR_BOT] = A.nbot[g];
        r[LR_TOP] = A.ntop[g];
        const uint64_t k = A.nkey[g];
        r[LR_KEY_LO] = (int32_t)(uint32_t)k;
        r[LR_KEY_HI] = (int32_t)(uint32_t)(k >> 32);
        r[LR_NSRC] = leaf_ranges(A, g, r + LR_RNG);
        int4 *o = (int4 *)(rec + i * LEAF_REC_WORDS);
#pragma unroll
        for (int q = 0; q < LEAF_REC_WORDS / 4; q++) o[q] = make_int4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
    }
}

// the leaf records of the plan's leaf list (part of the tree build)
void build_leaf_records(kifmm_plan *P) {
    P->leaf_rec.alloc((size_t)(P->n_leaf_list ? P->n_leaf_list : 1) * LEAF_REC_WORDS);
    if (!P->n_leaf_list) return;
    PassArgs A = make_pass_args(P);
    k_leaf_records<<<grid_for(P->n_leaf_list, 128, P->num_sms * 8), 128, 0, P->stream>>>(
        A, P->leaf_list.p, P->n_leaf_list, P->leaf_rec.p);
    KIFMM_LAUNCHED();
}

// M2L target order.  The entries of each level are grouped by the set of
// directions in which they have V-list sources (an 8-bit mask; entries that
// are not split go last), so that an M2L tile of consecutive targets mostly
// shares one set and skips every absent direction instead of multiplying
// zero vectors.  The mask depends on the tree only: the order is built once
// per tree.  Within a group the order is whatever the atomics give; the M2L
// result of a target does not depend on which other targets share its tile.
__global__ void k_m2l_keys(PassArgs A, int64_t n_ent, uint16_t *__restrict__ key, int32_t *__restrict__ src8,
                           unsigned *__restrict__ hist) {
    pdl_trigger();
    pdl_wait();
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool in = j < n_ent;
    unsigned bin = 0xffffffffu;
    if (in) {
        const uint64_t ej = A.ent[j];
        const int l = (int)(ej >> ENT_LEVEL_SHIFT);
        const bool split = !(ej & 1);
        int k = split ? 0 : 256, sv[8];
#pragma unroll
        for (int dd = 0; dd < 8; dd++) {
            const int d = dd < 4 ? dd : dd + 1;
            sv[dd] = split ? m2l_source_entry(A.ncoll, A.nent, A.nbot, A.ntop, A.ent_node[j], d) : -1;
            if (sv[dd] >= 0) k |= 1 << dd;
        }
        int4 *o = (int4 *)(src8 + 8 * j);
        o[0] = make_int4(sv[0], sv[1], sv[2], sv[3]);
        o[1] = make_int4(sv[4], sv[5], sv[6], sv[7]);
        key[j] = (uint16_t)k;
        bin = (unsigned)(l * M2L_KEYS + k);
    }
    const unsigned peers = __match_any_sync(0xffffffffu, bin);
    if (in && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&hist[bin], (unsigned)__popc(peers));
}

// counts -> first position of each (level, key) group, from the level's
// eoff: one block per level, an exclusive scan over the 257 keys
constexpr int M2L_SCAN_THREADS = 288;  // >= M2L_KEYS, a whole number of warps
__global__ void __launch_bounds__(M2L_SCAN_THREADS) k_m2l_cursors(LevelTable T, unsigned *__restrict__ hist) {
    __shared__ unsigned wsum[M2L_SCAN_THREADS / 32];
    pdl_trigger();
    pdl_wait();
    const int l = blockIdx.x, k = threadIdx.x, lane = k & 31, w = k >> 5;
    const unsigned c = k < M2L_KEYS ? hist[l * M2L_KEYS + k] : 0u;
    unsigned v = c;  // inclusive scan within the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    if (lane == 31) wsum[w] = v;
    __syncthreads();
    unsigned before = (unsigned)T.eoff[l];
    for (int i = 0; i < w; i++) before += wsum[i];
    if (k < M2L_KEYS) hist[l * M2L_KEYS + k] = before + v - c;
}

__global__ void k_m2l_place(const uint64_t *__restrict__ ent, const uint16_t *__restrict__ key, int64_t n_ent,
                            unsigned *__restrict__ cursor, int32_t *__restrict__ perm) {
    pdl_trigger();
    pdl_wait();
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool in = j < n_ent;
    const int lane = threadIdx.x & 31;
    const unsigned bin = in ? (unsigned)((int)(ent[j] >> ENT_LEVEL_SHIFT) * M2L_KEYS + key[j]) : 0xffffffffu;
    const unsigned peers = __match_any_sync(0xffffffffu, bin);
    const int leader = __ffs(peers) - 1;
    unsigned base = 0;
    if (in && lane == leader) base = atomicAdd(&cursor[bin], (unsigned)__popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (in) perm[base + __popc(peers & ((1u << lane) - 1))] = (int32_t)j;
}

void build_m2l_order(kifmm_plan *P) {
    const int64_t n = P->n_ent;
    P->m2l_perm.alloc(n ? n : 1);
    if (!n) return;
    KIFMM_REQUIRE(P->L <= MAX_LEVELS + 1 && n < (1ll << 31), KIFMM_ERR_ARG, "M2L order: tree too large");
    P->m2l_key.alloc(n);
    P->m2l_src8.alloc((size_t)8 * n);
    // m2l_hist ([MAX_LEVELS + 1][M2L_KEYS] counts) is allocated and cleared by
    // build_tree with the split-cell set
    PassArgs A = make_pass_args(P);
    const unsigned gr = (unsigned)((n + 255) / 256);
    launch_pdl(k_m2l_keys, dim3(gr), dim3(256), 0, P->stream, A, n, P->m2l_key.p, P->m2l_src8.p, P->m2l_hist.p);
    launch_pdl(k_m2l_cursors, dim3((unsigned)std::min(P->L, MAX_LEVELS + 1)), dim3(M2L_SCAN_THREADS), 0, P->stream,
               P->lt, P->m2l_hist.p);
    launch_pdl(k_m2l_place, dim3(gr), dim3(256), 0, P->stream, (const uint64_t *)P->ent.p,
               (const uint16_t *)P->m2l_key.p, n, P->m2l_hist.p, P->m2l_perm.p);
    KIFMM_LAUNCHED();
}

// M2M and L2L as small FP64 GEMMs per level, C[M x n] = Op[M x K] X[K x n]:
//   M2M: M = Q, K = 4Q, X = the entries' children groups (contiguous), C -> the
//        entries' own rows of u_up;
//   L2L: M = 4Q, K = Q, X = the split entries' u_down (gathered), C added to
//        their children groups.
// A block stages the whole operator and NT columns of X in shared memory and
// each thread accumulates a 4 x 4 register tile.
template <int MODE>
__global__ void __launch_bounds__(256) k_lvl_gemm_d(PassArgs A, int l, int M, int K, int NT) {
    extern __shared__ double sm_g[];
    double *opS = sm_g;                       // [K][M]
    double *xS = sm_g + (size_t)K * M;        // [NT][K + 1]
    const int ldx = K + 1;
    const int Q = A.Q;
    const int64_t ne = A.T.ne[l], eoff = A.T.eoff[l], e0 = (int64_t)blockIdx.x * NT;
    const double *op = A.ops + (size_t)l * A.stride + (MODE == 0 ? A.off_m2m : A.off_l2l);
    // operator: 16-byte loads when aligned (odd Nequiv gives odd offsets)
    if ((((uintptr_t)op) & 15) == 0 && (K * M) % 2 == 0)
        for (int i = threadIdx.x; i < K * M / 2; i += blockDim.x) ((double2 *)opS)[i] = ((const double2 *)op)[i];
    else
        for (int i = threadIdx.x; i < K * M; i += blockDim.x) opS[i] = op[i];
    const double *src0 = A.uup + (size_t)(A.T.off[l + 1] + 4 * e0) * Q;
    if (MODE == 0 && (((uintptr_t)src0) & 15) == 0) {  // children groups of consecutive entries: one block
        const int64_t nt = min((int64_t)NT, ne - e0);
        const double2 *src = (const double2 *)src0;
        for (int i = threadIdx.x; i < NT * K / 2; i += blockDim.x) {
            int t = (2 * i) / K, c = (2 * i) % K;
            double2 v = t < nt ? src[i] : make_double2(0.0, 0.0);
            xS[t * ldx + c] = v.x;
            xS[t * ldx + c + 1] = v.y;
        }
    } else {
        for (int i = threadIdx.x; i < NT * K; i += blockDim.x) {
            int t = i / K, c = i % K;
            int64_t e = e0 + t;
            double v = 0.0;
            if (e < ne) {
                if (MODE == 0) v = src0[(size_t)t * K + c];
                else if (!(A.ent[eoff + e] & 1)) v = A.udown[(size_t)A.ent_node[eoff + e] * Q + c];
            }
            xS[t * ldx + c] = v;
        }
    }
    __syncthreads();
    const int TMr = (M + 3) / 4;
    const int tx = threadIdx.x % TMr, ty = threadIdx.x / TMr;
    if (ty * 4 >= NT) return;
    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0;
    const int r0 = tx * 4;
    for (int c = 0; c < K; c++) {
        double a[4], bb[4];
#pragma unroll
        for (int i = 0; i < 4; i++) a[i] = r0 + i < M ? opS[c * M + r0 + i] : 0.0;
#pragma unroll
        for (int j = 0; j < 4; j++) bb[j] = xS[(ty * 4 + j) * ldx + c];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = fma(a[i], bb[j], acc[i][j]);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        int64_t e = e0 + ty * 4 + j;
        if (e >= ne) continue;
        if (MODE == 0) {
            double *dst = A.uup + (size_t)A.ent_node[eoff + e] * Q;
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (r0 + i < M) dst[r0 + i] = acc[i][j];
        } else {
            if (A.ent[eoff + e] & 1) continue;
            double *dst = A.udown + (size_t)(A.T.off[l + 1] + 4 * e) * Q;
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (r0 + i < M) dst[r0 + i] += acc[i][j];
        }
    }
}

// The same products with the operator held once per block and one entry per
// lane: warp w of a block takes 32 entries and RPT rows of the operator, so
// every operator read is a shared-memory broadcast (two rows per 16-byte
// load) and each thread's RPT accumulators are FP64-pipe bound.  Rows are
// padded to Mp = RG * RPT with zeros.  Blocks hold NT = 32 * S entries, S
// sets of wps = min(RG, 8) warps; with RG > 8 a warp loops over row groups.
constexpr int LG_THREADS = 256;

// Copy n doubles from global memory through store(i, v), i in [0, n), with
// eight independent loads per thread in flight (16-byte loads when src is
// 16-byte aligned and n even).  Small staging loops are otherwise bound by
// one load latency per iteration.
template <int NTHR, class F>
__device__ __forceinline__ void stage_f64(const double *__restrict__ src, int n, F store) {
    if ((((uintptr_t)src) & 15) == 0 && (n & 1) == 0) {
        const double2 *s2 = (const double2 *)src;
        const int n2 = n >> 1;
        for (int i0 = threadIdx.x; i0 < n2; i0 += 8 * NTHR) {
            double2 v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int i = i0 + k * NTHR;
                v[k] = i < n2 ? s2[i] : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int i = i0 + k * NTHR;
                if (i < n2) {
                    store(2 * i, v[k].x);
                    store(2 * i + 1, v[k].y);
                }
            }
        }
    } else {
        for (int i0 = threadIdx.x; i0 < n; i0 += 8 * NTHR) {
            double v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int i = i0 + k * NTHR;
                v[k] = i < n ? src[i] : 0.0;
            }
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int i = i0 + k * NTHR;
                if (i < n) store(i, v[k]);
            }
        }
    }
}
template <int MODE, int RPT>
__global__ void __launch_bounds__(LG_THREADS) k_lvl_gemm_b(PassArgs A, int l, int M, int K, int Mp, int NT) {
    extern __shared__ __align__(16) double sm_b[];
    double *opS = sm_b;                    // [K][Mp]
    double *xS = sm_b + (size_t)K * Mp;    // [NT][K + 1]
    const int ldx = K + 1, Q = A.Q;
    const int64_t ne = A.T.ne[l], eoff = A.T.eoff[l], e0 = (int64_t)blockIdx.x * NT;
    const int nt = (int)min((int64_t)NT, ne - e0);
    const double *op = A.ops + (size_t)l * A.stride + (MODE == 0 ? A.off_m2m : A.off_l2l);  // [K][M]
    // staging: eight independent loads per thread in flight
    if (Mp != M)
        for (int i = threadIdx.x; i < K * Mp; i += LG_THREADS) opS[i] = 0.0;
    stage_f64<LG_THREADS>(op, K * M, [&](int i, double v) {
        const int c = i / M;
        opS[c * Mp + (i - c * M)] = v;
    });
    if (MODE == 0) {  // children groups of consecutive entries are contiguous
        const double *src0 = A.uup + (size_t)(A.T.off[l + 1] + 4 * e0) * Q;
        for (int i = nt * K + threadIdx.x; i < NT * K; i += LG_THREADS) {
            const int t = i / K;
            xS[t * ldx + (i - t * K)] = 0.0;
        }
        stage_f64<LG_THREADS>(src0, nt * K, [&](int i, double v) {
            const int t = i / K;
            xS[t * ldx + (i - t * K)] = v;
        });
    } else {
        for (int i0 = threadIdx.x; i0 < NT * K; i0 += 8 * LG_THREADS) {
            double v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int i = i0 + k * LG_THREADS, t = i / K;
                v[k] = 0.0;
                if (i < NT * K && t < nt && !(A.ent[eoff + e0 + t] & 1))
                    v[k] = A.udown[(size_t)A.ent_node[eoff + e0 + t] * Q + (i - t * K)];
            }
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int i = i0 + k * LG_THREADS, t = i / K;
                if (i < NT * K) xS[t * ldx + (i - t * K)] = v[k];
            }
        }
    }
    __syncthreads();
    const int RG = Mp / RPT, wps = RG < 8 ? RG : 8, S = 8 / wps;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int set = warp / wps;
    if (set >= S) return;
    const int t = set * 32 + lane;
    const double *xp = xS + (size_t)t * ldx;
    for (int rg = warp % wps; rg < RG; rg += wps) {
        double acc[RPT];
#pragma unroll
        for (int i = 0; i < RPT; i++) acc[i] = 0.0;
        const double *ap = opS + rg * RPT;
#pragma unroll 2
        for (int c = 0; c < K; c++) {
            const double xv = xp[c];
            const double2 *a2 = (const double2 *)(ap + (size_t)c * Mp);
#pragma unroll
            for (int i = 0; i < RPT / 2; i++) {
                const double2 a = a2[i];
                acc[2 * i] = fma(a.x, xv, acc[2 * i]);
                acc[2 * i + 1] = fma(a.y, xv, acc[2 * i + 1]);
            }
        }
        if (t < nt) {
            const int64_t e = e0 + t;
            const int r0 = rg * RPT;
            if (MODE == 0) {
                double *dst = A.uup + (size_t)A.ent_node[eoff + e] * Q + r0;
#pragma unroll
                for (int i = 0; i < RPT; i++)
                    if (r0 + i < M) dst[i] = acc[i];
            } else if (!(A.ent[eoff + e] & 1)) {
                double *dst = A.udown + (size_t)(A.T.off[l + 1] + 4 * e) * Q + r0;
#pragma unroll
                for (int i = 0; i < RPT; i++)
                    if (r0 + i < M) dst[i] += acc[i];
            }
        }
    }
}

// The same products on the FP64 tensor path (mma.sync m8n8k4 .f64), Q = 4 KS.
// A block takes 8 entries at a time; warps 2 c and 2 c + 1 take child c of
// them, half of its row tiles (8 rows) each.  Every operand goes straight from
// L2 into the fragments' registers: the warp's part of the operator before the
// wait for the previous level's kernel, then, all loads in flight at once, the
// entries' vectors (M2M: child c's; L2L: the entry's own, and the child's
// current values as the accumulators' start).  M2M adds the children's four
// products in shared memory; L2L stores its fragments.  Fragments:
// A[row = lane/4][k = lane%4], B[k = lane%4][n = lane/4],
// C[row = lane/4][n = 2*(lane%4) + {0,1}].
//
// A level holds 10 to 10,000 entries, and the levels depend on one another: what
// counts is the time from the previous kernel's end to this one's, here one
// L2 round trip, KS multiply-adds deep, and the stores.  With the operator and
// the vectors staged in shared memory by one bulk copy per row (about 86
// clocks each from one warp) and 32 entries to a warp, a level took 6.8 us
// (M2M) and 8.3 us (L2L) whatever its size.  Values that the previous kernel
// wrote are read past L1 (__ldcg).
constexpr int LD_THREADS = 256, LD_TE = 8;
template <int MODE, int KS>
struct LvlTile {
    static constexpr int Q = 4 * KS, NR = (Q + 7) / 8, NRW = (NR + 1) / 2;
    double red[MODE == 0 ? 2 : 1][MODE == 0 ? 4 : 1][MODE == 0 ? LD_TE : 1][MODE == 0 ? 8 * NR + 1 : 1];
    int snode[2][LD_TE];
};
// the warp's part of level l's operator
template <int MODE, int KS>
__device__ __forceinline__ void lvl_operator(const PassArgs &A, int l, double (&a)[LvlTile<MODE, KS>::NRW][KS]) {
    constexpr int Q = 4 * KS, NRW = LvlTile<MODE, KS>::NRW;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int child = warp >> 1, rt0 = (warp & 1) * NRW;
    const double *op = A.ops + (size_t)l * A.stride + (MODE == 0 ? A.off_m2m : A.off_l2l);
#pragma unroll
    for (int i = 0; i < NRW; i++) {
        const int r = 8 * (rt0 + i) + g;
#pragma unroll
        for (int k = 0; k < KS; k++) {
            const int c = 4 * k + t;  // M2M: [4Q columns][Q rows]; L2L: [Q columns][4Q rows]
            a[i][k] = r < Q ? (MODE == 0 ? op[(size_t)(child * Q + c) * Q + r] : op[(size_t)c * 4 * Q + child * Q + r]) : 0.0;
        }
    }
}
// one tile (LD_TE entries) of level l by the whole block; wait: the previous
// kernel's results have not been waited for
template <int MODE, int KS>
__device__ __forceinline__ void lvl_tile(const PassArgs &A, int l, int64_t tile, int par, bool wait,
                                         const double (&a)[LvlTile<MODE, KS>::NRW][KS], LvlTile<MODE, KS> &S) {
    constexpr int Q = 4 * KS, NR = LvlTile<MODE, KS>::NR, NRW = LvlTile<MODE, KS>::NRW;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int child = warp >> 1, rt0 = (warp & 1) * NRW;
    const int64_t ne = A.T.ne[l], eoff = A.T.eoff[l], e0 = tile * LD_TE, en = e0 + g;
    // nodes of the tile's entries (tree data); L2L passes the X-list cells over
    int node = -1;
    if (en < ne && (MODE == 0 || !(A.ent[eoff + en] & 1))) node = A.ent_node[eoff + en];
    if (warp == 0 && t == 0) S.snode[par][g] = node;
    if (wait) pdl_wait();
    if (MODE == 1) __syncthreads();
    double acc[NRW][2], b[KS];
    const double *src = MODE == 0 ? A.uup + (size_t)(A.T.off[l + 1] + 4 * en + child) * Q : A.udown + (size_t)node * Q;
#pragma unroll
    for (int k = 0; k < KS; k++) b[k] = node >= 0 ? __ldcg(src + 4 * k + t) : 0.0;
#pragma unroll
    for (int i = 0; i < NRW; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int r = 8 * (rt0 + i) + g, n = 2 * t + j;
            acc[i][j] = 0.0;
            if (MODE == 1 && r < Q && S.snode[par][n] >= 0)
                acc[i][j] = __ldcg(A.udown + (size_t)(A.T.off[l + 1] + 4 * (e0 + n) + child) * Q + r);
        }
#pragma unroll
    for (int k = 0; k < KS; k++)
#pragma unroll
        for (int i = 0; i < NRW; i++) dmma_8x8x4(acc[i][0], acc[i][1], a[i][k], b[k]);
    if (MODE == 0) {
#pragma unroll
        for (int i = 0; i < NRW; i++)
            if (rt0 + i < NR) {
                S.red[par][child][2 * t][8 * (rt0 + i) + g] = acc[i][0];
                S.red[par][child][2 * t + 1][8 * (rt0 + i) + g] = acc[i][1];
            }
        __syncthreads();
        for (int i = tid; i < LD_TE * Q; i += LD_THREADS) {
            const int n = i / Q, r = i - n * Q, nd = S.snode[par][n];
            if (nd >= 0)
                A.uup[(size_t)nd * Q + r] =
                    (S.red[par][0][n][r] + S.red[par][1][n][r]) + (S.red[par][2][n][r] + S.red[par][3][n][r]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < NRW; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int r = 8 * (rt0 + i) + g, n = 2 * t + j;
                if (r < Q && S.snode[par][n] >= 0)
                    A.udown[(size_t)(A.T.off[l + 1] + 4 * (e0 + n) + child) * Q + r] = acc[i][j];
            }
    }
}
template <int MODE, int KS>
__global__ void __launch_bounds__(LD_THREADS) k_lvl_dmma(PassArgs A, int l) {
    __shared__ LvlTile<MODE, KS> S;
    const int64_t ntile = (A.T.ne[l] + LD_TE - 1) / LD_TE;
    double a[LvlTile<MODE, KS>::NRW][KS];
    lvl_operator<MODE, KS>(A, l, a);
    pdl_trigger();
    int par = 0;
    for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x, par ^= 1)
        lvl_tile<MODE, KS>(A, l, tile, par, tile == blockIdx.x, a, S);
}
// M2M of a run of consecutive small levels l0, l0 - 1, ... (count of them, at
// most LC_TILES tiles each) by one cluster: a barrier of the cluster takes the
// place of a launch between levels (2.9 us a level against 5.8 for five levels
// of 1k points, and one launch to issue).  The blocks exchange the levels'
// vectors through L2: stores before the barrier's release, reads past L1 after
// its acquire.  L2L levels, without the sum over children, take 2.6-3.0 us as
// launches of their own, the same as in a cluster.
constexpr int LC_BLOCKS = 8, LC_TILES = 16;
template <int KS>
__global__ void __launch_bounds__(LD_THREADS) k_m2m_chain(PassArgs A, int l0, int count) {
    constexpr int MODE = 0, NRW = LvlTile<MODE, KS>::NRW;
    constexpr bool AHEAD = NRW * KS <= 40;  // the next level's operator is loaded before the barrier (registers)
    __shared__ LvlTile<MODE, KS> S;
    int par = 0;
    double a[NRW][KS];
    lvl_operator<MODE, KS>(A, l0, a);
    pdl_trigger();
    for (int i = 0; i < count; i++) {
        const int l = l0 - i;
        const int64_t ntile = (A.T.ne[l] + LD_TE - 1) / LD_TE;
        for (int64_t tile = blockIdx.x; tile < ntile; tile += LC_BLOCKS, par ^= 1)
            lvl_tile<MODE, KS>(A, l, tile, par, i == 0 && tile == blockIdx.x, a, S);
        if (i == 0 && blockIdx.x >= ntile) pdl_wait();
        if (i + 1 == count) break;
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        if (AHEAD) lvl_operator<MODE, KS>(A, l - 1, a);
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (!AHEAD) lvl_operator<MODE, KS>(A, l - 1, a);
    }
}
template <int MODE, int KS>
static void launch_lvl_dmma(kifmm_plan *P, const PassArgs &A, int l) {
    if constexpr (KS > 1)
        if (4 * KS != P->Q) return launch_lvl_dmma<MODE, KS - 1>(P, A, l);
    // past four blocks per SM a block takes several tiles: the operator is read once
    const int64_t tiles = (P->lt.ne[l] + LD_TE - 1) / LD_TE;
    launch_pdl(k_lvl_dmma<MODE, KS>, dim3((unsigned)std::min<int64_t>(tiles, (int64_t)P->num_sms * 4)), dim3(LD_THREADS),
               0, P->stream, A, l);
}
template <int KS>
static void launch_m2m_chain(kifmm_plan *P, const PassArgs &A, int l, int count) {
    if constexpr (KS > 1)
        if (4 * KS != P->Q) return launch_m2m_chain<KS - 1>(P, A, l, count);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(LC_BLOCKS);
    cfg.blockDim = dim3(LD_THREADS);
    cfg.stream = P->stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = LC_BLOCKS;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    KIFMM_CUDA(cudaLaunchKernelEx(&cfg, k_m2m_chain<KS>, A, l, count));
    KIFMM_LAUNCHED();
}

// NT columns per block: (ceil(M/4)) x (NT/4) threads <= 256 and at most
// 200 KB of shared memory
static int lvl_gemm_nt(int M, int K) {
    int tm = (M + 3) / 4;
    int nt = (256 / tm) * 4;
    if (nt > 32) nt = 32;  // more blocks per level: the levels are small
    int cap = (int)(((200 << 10) / 8 - (int64_t)K * M) / (K + 1)) / 4 * 4;
    if (nt > cap) nt = cap;
    return nt < 4 ? 4 : nt;
}

template <int MODE>
static void launch_lvl_gemm(kifmm_plan *P, const PassArgs &A, int l) {
    const int Q = P->Q;
    const int M = MODE == 0 ? Q : 4 * Q, K = MODE == 0 ? 4 * Q : Q;
    const int64_t ne = P->lt.ne[l];
    {  // broadcast form when the operator and the entry tile fit in shared memory
        constexpr int RPT = MODE == 0 ? 8 : 16;
        const int RG = (M + RPT - 1) / RPT, Mp = RG * RPT;
        const int wps = RG < 8 ? RG : 8, NT = 32 * (8 / wps);
        const size_t smem = ((size_t)K * Mp + (size_t)NT * (K + 1)) * sizeof(double);
        if (smem <= (size_t)(220 << 10)) {
            ensure_dyn_smem(k_lvl_gemm_b<MODE, RPT>, smem);
            k_lvl_gemm_b<MODE, RPT><<<(unsigned)((ne + NT - 1) / NT), LG_THREADS, smem, P->stream>>>(A, l, M, K, Mp,
                                                                                                     NT);
            KIFMM_LAUNCHED();
            return;
        }
    }
    int nt = lvl_gemm_nt(M, K);
    int threads = ((M + 3) / 4) * (nt / 4);
    size_t smem = ((size_t)K * M + (size_t)nt * (K + 1)) * sizeof(double);
    ensure_dyn_smem(k_lvl_gemm_d<MODE>, smem);
    k_lvl_gemm_d<MODE><<<(unsigned)((ne + nt - 1) / nt), threads, smem, P->stream>>>(A, l, M, K, nt);
    KIFMM_LAUNCHED();
}

// The upward M2M over levels L-2 .. 2 and the downward L2L over 2 .. L-2: on the
// FP64 tensor path for Nequiv a multiple of four (up to 64), with runs of small
// M2M levels in one launch.
void run_m2m_levels(kifmm_plan *P, const PassArgs &A) {
    for (int l = P->L - 2, count; l >= 2; l -= count) {
        count = 0;
        while (l - count >= 2 && P->lt.ne[l - count] > 0 && P->lt.ne[l - count] <= LC_TILES * LD_TE) count++;
        if (P->Q % 4 == 0 && count > 1) {
            launch_m2m_chain<16>(P, A, l, count);
            continue;
        }
        count = 1;
        if (!P->lt.ne[l]) continue;
        if (P->Q % 4 == 0) launch_lvl_dmma<0, 16>(P, A, l);
        else launch_lvl_gemm<0>(P, A, l);
    }
}
void run_l2l_levels(kifmm_plan *P, const PassArgs &A) {
    for (int l = 2; l <= P->L - 2; l++) {
        if (!P->lt.ne[l]) continue;
        if (P->Q % 4 == 0) launch_lvl_dmma<1, 16>(P, A, l);
        else launch_lvl_gemm<1>(P, A, l);
    }
}

// Buffers of an apply, its cleared flags and expansions, and the densities in
// tree order.
void apply_prologue(kifmm_plan *P) {
    cudaStream_t s = P->stream;
    const int Q = P->Q;
    int64_t n = P->N, NN = P->n_nodes;
    const int64_t vw = P->cplx ? 2 : 1;  // doubles per density value
    P->taus.alloc(n * vw);
    P->pots.alloc(n * vw);
    P->uup.alloc((size_t)NN * Q);
    P->udown.alloc((size_t)NN * Q);
    // Expansions start at zero, once per tree: every apply writes the same nodes'
    // (P2M the leaves with points, M2M the entries, M2L every child of a split
    // entry), and the others stay zero.
    if (!P->exp_zeroed) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        KIFMM_CUDA(cudaStreamIsCapturing(s, &cap));
        KIFMM_CUDA(cudaMemsetAsync(P->uup.p, 0, (size_t)NN * Q * sizeof(double), s));
        KIFMM_CUDA(cudaMemsetAsync(P->udown.p, 0, (size_t)NN * Q * sizeof(double), s));
        P->exp_zeroed = cap == cudaStreamCaptureStatusNone;  // (captured: they run with the graph)
    }
    if (P->opt.planned) {
        ops_wait_now(P);
        build_plan_matrices(P);  // first apply after build_tree / precompute
    }
    ops_wait_circles(P);  // the P2M's check points
    if (P->cplx)
        launch_gather_tau_c(P);
    else
        launch_pdl(k_gather_tau, dim3(grid_for(n, 256, P->num_sms * 8)), dim3(256), 0, s, P->tau_src,
                   (const int32_t *)P->perm.p, n, P->taus.p, P->scal.p + KIFMM_SCAL_PASS_ERR,
                   KIFMM_SCAL_WORDS - KIFMM_SCAL_PASS_ERR);
}

void run_upward_downward(kifmm_plan *P) {
    const int Q = P->Q, L = P->L;
    near_join(P);  // the previous apply's near-field pass, if never evaluated
    apply_prologue(P);
    if (P->opt.precision == KIFMM_PREC_MIXED) {
        run_passes_mixed(P);
        ops_wait_now(P);  // (L < 3: the evaluation reads them)
        return;
    }
    if (L < 3) {  // no level has well-separated boxes
        ops_wait_now(P);
        return;
    }
    // a planned near field (bound by HBM) beside the chain, as the mixed apply's
    const bool near = planned_ready(P) && near_possible(P), early = near && near_split(P);
    if (early) near_fork(P);
    HighPriorityFork fork(P, near && !early);
    PassArgs A = make_pass_args(P);
    if (P->n_p2m_list) {
        PhaseScope ph(P, KIFMM_PHASE_P2M);
        if (planned_ready(P)) launch_planned_p2m(P, A);
        else launch_p2m_d(P, A);
    }
    ops_wait_now(P);  // the P2M reads only the check circles
    {
        PhaseScope ph_m2m(P, KIFMM_PHASE_M2M);
        run_m2m_levels(P, A);
    }
    if (near && !early) near_fork(P);
    if (m2l_uses_dmma(P)) {
        // FP64 tensor path: all levels' M2L in one launch, then the L2L chain
        {
            PhaseScope ph(P, KIFMM_PHASE_M2L);
            launch_m2l_dmma(P, A, 1, L - 2);
        }
        PhaseScope ph(P, KIFMM_PHASE_L2L);
        run_l2l_levels(P, A);
        return;
    }
    PhaseScope ph(P, KIFMM_PHASE_M2L);
    int thr = ((4 * Q + 31) / 32) * 32;
    size_t smem = (size_t)M2L_TE * 4 * Q * sizeof(double);
    ensure_dyn_smem(k_m2l_d, smem);
    for (int l = 1; l <= L - 2; l++) {
        int64_t ne = P->lt.ne[l];
        if (!ne) continue;
        k_m2l_d<<<(unsigned)((ne + M2L_TE - 1) / M2L_TE), thr, smem, P->stream>>>(A, l);  // (maybe the far stream)
        KIFMM_LAUNCHED();
    }
}

// potentials from tree order to the caller's order
void launch_scatter_pot(kifmm_plan *P, double *pot) {
    const int64_t n = P->N;
    launch_pdl(k_scatter_pot, dim3(grid_for(n, 256, P->num_sms * 8)), dim3(256), 0, P->stream,
               (const double *)P->pots.p, (const int32_t *)P->perm.p, n, pot);
}

// Potentials at the sources into pot (device, caller's order).  The FP64 and
// the planned leaf passes write them there themselves.
void run_eval_sources(kifmm_plan *P, int check_self, double *pot) {
    PassArgs A = make_pass_args(P);
    A.out = pot;
    A.perm = P->perm.p;
    const bool planned = check_self && planned_ready(P);
    if (!planned && planned_ready(P)) near_join(P);  // (a planned near field is not the one asked for)
    if (!planned && P->opt.precision == KIFMM_PREC_MIXED) {
        run_eval_sources_mixed(P, A, check_self);
        return;
    }
    if (!P->n_leaf_list) return;
    PhaseScope ph(P, KIFMM_PHASE_LEAF);
    if (planned) run_planned_leaf(P, A);
    else launch_leaf_eval_d(P, A, check_self);
}

// ------------------------------------------------ kernel-function utilities
// KAS restricted to targets (class_fmm.py:134-143): one block per target.
__global__ void k_direct_d(int kind, double k, const double *__restrict__ x, const double *__restrict__ y,
                           const double *__restrict__ tau, int64_t n, const int64_t *__restrict__ tg,
                           double *__restrict__ out) {
    __shared__ double red[32];
    int64_t j = tg[blockIdx.x];
    if (j < 0 || j >= n) {  // caller index out of range: report NaN, touch nothing
        if (threadIdx.x == 0) out[blockIdx.x] = __longlong_as_double(0x7ff8000000000000ll);
        return;
    }
    double px = x[j], py = y[j], acc = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        if (i == j) continue;
        double dx = px - x[i], dy = py - y[i];
        acc += green_d(kind, k, dx * dx + dy * dy) * tau[i];
    }
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) out[blockIdx.x] = v;
    }
}

__global__ void k_kmatrix_d(int kind, double k, const double *sx, const double *sy, int64_t ns, const double *tx,
                            const double *ty, int64_t nt, double *out) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ns * nt; e += (int64_t)gridDim.x * blockDim.x) {
        int64_t j = e / ns, i = e % ns;
        double dx = tx[j] - sx[i], dy = ty[j] - sy[i];
        out[e] = green_d(kind, k, dx * dx + dy * dy);
    }
}

__global__ void k_kapply_d(int kind, double k, const double *sx, const double *sy, int64_t ns, const double *tx,
                           const double *ty, int64_t nt, const double *tau, double *out) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nt; j += (int64_t)gridDim.x * blockDim.x) {
        double acc = 0.0;
        for (int64_t i = 0; i < ns; i++) {
            double dx = tx[j] - sx[i], dy = ty[j] - sy[i];
            acc += green_d(kind, k, dx * dx + dy * dy) * tau[i];
        }
        out[j] = acc;
    }
}

void direct_sum_device_c(const kifmm_kernel &kn, const double *x, const double *y, const double *tau, int64_t n,
                         const int64_t *tg, int64_t nt, double *out, cudaStream_t s);
void kernel_matrix_device_c(const kifmm_kernel &kn, const double *sx, const double *sy, int64_t ns, const double *tx,
                            const double *ty, int64_t nt, double *out, cudaStream_t s);
void kernel_apply_device_c(const kifmm_kernel &kn, const double *sx, const double *sy, int64_t ns, const double *tx,
                           const double *ty, int64_t nt, const double *tau, double *out, cudaStream_t s);

void direct_sum_device(const kifmm_kernel &kn, const double *x, const double *y, const double *tau, int64_t n,
                       const int64_t *tg, int64_t nt, double *out, cudaStream_t s) {
    if (kn.kind == KIFMM_KERNEL_HELMHOLTZ) return direct_sum_device_c(kn, x, y, tau, n, tg, nt, out, s);
    if (nt <= 0) return;
    KIFMM_REQUIRE(nt < (1ll << 31), KIFMM_ERR_ARG, "direct_sum: too many targets");
    k_direct_d<<<(unsigned)nt, 256, 0, s>>>(kn.kind, kn.k, x, y, tau, n, tg, out);
    KIFMM_LAUNCHED();
}

void kernel_matrix_device(const kifmm_kernel &kn, const double *sx, const double *sy, int64_t ns, const double *tx,
                          const double *ty, int64_t nt, double *out, cudaStream_t s) {
    if (kn.kind == KIFMM_KERNEL_HELMHOLTZ) return kernel_matrix_device_c(kn, sx, sy, ns, tx, ty, nt, out, s);
    if (ns * nt <= 0) return;
    k_kmatrix_d<<<grid_for(ns * nt, 256, 8192), 256, 0, s>>>(kn.kind, kn.k, sx, sy, ns, tx, ty, nt, out);
    KIFMM_LAUNCHED();
}

void kernel_apply_device(const kifmm_kernel &kn, const double *sx, const double *sy, int64_t ns, const double *tx,
                         const double *ty, int64_t nt, const double *tau, double *out, cudaStream_t s) {
    if (kn.kind == KIFMM_KERNEL_HELMHOLTZ) return kernel_apply_device_c(kn, sx, sy, ns, tx, ty, nt, tau, out, s);
    if (nt <= 0) return;
    k_kapply_d<<<grid_for(nt, 128, 8192), 128, 0, s>>>(kn.kind, kn.k, sx, sy, ns, tx, ty, nt, tau, out);
    KIFMM_LAUNCHED();
}

}  // namespace kifmm
