// passes_mixed.cu -- mixed-precision passes.
//
// Same algorithm as passes.cu (reference class_fmm.py:299-399) with
//   * P2P in FP32 on coordinates relative to the box centre (FP64
//     subtraction, then rounding: nearby points keep their relative precision
//     wherever the box sits, as the reference's L2P does with tx = x - xmid,
//     class_fmm.py:81-82);
//   * P2M and L2P in FP64: their terms are weighted by equivalent densities
//     of alternating sign, and FP32 logs there cost ~1.6e-7 each at 1M points
//     (measured), while they are only Q evaluations per point;
//   * check potentials u_up / u_down kept in FP64, M2M and L2L in FP64 (a few
//     percent of the work);
//   * M2L on the tensor cores (m2l_tc.cu): int8 slices with exact int32
//     accumulation (default), or bf16 / fp16 hi-lo splits with FP32
//     accumulation; or FP32 tiles on the CUDA cores (this file);
//   * the local expansion's equivalent density Inv_l u_down formed in FP64.
// Coincident source/target pairs contribute zero, as in the reference.
#include "leaf_f32.cuh"
#include "passes.cuh"

namespace kifmm {

constexpr float LN2_OVER_4PI = 0.05515890934390497f;   // ln 2 / (4 pi)
constexpr float INV_2PI_F = 0.15915494309189535f;

// scale of the near sums: Laplace sums log2(r^2)
template <int KIND>
__device__ __forceinline__ float gsum_scale() {
    return KIND == KIFMM_KERNEL_LAPLACE ? -LN2_OVER_4PI : INV_2PI_F;
}

// FP32 M2L + L2L on the CUDA cores (FP64 state in and out): block = 4Q rows x
// TE target groups.
constexpr int M2LF_TE = 32;
__global__ void k_m2l_f(PassArgs A, int l) {
    extern __shared__ float smf[];
    const int Q = A.Q, Q4 = 4 * Q, r = threadIdx.x;
    float *src = smf;  // [TE][4Q]
    __shared__ int64_t sgrp[M2LF_TE];
    __shared__ int spar[M2LF_TE];
    __shared__ int64_t schild[M2LF_TE];
    const int64_t e0 = (int64_t)blockIdx.x * M2LF_TE;
    const int64_t ne = A.T.ne[l];
    if (r < M2LF_TE) {
        int64_t e = e0 + r;
        bool act = e < ne && !(A.ent[A.T.eoff[l] + e] & 1);
        spar[r] = act ? A.ent_node[A.T.eoff[l] + e] : -1;
        schild[r] = act ? A.T.off[l + 1] + 4 * e : -1;
    }
    __syncthreads();
    float acc[M2LF_TE];
#pragma unroll
    for (int t = 0; t < M2LF_TE; t++) acc[t] = 0.f;
    const float *opl = A.ops_f + (size_t)(l + 1) * A.stride + A.off_m2l;
    for (int d = 0; d < 9; d++) {
        if (d == 4) continue;
        if (r < M2LF_TE) {
            int p = spar[r];
            int64_t grp = -1;
            if (p >= 0) {
                const int je = m2l_source_entry(A.ncoll, A.nent, A.nbot, A.ntop, p, d);
                if (je >= 0) grp = A.T.off[l + 1] + 4 * (je - A.T.eoff[l]);
            }
            sgrp[r] = grp;
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < M2LF_TE * Q4; idx += blockDim.x) {
            int t = idx / Q4, c = idx % Q4;
            int64_t grp = sgrp[t];
            src[idx] = grp >= 0 ? (float)A.uup[(size_t)grp * Q + c] : 0.f;
        }
        __syncthreads();
        const float *op = opl + (size_t)d * Q4 * Q4;
        if (r < Q4)
            for (int c = 0; c < Q4; c++) {
                float a = op[(size_t)c * Q4 + r];
#pragma unroll
                for (int t = 0; t < M2LF_TE; t++) acc[t] = fmaf(a, src[t * Q4 + c], acc[t]);
            }
        __syncthreads();
    }
    if (l >= 2) {
        for (int idx = threadIdx.x; idx < M2LF_TE * Q; idx += blockDim.x) {
            int t = idx / Q, c = idx % Q;
            int p = spar[t];
            src[idx] = p >= 0 ? (float)A.udown[(size_t)p * Q + c] : 0.f;
        }
        __syncthreads();
        const float *op = A.ops_f + (size_t)l * A.stride + A.off_l2l;
        if (r < Q4)
            for (int c = 0; c < Q; c++) {
                float a = op[(size_t)c * Q4 + r];
#pragma unroll
                for (int t = 0; t < M2LF_TE; t++) acc[t] = fmaf(a, src[t * Q + c], acc[t]);
            }
    }
    if (r < Q4)
#pragma unroll
        for (int t = 0; t < M2LF_TE; t++)
            if (schild[t] >= 0) A.udown[(size_t)schild[t] * Q + r] = (double)acc[t];
}

// Taylor coefficients of every leaf's local expansion (Laplace, levels >= 2),
// FP64 on the tensor path: C[R x leaves] = Taylor_l[R x Q] . u_down[Q x leaves],
// one block per 32 consecutive leaves of one level (leaf_list is level-major).
// Warp w computes all R rows (MTR 8-row tiles) for leaves 8w..8w+7; the block
// writes its 32 x R coefficients as one contiguous run.
struct TaylorArgs {
    PassArgs A;
    const int32_t *list;
    double *coef;
    const double *den;  // [leaf_list index][Q] densities, null where no point lies outside the root box
    int lmin, lmax;
    int64_t loff[MAX_LEVELS + 1];  // leaf_list range of each level
    int64_t toff[MAX_LEVELS + 1];  // first block of each level
};
constexpr int TY_THREADS = 128;
constexpr int TY_R = 2 * KIFMM_TAYLOR_P + 1, TY_MTR = (TY_R + 7) / 8;
__global__ void __launch_bounds__(TY_THREADS) k_leaf_taylor(TaylorArgs T) {
    extern __shared__ __align__(16) double sm_ty[];
    const PassArgs &A = T.A;
    const int Q = A.Q, R = TY_R, ldt = pad4mod16(8 * TY_MTR), ldx = pad4mod16(Q);
    double *tS = sm_ty;                      // [Q][ldt]: element (row r, col k) at k * ldt + r
    double *xS = tS + (size_t)Q * ldt;       // [32 leaves][ldx]
    double *cS = xS + 32 * (size_t)ldx;      // [32 leaves][R]
    pdl_trigger();
    const int64_t b = blockIdx.x;
    int l = T.lmin;
    while (l < T.lmax && T.toff[l + 1] <= b) l++;
    const int64_t w0 = T.loff[l] + (b - T.toff[l]) * 32;
    const int nt = (int)min((int64_t)32, T.loff[l + 1] - w0);
    const int tid = threadIdx.x;
    // the level's map (precomputed, independent of the previous kernel), rows padded with zeros
    const double *tl = A.taylor + (size_t)l * Q * R;
    for (int i0 = tid; i0 < Q * ldt; i0 += 4 * TY_THREADS) {
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int i = i0 + q * TY_THREADS, k = i / ldt, r = i - k * ldt;
            v[q] = (i < Q * ldt && r < R) ? tl[(size_t)k * R + r] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int i = i0 + q * TY_THREADS;
            if (i < Q * ldt) tS[i] = v[q];
        }
    }
    pdl_wait();  // u_down comes from the L2L chain
    for (int i0 = tid; i0 < 32 * Q; i0 += 4 * TY_THREADS) {
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int i = i0 + q * TY_THREADS, n = i / Q, k = i - n * Q;
            v[q] = (i < 32 * Q && n < nt) ? A.udown[(size_t)T.list[w0 + n] * Q + k] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int i = i0 + q * TY_THREADS, n = i / Q, k = i - n * Q;
            if (i < 32 * Q) xS[n * ldx + k] = v[q];
        }
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, n0 = warp * 8;
    if (n0 < nt) {
        double acc[TY_MTR][2];
#pragma unroll
        for (int i = 0; i < TY_MTR; i++) acc[i][0] = acc[i][1] = 0.0;
        const double *xb = xS + (size_t)(n0 + g) * ldx + t;
        const double *ab = tS + (size_t)t * ldt + g;
        for (int k0 = 0; k0 < Q; k0 += 4) {
            const double bv = xb[k0];
#pragma unroll
            for (int i = 0; i < TY_MTR; i++) dmma_8x8x4(acc[i][0], acc[i][1], ab[(size_t)k0 * ldt + 8 * i], bv);
        }
#pragma unroll
        for (int i = 0; i < TY_MTR; i++) {
            const int r = 8 * i + g;
            if (r < R) {
                cS[(n0 + 2 * t) * R + r] = acc[i][0];
                cS[(n0 + 2 * t + 1) * R + r] = acc[i][1];
            }
        }
    }
    __syncthreads();
    double *out = T.coef + (size_t)w0 * R;
    for (int i = tid; i < nt * R; i += TY_THREADS) out[i] = cS[i];
}

// L2P + P2P: one warp per target leaf.  The sources of the leaf and its eight
// colleagues are staged in shared memory as one list (the leaf's own points
// first), in chunks of LEAF_CHUNK.  A tile of nt <= 32 targets is spread over
// the warp in ng groups (two targets per lane for the Laplace kernel, one
// otherwise) with sp = 32 / ng lanes per group, each lane taking every sp-th
// source, so a leaf of 15 points keeps 32 lanes busy and no lane idles on a
// short colleague; the Laplace pair loop runs on packed FP32 pairs (f32x2),
// one instruction for both of a lane's targets.  For the Laplace kernel the
// offsets are scaled by 1/w (w the leaf width) so every log2 term is O(1); the
// remainder log2(w^2) * sum(tau) is added in FP64.  The inner loop is
// branch-free: r^2 is floored at FLT_MIN (r^2 + FLT_MIN) and short chunks are
// padded with far, uncharged sources.  The pairs inside the leaf itself that
// meet the floor (the target's own point and exact duplicates, which the
// reference skips, class_fmm.py:107) are counted in the first passes, over
// the leaf's own points, and taken back out.  Distinct points of different
// leaves closer than about 2^-24 leaf widths round to the same FP32 offsets
// and keep log2(FLT_MIN) for their pair; the FP64 near field (near_fp64)
// resolves such pairs.  FP32 partial sums of at most 32 terms are accumulated
// in FP64.
// one warp per block: leaves differ in work by more than 10x, and a block of
// several warps would hold its SM slot until its slowest warp is done
constexpr int LEAF_WARPS = 1;
// 32 one-warp blocks per SM (64 registers) with 96-source chunks measured 2%
// faster than 28 blocks (72 registers) with 128-source chunks on the 1M
// mixture (0.240 against 0.244 ms), and those 8% faster than 20 blocks (96
// registers) with 256-source chunks; shared memory per block sets the ceiling
#ifndef KIFMM_LEAF_BLOCKS_PER_SM
#define KIFMM_LEAF_BLOCKS_PER_SM 32
#endif
#ifndef KIFMM_LEAF_CHUNK
#define KIFMM_LEAF_CHUNK 96
#endif
constexpr int LEAF_BLOCKS_PER_SM = KIFMM_LEAF_BLOCKS_PER_SM;  // resident blocks per SM at the register bound
constexpr int LEAF_CHUNK = KIFMM_LEAF_CHUNK;                  // sources staged per pass
static_assert(LEAF_CHUNK + 31 <= 200, "the leaf kernel's quotients (small_div) need cn + sp - 1 <= 200");

constexpr f32x2 F2_FLOOR = 0x0080000000800000ull;  // (FLT_MIN, FLT_MIN)
// r^2 + FLT_MIN of both targets to one source: the floor rides in the multiply-add
// instead of a separate clamp.  Every pair of distinct points has r^2 >= 2^-48
// (scaled FP32 offsets of O(1)), where adding 2^-126 changes nothing; coincident
// points give FLT_MIN exactly, as a clamp does.
__device__ __forceinline__ f32x2 pair2_r2_floor(f32x2 tx, f32x2 ty, const ulonglong2 &s) {
    const f32x2 dx = f2_sub(tx, s.x), dy = f2_sub(ty, s.y);
    return f2_fma(dx, dx, f2_fma(dy, dy, F2_FLOOR));
}
// Laplace pair sums of one lane holding two targets (tx, ty packed): over its
// sources at list positions j + k SP, k in [k0, k1), of z log2(r^2 + FLT_MIN),
// in FP32 blocks of at most 32 sources (two chains per target, alternating
// sources) added to na, nb in FP64.  OWN: the positions are the leaf's own
// points below en, where coincident pairs (the target itself, duplicates) meet
// the floor; their charges are summed into exa, exb to be taken out.  SP is a
// template argument so that the strided shared-memory loads take immediate
// offsets.
template <int SP_, bool OWN>
__device__ __forceinline__ void leaf_pairs2(const ulonglong2 *__restrict__ sxy, const f32x2 *__restrict__ sz, int j,
                                            int k0, int k1, f32x2 tx, f32x2 ty, int en, double &na, double &nb,
                                            float &exa, float &exb, int sp_rt = 0) {
    constexpr float FLOOR2 = 2.0f * 1.17549435e-38f;
    const int SP = SP_ ? SP_ : sp_rt;
    for (int kb = k0; kb < k1; kb += 32) {
        const int ke = min(k1, kb + 32);
        f32x2 acc0 = 0ull, acc1 = 0ull;
        const ulonglong2 *p = sxy + j + kb * SP;
        const f32x2 *q = sz + j + kb * SP;
        int k = kb;
        if (OWN) {
            for (; k < ke; k++, p += SP, q += SP) {
                const f32x2 r = pair2_r2_floor(tx, ty, *p), z = *q;
                acc0 = f2_fma(z, lg2_pair(r), acc0);
                float ra, rb, zs, zu;
                f2_unpack(r, ra, rb);
                f2_unpack(z, zs, zu);
                const bool in = j + k * SP < en;
                exa += (in && ra < FLOOR2) ? zs : 0.f;
                exb += (in && rb < FLOOR2) ? zs : 0.f;
            }
        } else {
#pragma unroll 1
            for (; k + 3 < ke; k += 4, p += 4 * SP, q += 4 * SP) {
                const ulonglong2 s0 = p[0], s1 = p[SP], s2 = p[2 * SP], s3 = p[3 * SP];
                const f32x2 z0 = q[0], z1 = q[SP], z2 = q[2 * SP], z3 = q[3 * SP];
                acc0 = f2_fma(z0, lg2_pair(pair2_r2_floor(tx, ty, s0)), acc0);
                acc1 = f2_fma(z1, lg2_pair(pair2_r2_floor(tx, ty, s1)), acc1);
                acc0 = f2_fma(z2, lg2_pair(pair2_r2_floor(tx, ty, s2)), acc0);
                acc1 = f2_fma(z3, lg2_pair(pair2_r2_floor(tx, ty, s3)), acc1);
            }
            for (; k + 1 < ke; k += 2, p += 2 * SP, q += 2 * SP) {
                acc0 = f2_fma(q[0], lg2_pair(pair2_r2_floor(tx, ty, p[0])), acc0);
                acc1 = f2_fma(q[SP], lg2_pair(pair2_r2_floor(tx, ty, p[SP])), acc1);
            }
            if (k < ke) acc0 = f2_fma(q[0], lg2_pair(pair2_r2_floor(tx, ty, p[0])), acc0);
        }
        float sa, sb;
        f2_unpack(f2_add(acc0, acc1), sa, sb);
        na += (double)sa;
        nb += (double)sb;
    }
}
// leaf_pairs2 for a run-time lane stride sp = 32 / groups, groups in 1..16
template <bool OWN>
__device__ __forceinline__ void leaf_pairs2_sp(int sp, const ulonglong2 *sxy, const f32x2 *sz, int j, int k0, int k1,
                                               f32x2 tx, f32x2 ty, int en, double &na, double &nb, float &exa,
                                               float &exb) {
#define KIFMM_LEAF_SP(S)                                                          \
    case S:                                                                       \
        leaf_pairs2<S, OWN>(sxy, sz, j, k0, k1, tx, ty, en, na, nb, exa, exb); \
        break;
#ifndef KIFMM_LEAF_SP_MODE
#define KIFMM_LEAF_SP_MODE 1
#endif
#if KIFMM_LEAF_SP_MODE == 0
    leaf_pairs2<0, OWN>(sxy, sz, j, k0, k1, tx, ty, en, na, nb, exa, exb, sp);
#elif KIFMM_LEAF_SP_MODE == 1
    if (sp == 2) leaf_pairs2<2, OWN>(sxy, sz, j, k0, k1, tx, ty, en, na, nb, exa, exb);
    else leaf_pairs2<0, OWN>(sxy, sz, j, k0, k1, tx, ty, en, na, nb, exa, exb, sp);
#else
    switch (sp) {
        KIFMM_LEAF_SP(2)
        KIFMM_LEAF_SP(3)
        KIFMM_LEAF_SP(4)
        KIFMM_LEAF_SP(5)
        KIFMM_LEAF_SP(6)
        KIFMM_LEAF_SP(8)
        KIFMM_LEAF_SP(10)
        KIFMM_LEAF_SP(16)
        default:
            leaf_pairs2<32, OWN>(sxy, sz, j, k0, k1, tx, ty, en, na, nb, exa, exb);
    }
#endif
#undef KIFMM_LEAF_SP
}

// K0 of two pairs of one target in packed FP32, for 0 < x <= 2 on both sides: the
// operations of k0_f, in its order, so that the values are the same to the bit.
// The square root of r^2 is one Newton step on the reciprocal square root
// (s = r^2 y, s + (r^2 - s^2) y / 2), equal to sqrtf for every FP32 mantissa
// (checked over all 2^24 of [1, 4); r^2 is held above 2^-80 so that nothing
// underflows).  The logarithms stay the math library's.
__device__ __forceinline__ f32x2 f2_dup(float a) { return f2_pack(a, a); }
__device__ __forceinline__ f32x2 k0_pair_x(f32x2 r2, f32x2 kk) {
    float ra, rb, ya, yb;
    f2_unpack(r2, ra, rb);
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(ya) : "f"(ra));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yb) : "f"(rb));
    const f32x2 y = f2_pack(ya, yb), s = f2_mul(r2, y), e = f2_fma(s ^ 0x8000000080000000ull, s, r2);
    return f2_mul(kk, f2_fma(e, f2_mul(y, f2_dup(0.5f)), s));
}
__device__ __forceinline__ f32x2 k0_pair(f32x2 x) {
    const f32x2 t = f2_mul(x, x);
    f32x2 a = f2_dup(K0_I0_F[K0_I0_F_N - 1]), b = f2_dup(K0_P_F[K0_P_F_N - 1]);
#pragma unroll
    for (int i = K0_I0_F_N - 2; i >= 0; i--) a = f2_fma(a, t, f2_dup(K0_I0_F[i]));
#pragma unroll
    for (int i = K0_P_F_N - 2; i >= 0; i--) b = f2_fma(b, t, f2_dup(K0_P_F[i]));
    float ha, hb;
    f2_unpack(f2_mul(x, f2_dup(0.5f)), ha, hb);
    return f2_fma(f2_pack(-logf(ha), -logf(hb)), a, b);
}
// K0 pair sums of one lane's target over its sources at list positions j + k
// sp, k in [0, it), in FP32 blocks of 32 added to `near` in FP64.  Two sources
// at a time: every value a packed instruction's half, the sum still one after
// the other.  Position it (past the end) is an uncharged pad.  Bound by issue
// (81%) and the FMA pipe (59%), a third of both the logarithms': 2M points, k 5,
// 4.3e8 pairs: 1.18 ms, 1.43 one source at a time.
__device__ __forceinline__ void leaf_pairs_k0(const float *__restrict__ sx, const float *__restrict__ sy,
                                              const float *__restrict__ sz, int j, int sp, int it, float tx, float ty,
                                              float kk, double &near) {
    const f32x2 tx2 = f2_dup(tx), ty2 = f2_dup(ty), kk2 = f2_dup(kk);
    for (int kb = 0; kb < it; kb += 32) {
        const int ke = min(it, kb + 32);
        float acc = 0.f;
#pragma unroll 1
        for (int k = kb; k < ke; k += 2) {
            const int u = j + k * sp, v = u + sp;
            const f32x2 dx = f2_sub(tx2, f2_pack(sx[u], sx[v])), dy = f2_sub(ty2, f2_pack(sy[u], sy[v]));
            const f32x2 r2 = f2_fma(dx, dx, f2_mul(dy, dy)), x = k0_pair_x(r2, kk2);
            const float za = sz[u], zb = sz[v];
            float ra, rb, xa, xb;
            f2_unpack(r2, ra, rb);
            f2_unpack(x, xa, xb);
            if (ra >= 0x1p-80f && rb >= 0x1p-80f && xa <= 2.f && xb <= 2.f) {
                float ga, gb;
                f2_unpack(k0_pair(x), ga, gb);
                acc = fmaf(za, ga, acc);
                acc = fmaf(zb, gb, acc);
            } else {  // the target itself, far pairs, not-a-number
                if (ra > 0.f) acc = fmaf(za, k0_f(kk * sqrtf(ra)), acc);
                if (rb > 0.f) acc = fmaf(zb, k0_f(kk * sqrtf(rb)), acc);
            }
        }
        near += (double)acc;
    }
}

// x / d for 0 <= x <= 200 and 1 <= d <= 32 as a multiply and a shift (the
// lane-layout quotients of the leaf kernel; a division by a run-time value
// costs a reciprocal and a dozen fix-up instructions): c = ceil(2^16 / d)
// gives floor(x c / 2^16) = floor(x / d) whenever x < 2^16 / d.
__constant__ unsigned c_recip16[33] = {
    0,    65536, 32768, 21846, 16384, 13108, 10923, 9363, 8192, 7282, 6554, 5958, 5462, 5042, 4682, 4370, 4096,
    3856, 3641,  3450,  3277,  3121,  2979,  2850,  2731, 2622, 2521, 2428, 2341, 2260, 2185, 2115, 2048};
__device__ __forceinline__ int small_div(int x, int d) { return (int)(((unsigned)x * c_recip16[d]) >> 16); }

// the P2P of leaf w of A's leaf list, by one warp: its 32-target tiles [tile0,
// tile1) (all of them by default), into pots
template <int KIND>
__device__ __forceinline__ void leaf_near_f(const PassArgs &A, int64_t w, int tile0 = 0, int tile1 = 1 << 20) {
    constexpr float CLAMP = 1.17549435e-38f;  // FLT_MIN
    constexpr bool LAP = KIND == KIFMM_KERNEL_LAPLACE;
    // Laplace: (x, x | y, y) and (z, z) per staged source; K0: x, y, z apart
    __shared__ ulonglong2 sxys[LAP ? LEAF_WARPS : 1][LAP ? LEAF_CHUNK + 32 : 1];
    __shared__ f32x2 szs[LAP ? LEAF_WARPS : 1][LAP ? LEAF_CHUNK + 32 : 1];
    __shared__ float sks[LAP ? 1 : LEAF_WARPS][3][LAP ? 1 : LEAF_CHUNK + 64];
    __shared__ double red[LEAF_WARPS][2][32];
    __shared__ float redf[LEAF_WARPS][2][32];
    __shared__ int rngs[LEAF_WARPS][18];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    {
        // the leaf record: node, level, point range, cell key and source ranges
        // in one coalesced load (list[w] is the record's node)
        const int rv = A.leaf_rec[w * LEAF_REC_WORDS + lane];
        const int l = __shfl_sync(0xffffffffu, rv, LR_LEVEL);
        const uint64_t key = (uint64_t)(uint32_t)__shfl_sync(0xffffffffu, rv, LR_KEY_LO) |
                             ((uint64_t)(uint32_t)__shfl_sync(0xffffffffu, rv, LR_KEY_HI) << 32);
        double cx, cy;
        {
            const double wl = ldexp(A.W, -l);
            cx = A.root + ((double)compact2(key >> 1) + 0.5) * wl;
            cy = A.root + ((double)compact2(key) + 0.5) * wl;
        }
        const bool lap = KIND == KIFMM_KERNEL_LAPLACE;
        ulonglong2 *sxy = sxys[LAP ? wib : 0];
        f32x2 *sz = szs[LAP ? wib : 0];
        float(*sk)[LAP ? 1 : LEAF_CHUNK + 64] = sks[LAP ? 0 : wib];
        const double width = ldexp(A.W, -l);
        const double sc = lap ? 1.0 / width : 1.0;     // coordinate scale
        const double lw = lap ? -2.0 * log2(sc) : 0.0; // log2 of the squared length unit
        const float kk = (float)A.k;
        const float lclamp = lg2_ftz(CLAMP);
        const int b = __shfl_sync(0xffffffffu, rv, LR_BOT), e = __shfl_sync(0xffffffffu, rv, LR_TOP);
        const int ns = __shfl_sync(0xffffffffu, rv, LR_NSRC);
        // source ranges: the leaf itself, then its colleagues in direction order;
        // list element p lies in the last range i with pre[i] <= p, at p + off[i]
        // (kept in shared memory: registers are scarce in the pair loop)
        int *rng = rngs[wib];
        if (lane >= LR_RNG && lane < LR_RNG + 18) rng[lane - LR_RNG] = rv;
        double tsum = 0.0;  // FP64 sum of the near sources' charges (Laplace)
        // stage sources [c0, c0 + cn) of the list, padded with 32 far, uncharged
        // ones (K0: 64 uncharged ones at the centre); four elements per lane per pass, loads issued before any is used
        auto gather = [&](int c0, int cn, bool sum) {
            __syncwarp();
            int pre[9], off[9];
    #pragma unroll
            for (int i = 0; i < 9; i++) {
                pre[i] = rng[i];
                off[i] = rng[9 + i];
            }
            for (int q0 = 0; q0 < cn; q0 += 128) {
                int si[4];
    #pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int q = q0 + lane + 32 * k, p = c0 + q;
                    int sv = p + off[0];
    #pragma unroll
                    for (int i = 1; i < 9; i++) sv = p >= pre[i] ? p + off[i] : sv;
                    si[k] = q < cn ? sv : -1;
                }
                double vx[4], vy[4], vt[4];
    #pragma unroll
                for (int k = 0; k < 4; k++)
                    if (si[k] >= 0) {
                        vx[k] = A.xs[si[k]];
                        vy[k] = A.ys[si[k]];
                        vt[k] = A.taus[si[k]];
                    }
    #pragma unroll
                for (int k = 0; k < 4; k++)
                    if (si[k] >= 0) {
                        const float fx = (float)((vx[k] - cx) * sc), fy = (float)((vy[k] - cy) * sc);
                        const float fz = (float)vt[k];
                        const int o = q0 + lane + 32 * k;
                        if (LAP) {
                            sxy[o] = make_ulonglong2(f2_pack(fx, fx), f2_pack(fy, fy));
                            sz[o] = f2_pack(fz, fz);
                        } else {
                            sk[0][o] = fx;
                            sk[1][o] = fy;
                            sk[2][o] = fz;
                        }
                        if (sum) tsum += vt[k];
                    }
            }
            if (LAP) {
                sxy[cn + lane] = make_ulonglong2(f2_pack(1e18f, 1e18f), f2_pack(1e18f, 1e18f));
                sz[cn + lane] = 0ull;
            } else {
#pragma unroll
                for (int h = 0; h < 64; h += 32) sk[0][cn + h + lane] = sk[1][cn + h + lane] = sk[2][cn + h + lane] = 0.f;
            }
            __syncwarp();
        };
        __syncwarp();
        const int tfirst = b + 32 * tile0, tend = (int)min((int64_t)e, (int64_t)b + 32 * (int64_t)tile1);
        for (int t0 = tfirst; t0 < tend; t0 += 32) {
            const int nt = min(32, e - t0);
            // Lane layout: the tile's targets form ng groups of tb targets
            // (two for the Laplace kernel, one otherwise); sp = 32 / ng lanes
            // share a group, lane (gi, j) taking sources j, j + sp, ...  Two
            // targets per lane share each source load and every packed
            // (f32x2) instruction of the pair loop.
            const int ng = lap ? (nt + 1) >> 1 : nt, sp = small_div(32, ng);
            const int j = small_div(lane, ng), gi = lane - j * ng;
            const int ia = gi, ib = lap && gi + ng < nt ? gi + ng : gi;  // second slot repeats the first when unused
            const float txa = (float)((A.xs[t0 + ia] - cx) * sc), tya = (float)((A.ys[t0 + ia] - cy) * sc);
            const float txb = (float)((A.xs[t0 + ib] - cx) * sc), tyb = (float)((A.ys[t0 + ib] - cy) * sc);
            const f32x2 tx2 = f2_pack(txa, txb), ty2 = f2_pack(tya, tyb);
            double neara = 0.0, nearb = 0.0;
            float exa = 0.f, exb = 0.f;  // charges of the leaf's own points met at the floor
            for (int c0 = 0; c0 < ns; c0 += LEAF_CHUNK) {
                const int cn = min(LEAF_CHUNK, ns - c0);
                if (t0 == tfirst || ns > LEAF_CHUNK) gather(c0, cn, lap && t0 == tfirst);
                // lane (gi, j) takes sources j, j + sp, ...; j + (it - 1) sp < cn + 32
                const int it = small_div(cn + sp - 1, sp);
                if (KIND == KIFMM_KERNEL_LAPLACE) {
                    // the list starts with the leaf's own points, local [0, en): the
                    // first kown passes count the pairs there that meet the floor
                    const int en = min(e - b - c0, cn);
                    const int kown = en > 0 ? small_div(en + sp - 1, sp) : 0;
                    leaf_pairs2_sp<true>(sp, sxy, sz, j, 0, kown, tx2, ty2, en, neara, nearb, exa, exb);
                    leaf_pairs2_sp<false>(sp, sxy, sz, j, kown, it, tx2, ty2, en, neara, nearb, exa, exb);
                } else {
                    leaf_pairs_k0(sk[0], sk[1], sk[2], j, sp, it, txa, tya, kk, neara);
                }
            }
            if (lap && t0 == tfirst)
                for (int o = 16; o; o >>= 1) tsum += __shfl_xor_sync(0xffffffffu, tsum, o);
            // per-lane shares with the clamped own pairs taken out
            red[wib][0][lane] = lap ? neara - (double)exa * (double)lclamp : neara;
            red[wib][1][lane] = lap ? nearb - (double)exb * (double)lclamp : nearb;
            redf[wib][0][lane] = exa;
            redf[wib][1][lane] = exb;
            __syncwarp();
            if (lane < nt) {
                const int t = t0 + lane;
                const int slot = lane < ng ? 0 : 1, grp = lane - slot * ng;
                double v = 0.0;
                float ex = 0.f;
                for (int m = 0; m < sp; m++) {
                    v += red[wib][slot][grp + m * ng];
                    ex += redf[wib][slot][grp + m * ng];
                }
                if (lap) {
                    // the skipped charges leave log2(w^2) * sum(tau); the one skipped
                    // pair is almost always the target itself: take its FP64 charge
                    const double tau_t = A.taus[t];
                    const double exd = ex == (float)tau_t ? tau_t : (double)ex;
                    v += lw * (tsum - exd);
                }
                A.pots[t] = v * (double)gsum_scale<KIND>();
            }
            __syncwarp();
        }
    }
}

// One warp per leaf, or with SPLIT (a leaf list smaller than half a wave of the
// GPU, where the kernel lasts as long as its heaviest leaf) two: the second takes
// the tiles after the leaf's first 32 points and leaves at once where there are
// none.
template <int KIND, bool SPLIT>
__global__ void __launch_bounds__(32 * LEAF_WARPS, LEAF_BLOCKS_PER_SM) k_leaf_near_f(PassArgs A, int64_t nlist) {
    pdl_trigger();
    pdl_wait();
    const int64_t w = (int64_t)blockIdx.x * LEAF_WARPS + (threadIdx.x >> 5);
    if (!SPLIT) {
        if (w < nlist) leaf_near_f<KIND>(A, w);
    } else if (w < 2 * nlist) {
        leaf_near_f<KIND>(A, w >> 1, w & 1, w & 1 ? 1 << 20 : 1);
    }
}

// The far field of the Laplace leaves, added to the near field that pots holds,
// with every lane busy: one block per 32 consecutive leaves of one level (the
// k_leaf_taylor tiling), each thread a target of those leaves.  The leaves'
// Taylor coefficients (written by k_leaf_taylor) are staged in shared memory,
// orders >= 9 as FP32 and orders <= 8 as FP64.  Targets beyond the series radius
// (points outside the root box; no others) take the direct sum over the
// equivalent points with the leaves' densities (k_leaf_density): formed per
// target from the inverse, a dozen such points in a million made this kernel
// 149 us long where it takes 21.
constexpr int FT_THREADS = 128;
__global__ void __launch_bounds__(FT_THREADS) k_leaf_far_taylor(TaylorArgs T) {
    constexpr int R = 2 * KIFMM_TAYLOR_P + 1;
    __shared__ float qf[32][R + 1];
    __shared__ double qd[32][17];  // orders 0..8
    __shared__ double scx[32], scy[32], ssc[32];
    __shared__ int sbot[32], spre[33], slev[32];
    const PassArgs &A = T.A;
    pdl_trigger();
    const int64_t b = blockIdx.x;
    int l = T.lmin;
    while (l < T.lmax && T.toff[l + 1] <= b) l++;
    const int64_t w0 = T.loff[l] + (b - T.toff[l]) * 32;
    const int nt = (int)min((int64_t)32, T.loff[l + 1] - w0);
    const int tid = threadIdx.x;
    pdl_wait();  // coefficients from k_leaf_taylor; near field in pots
    if (tid < 32) {
        int cnt = 0;
        if (tid < nt) {
            const int32_t *rec = A.leaf_rec + (w0 + tid) * LEAF_REC_WORDS;
            const int lv = rec[LR_LEVEL];
            const uint64_t key = (uint64_t)(uint32_t)rec[LR_KEY_LO] | ((uint64_t)(uint32_t)rec[LR_KEY_HI] << 32);
            const double wl = ldexp(A.W, -lv);
            scx[tid] = A.root + ((double)compact2(key >> 1) + 0.5) * wl;
            scy[tid] = A.root + ((double)compact2(key) + 0.5) * wl;
            ssc[tid] = 1.0 / wl;
            sbot[tid] = rec[LR_BOT];
            slev[tid] = lv;
            cnt = rec[LR_TOP] - rec[LR_BOT];
        }
        int v = cnt;  // inclusive scan of the leaves' point counts
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (tid >= o) v += u;
        }
        spre[tid + 1] = v;
        if (tid == 0) spre[0] = 0;
    }
    for (int i = tid; i < nt * R; i += FT_THREADS) {
        const int n = i / R, r = i - n * R;
        const double c = T.coef[(w0 + n) * R + r];
        qf[n][r] = (float)c;
        if (r < 17) qd[n][r] = c;
    }
    __syncthreads();
    const int total = spre[nt];
    for (int i = tid; i < total; i += FT_THREADS) {
        int n = 0;  // the leaf of flat target i: the last n with spre[n] <= i
        for (int step = 16; step; step >>= 1)
            if (n + step < nt && spre[n + step] <= i) n += step;
        const int t = sbot[n] + (i - spre[n]);
        const double pxd = A.xs[t] - scx[n], pyd = A.ys[t] - scy[n];
        const double zx = pxd * ssc[n], zy = pyd * ssc[n];
        double far;
        if (!T.den || zx * zx + zy * zy <= 0.5625) {
            const float zxf = (float)zx, zyf = (float)zy;
            float fr = qf[n][R - 2], fi = qf[n][R - 1];
            for (int jj = KIFMM_TAYLOR_P - 1; jj >= 9; jj--) {
                const float nr = fmaf(fr, zxf, fmaf(-fi, zyf, qf[n][2 * jj - 1]));
                const float ni = fmaf(fr, zyf, fmaf(fi, zxf, qf[n][2 * jj]));
                fr = nr;
                fi = ni;
            }
            double sr = fr, si = fi;
            for (int jj = 8; jj >= 1; jj--) {
                double nr = fma(sr, zx, fma(-si, zy, qd[n][2 * jj - 1]));
                double ni = fma(sr, zy, fma(si, zx, qd[n][2 * jj]));
                sr = nr;
                si = ni;
            }
            far = qd[n][0] + (sr * zx - si * zy);
        } else {
            const double *lgd = A.ops + (size_t)slev[n] * A.stride + A.off_large, *den = T.den + (size_t)(w0 + n) * A.Q;
            far = 0.0;
            for (int q = 0; q < A.Q; q++) {
                const double dx = pxd - lgd[q], dy = pyd - lgd[A.Q + q];
                far = fma(green_d(A.kind, A.k, dx * dx + dy * dy), den[q], far);
            }
        }
        if (A.out) A.out[A.perm[t]] = A.pots[t] + far;
        else         A.pots[t] += far;
    }
}

// The near field of several plans in one launch (serving batches): warp w of
// the grid takes leaf w - off[r] of plan r, off[r] <= w < off[r + 1].
template <int KIND>
__global__ void __launch_bounds__(32 * LEAF_WARPS, LEAF_BLOCKS_PER_SM)
    k_leaf_near_f_batch(const PassArgs *__restrict__ args, const int64_t *__restrict__ off, int nplan) {
    pdl_trigger();
    pdl_wait();
    const int64_t w = (int64_t)blockIdx.x * LEAF_WARPS + (threadIdx.x >> 5);
    int lo = 0, hi = nplan;  // the last r with off[r] <= w
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (off[mid] <= w) lo = mid;
        else hi = mid;
    }
    if (w < off[nplan]) leaf_near_f<KIND>(args[lo], w - off[lo]);
}

// m2l_tc.cu / passes.cu
void run_m2l_tensor(kifmm_plan *P, const PassArgs &A);
void run_m2m_levels(kifmm_plan *P, const PassArgs &A);
void run_l2l_levels(kifmm_plan *P, const PassArgs &A);

void near_launch(kifmm_plan *P, cudaStream_t s);
// P2M and M2M of the mixed apply
void mixed_upward(kifmm_plan *P, const PassArgs &A) {
    if (P->n_p2m_list) {
        PhaseScope ph(P, KIFMM_PHASE_P2M);
        if (planned_ready(P)) launch_planned_p2m(P, A);
        else launch_p2m_d(P, A);
    }
    ops_wait_now(P);  // the P2M reads only the check circles
    PhaseScope ph(P, KIFMM_PHASE_M2M);
    run_m2m_levels(P, A);
}

// the L2L chain after the M2L
void mixed_l2l(kifmm_plan *P, const PassArgs &A) {
    PhaseScope ph(P, KIFMM_PHASE_L2L);
    run_l2l_levels(P, A);
}

void run_passes_mixed(kifmm_plan *P) {
    const int Q = P->Q, L = P->L;
    if (L < 3) return;  // expansions cleared by run_upward_downward
    // The near field at the sources on a low-priority stream.  A leaf list of
    // less than half a wave starts with the apply and runs beside the chain; a
    // larger one starts after the M2M chain, under a far-field chain on a
    // high-priority stream (launches and allocations swapped there, joined back
    // into the plan's stream at the end).
    const bool near = near_possible(P), early = near && near_split(P);
    if (early) near_fork(P);
    HighPriorityFork fork(P, near && !early);
    PassArgs A = make_pass_args(P);
    mixed_upward(P, A);
    if (near && !early) near_fork(P);  // after the M2M chain, under the M2L and L2L
    if (P->opt.m2l == KIFMM_M2L_FP32) {
        PhaseScope ph(P, KIFMM_PHASE_M2L);
        const int thr = ((4 * Q + 31) / 32) * 32;
        const size_t smem = (size_t)M2LF_TE * 4 * Q * sizeof(float);
        ensure_dyn_smem(k_m2l_f, smem);
        for (int l = 1; l <= L - 2; l++) {
            int64_t ne = P->lt.ne[l];
            if (!ne) continue;
            k_m2l_f<<<(unsigned)((ne + M2LF_TE - 1) / M2LF_TE), thr, smem, P->stream>>>(A, l);  // (the far stream)
            KIFMM_LAUNCHED();
        }
        return;
    }
    {
        PhaseScope ph(P, KIFMM_PHASE_M2L);
        run_m2l_tensor(P, A);  // all levels at once
    }
    mixed_l2l(P, A);
}

// the 32-leaf tiles of the leaves at levels >= 2 (k_leaf_taylor, k_leaf_far_taylor)
static TaylorArgs taylor_tiling(kifmm_plan *P, const PassArgs &A, int64_t *ntiles) {
    TaylorArgs T{};
    T.A = A;
    T.list = P->leaf_list.p;
    T.coef = P->leaf_coef.p;
    T.lmin = 2;
    T.lmax = P->L - 1;
    int64_t tiles = 0;
    for (int l = 0; l <= MAX_LEVELS; l++) {
        T.loff[l] = P->leaf_loff[l];
        T.toff[l] = tiles;
        if (l >= T.lmin && l <= T.lmax && l < MAX_LEVELS) tiles += (P->leaf_loff[l + 1] - P->leaf_loff[l] + 31) / 32;
    }
    *ntiles = tiles;
    return T;
}

// The far field at the sources, added to the near field in pots, to A.out.
// near_done (or null): the event after which pots holds the near field; the
// Taylor coefficients and densities do not wait for it.
void launch_scatter_pot(kifmm_plan *P, double *pot);  // passes.cu
void mixed_far(kifmm_plan *P, PassArgs A, cudaEvent_t near_done) {
    // leaves above level 2 have no far field: their potentials go out by the scatter
    const bool all = P->leaf_loff[2] == 0;
    double *pot = A.out;
    if (!all) A.out = nullptr;
    if (P->kern.kind == KIFMM_KERNEL_MOD_HELMHOLTZ) {
        if (P->L >= 3) launch_leaf_far_d(P, A, near_done), near_done = nullptr;
    } else if (P->l2p_taylor.p && P->L >= 3) {
        constexpr int R = 2 * KIFMM_TAYLOR_P + 1;
        KIFMM_REQUIRE(P->Q % 4 == 0, KIFMM_ERR_ARG, "mixed Laplace form: Nequiv must be a multiple of 4");
        P->leaf_coef.alloc((size_t)P->n_leaf_list * R);
        A.leaf_coef = P->leaf_coef.p;
        int64_t tiles = 0;
        TaylorArgs T = taylor_tiling(P, A, &tiles);
        if (tiles) {
            if (P->n_outside) T.den = launch_leaf_density(P, A);
            const size_t smem = ((size_t)P->Q * pad4mod16(8 * TY_MTR) + 32 * (size_t)pad4mod16(P->Q) + 32 * (size_t)R) *
                                sizeof(double);
            ensure_dyn_smem(k_leaf_taylor, smem);
            launch_pdl(k_leaf_taylor, dim3((unsigned)tiles), dim3(TY_THREADS), smem, P->stream, T);
            if (near_done) KIFMM_CUDA(cudaStreamWaitEvent(P->stream, near_done, 0));
            near_done = nullptr;
            launch_pdl(k_leaf_far_taylor, dim3((unsigned)tiles), dim3(FT_THREADS), 0, P->stream, T);
        }
    }
    if (near_done) KIFMM_CUDA(cudaStreamWaitEvent(P->stream, near_done, 0));
    if (!all) launch_scatter_pot(P, pot);
}

void run_eval_sources_mixed(kifmm_plan *P, PassArgs A, int check_self) {
    if (!P->n_leaf_list) return;
    PhaseScope ph(P, KIFMM_PHASE_LEAF);
    if (P->opt.near_fp64) {
        launch_leaf_eval_d(P, A, check_self);
        return;
    }
    // FP32 form: coincident pairs always contribute zero
    const bool pending = near_under_way(P);  // the near field is on its way into P->pots
    P->near_pending = false;
    if (!pending) near_launch(P, P->stream);
    mixed_far(P, A, pending ? P->near_done : nullptr);
}

// The near field at the sources (P2P of every leaf over its colleagues) needs
// only the sorted points and charges, none of the expansions, so the apply
// runs it on a stream of its own while the far-field chain leaves SMs idle,
// and the evaluation at the sources adds only the far field (mixed_far).
// Mixed FP32 near field, where the near sum does not depend on check_self
// (coincident pairs contribute zero), and the planned near matrices, which an
// evaluation that keeps self pairs does not use.  A later evaluation at other
// targets leaves the pass unused; a second one at the sources runs it again.
// The near pass runs on a stream of the lowest priority.  For large leaf lists
// the far-field chain runs on one of the highest, and the pass starts after the
// M2M chain, under the source slicing, M2L and L2L: started with the apply its
// blocks, filling every SM, held off the M2M chain's small level launches even
// with the priorities (M2M 0.086 -> 0.18 ms at 1M points).  Measured per step
// against the single leaf pass after the chain: 1M mixture 1.005 -> 0.953 ms
// (0.971-0.994 when started with the apply), 4M uniform 2.446 -> 2.444 ms, 2M K0
// annulus 6.02 -> 5.20 ms (the K0 near field is several times longer than the
// chain, which runs under it).  Lists of less than half a wave start with the
// apply.

// the plan's near stream (lowest priority) and far stream (highest), once,
// from the per-device pool
void aux_streams_acquire(int device, cudaStream_t *near, cudaStream_t *far);  // capi.cu: per-device pool
void ensure_aux_streams(kifmm_plan *P) {
    if (P->near_stream) return;
    aux_streams_acquire(P->device, &P->near_stream, &P->far_stream);
    for (cudaEvent_t *e : {&P->near_fork, &P->near_done, &P->far_fork, &P->far_done})
        KIFMM_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
}

// Whether the plan's stream is in a capture of the caller's.  A plan that was in one
// is marked: the caller may replay that graph at any time, without a call into this
// library that could join a near pass, so the plan's later applies join theirs.
bool callers_capture(kifmm_plan *P) {
    if (P->own_capture) return false;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    KIFMM_CUDA(cudaStreamIsCapturing(P->stream, &cap));
    if (cap == cudaStreamCaptureStatusNone) return false;
    P->callers_graph = true;
    return true;
}

// options with a near pass apart from the leaf pass
static bool near_form(const kifmm_plan *P) {
    return !P->cplx && (P->opt.planned || (P->opt.precision == KIFMM_PREC_MIXED && !P->opt.near_fp64));
}
bool near_possible(kifmm_plan *P) {
    if (!near_form(P) || P->n_leaf_list <= 0 || (P->opt.planned != 0) != planned_ready(P)) return false;
    if (P->opt.planned && !planned_near_fits(P)) return false;
    if (callers_capture(P)) return false;  // it may end between the apply and the evaluation that joins
    ensure_aux_streams(P);
    return true;
}
// fewer leaves than half a wave of warps: the big ones are split over two warps
bool near_split(const kifmm_plan *P) {
    return P->n_leaf_list < (int64_t)P->num_sms * LEAF_BLOCKS_PER_SM * LEAF_WARPS / 2;
}

// the near pass on stream s
void near_launch(kifmm_plan *P, cudaStream_t s) {
    const int64_t nl = P->n_leaf_list;
    const PassArgs A = make_pass_args(P);
    const bool split = near_split(P);
    const dim3 grid((unsigned)(((split ? 2 * nl : nl) + LEAF_WARPS - 1) / LEAF_WARPS)), block(32 * LEAF_WARPS);
    constexpr int LAP = KIFMM_KERNEL_LAPLACE, K0 = KIFMM_KERNEL_MOD_HELMHOLTZ;
    if (P->kern.kind == LAP) {
        if (split) launch_pdl(k_leaf_near_f<LAP, true>, grid, block, 0, s, A, nl);
        else launch_pdl(k_leaf_near_f<LAP, false>, grid, block, 0, s, A, nl);
    } else {
        if (split) launch_pdl(k_leaf_near_f<K0, true>, grid, block, 0, s, A, nl);
        else launch_pdl(k_leaf_near_f<K0, false>, grid, block, 0, s, A, nl);
    }
}

// ... on the near stream, forked from the plan's stream at this point
void near_fork(kifmm_plan *P) {
    KIFMM_CUDA(cudaEventRecord(P->near_fork, P->stream));
    KIFMM_CUDA(cudaStreamWaitEvent(P->near_stream, P->near_fork, 0));
    {
        struct Swap {  // the phase timer's events go to the near stream
            kifmm_plan *P;
            cudaStream_t main;
            Swap(kifmm_plan *p) : P(p), main(p->stream) { P->stream = P->near_stream; }
            ~Swap() { P->stream = main; }
        } sw(P);
        PhaseScope ph(P, KIFMM_PHASE_LEAF);
        if (planned_ready(P)) launch_planned_near(P, P->near_stream);
        else near_launch(P, P->near_stream);
    }
    KIFMM_CUDA(cudaEventRecord(P->near_done, P->near_stream));
    P->near_pending = true;
}

// Whether a near-field pass is in flight that an evaluation can wait for and use.
// A capture of the caller's that began after the apply cannot depend on it: there
// the host waits for it, and it is dropped.
bool near_under_way(kifmm_plan *P) {
    if (!near_form(P) || !callers_capture(P) || !P->near_pending) return P->near_pending;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    KIFMM_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    const cudaError_t rc = cudaEventSynchronize(P->near_done);
    cudaThreadExchangeStreamCaptureMode(&mode);
    KIFMM_CUDA(rc);
    P->near_pending = false;
    return false;
}

// a near-field pass in flight is waited for and dropped (a new tree or apply
// replaces the buffers it reads and writes)
void near_join(kifmm_plan *P) {
    if (!near_under_way(P)) return;
    KIFMM_CUDA(cudaStreamWaitEvent(P->stream, P->near_done, 0));
    P->near_pending = false;
}

// the FP32 near field of several plans of one kernel kind in one launch
void launch_leaf_f_batch(int kind, const PassArgs *dargs, const int64_t *doff, int nplan, int64_t nleaf,
                         cudaStream_t s) {
    const int64_t blocks = (nleaf + LEAF_WARPS - 1) / LEAF_WARPS;
    KIFMM_REQUIRE(blocks > 0 && blocks < (1ll << 31), KIFMM_ERR_ARG, "batch leaf pass: bad leaf count");
    if (kind == KIFMM_KERNEL_LAPLACE)
        k_leaf_near_f_batch<KIFMM_KERNEL_LAPLACE><<<(unsigned)blocks, 32 * LEAF_WARPS, 0, s>>>(dargs, doff, nplan);
    else
        k_leaf_near_f_batch<KIFMM_KERNEL_MOD_HELMHOLTZ><<<(unsigned)blocks, 32 * LEAF_WARPS, 0, s>>>(dargs, doff,
                                                                                                      nplan);
    KIFMM_LAUNCHED();
}

}  // namespace kifmm
