// radix_sort.cu -- stable LSD radix sort of 64-bit keys (optionally with int32
// payloads) for the Morton-key tree build.
//
// The plan's sorts use the onesweep form further down (one histogram kernel,
// then one kernel per 8-bit digit).  The no-allocation entry point keeps the
// three-kernel form, whose scratch is a fixed histogram table: each pass
// sorts one 8-bit digit in three kernels:
//   1. per-tile digit histograms (tile = 256 threads x 16 keys),
//   2. a per-digit exclusive scan over the tiles (one block per digit), which
//      also leaves the 256 digit totals behind the table,
//   3. a stable scatter: inside a tile, each warp ranks its 512 keys in order
//      with __match_any_sync, warps are combined by a per-digit prefix in
//      shared memory, and the tile's base is the digit's start (a scan of the
//      digit totals) plus the digit's scanned tile prefix.
#include <algorithm>

#include "kifmm_internal.cuh"

namespace kifmm {

constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 16;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
static_assert(RS_TILE == RADIX_TILE_KEYS, "histogram tables sized outside this file assume RADIX_TILE_KEYS per tile");
constexpr int RS_WARPS = RS_THREADS / 32;

__global__ void __launch_bounds__(RS_THREADS) k_rs_hist(const uint64_t *__restrict__ key, int64_t n, int shift,
                                                         uint32_t *__restrict__ hist, int nblocks) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    int64_t base = (int64_t)blockIdx.x * RS_TILE;
#pragma unroll 4
    for (int i = 0; i < RS_ITEMS; i++) {
        int64_t idx = base + i * RS_THREADS + threadIdx.x;
        if (idx < n) atomicAdd(&h[(key[idx] >> shift) & 255], 1u);
    }
    __syncthreads();
    hist[(size_t)threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

// Per-digit scan: block d turns hist[d][0..nb) into exclusive prefixes over
// the tiles and writes the digit's total to dtot[d] (dtot = hist + 256 * nb).
__global__ void __launch_bounds__(256) k_rs_scan(uint32_t *__restrict__ hist, int nblocks) {
    __shared__ uint32_t part[256];
    uint32_t *h = hist + (size_t)blockIdx.x * nblocks;
    const int chunk = (nblocks + 255) / 256;
    const int b = threadIdx.x * chunk, e = min(b + chunk, nblocks);
    uint32_t sum = 0;
    for (int i = b; i < e; i++) sum += h[i];
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int off = 1; off < 256; off <<= 1) {
        uint32_t v = threadIdx.x >= off ? part[threadIdx.x - off] : 0;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    uint32_t run = part[threadIdx.x] - sum;
    for (int i = b; i < e; i++) {
        uint32_t v = h[i];
        h[i] = run;
        run += v;
    }
    if (threadIdx.x == 255) hist[(size_t)256 * nblocks + blockIdx.x] = part[255];
}

template <bool PAIRS>
__global__ void __launch_bounds__(RS_THREADS) k_rs_scatter(const uint64_t *__restrict__ key, const int32_t *__restrict__ val,
                                                            uint64_t *__restrict__ okey, int32_t *__restrict__ oval,
                                                            int64_t n, int shift, const uint32_t *__restrict__ hist,
                                                            int nblocks) {
    __shared__ uint32_t wcnt[RS_WARPS][256];
    __shared__ uint32_t base[256];
    __shared__ uint32_t wsum[RS_WARPS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int d = threadIdx.x; d < 256 * RS_WARPS; d += RS_THREADS) (&wcnt[0][0])[d] = 0;
    {  // digit bases: exclusive scan of the 256 digit totals
        uint32_t t = hist[(size_t)256 * nblocks + threadIdx.x], x = t;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        uint32_t woff = 0;
        for (int i = 0; i < w; i++) woff += wsum[i];
        base[threadIdx.x] = woff + x - t + hist[(size_t)threadIdx.x * nblocks + blockIdx.x];
    }
    __syncthreads();
    const int64_t t0 = (int64_t)blockIdx.x * RS_TILE + (int64_t)w * (RS_ITEMS * 32);
    uint64_t k[RS_ITEMS];
    int32_t v[RS_ITEMS];
    uint32_t rank[RS_ITEMS];
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < RS_ITEMS; r++) {
        int64_t idx = t0 + r * 32 + lane;
        bool ok = idx < n;
        k[r] = ok ? key[idx] : 0;
        if (PAIRS) v[r] = ok ? val[idx] : 0;
        uint32_t d = ok ? (uint32_t)((k[r] >> shift) & 255) : 256u;
        unsigned peers = __match_any_sync(0xffffffffu, d);
        uint32_t before = d < 256 ? wcnt[w][d] : 0;
        rank[r] = before + __popc(peers & lt);
        __syncwarp();
        if (d < 256 && lane == __ffs(peers) - 1) wcnt[w][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // exclusive prefix over warps for each digit, folded into per-warp offsets
    {
        int d = threadIdx.x;
        uint32_t run = base[d];
#pragma unroll
        for (int ww = 0; ww < RS_WARPS; ww++) {
            uint32_t c = wcnt[ww][d];
            wcnt[ww][d] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ITEMS; r++) {
        int64_t idx = t0 + r * 32 + lane;
        if (idx < n) {
            uint32_t d = (uint32_t)((k[r] >> shift) & 255);
            uint32_t pos = wcnt[w][d] + rank[r];
            okey[pos] = k[r];
            if (PAIRS) oval[pos] = v[r];
        }
    }
}

// ---------------------------------------------------------------- onesweep
// The plan's sorts: one read of the keys counts the digits of every pass
// (k_os_hist), then each pass is ONE kernel (k_os_pass) that ranks a tile's
// keys as k_rs_scatter does and finds the tile's offset for each digit by a
// look-back over the tiles before it: every tile publishes its digit counts as
// soon as it has ranked its keys; the tiles of a pass all run at once, so
// instead of a chain of inclusive prefixes (one round trip per 32 tiles) the
// look-back has two levels, tiles within a group of 32 and group totals.
// Tiles take their index from a counter in the order they start, so every
// tile waited on is already running and publishes without waiting on later
// tiles.  Waits are bounded; one that runs out sets *err (the build fails).
constexpr int OS_MAX_PASSES = 8;
struct OsShifts {
    int n;
    int s[OS_MAX_PASSES];
};
constexpr uint32_t OS_AGG = 1u << 31;  // a look-back word that has been published (counts stay below 2^18)
constexpr int OS_GROUP = 32;  // tiles per look-back group

__device__ __forceinline__ void st_relaxed_u32(uint32_t *p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// digit counts of every pass; shifts packed 8 bits each in `packed` (no
// per-pass array in local memory), npass <= OS_MAX_PASSES
__global__ void __launch_bounds__(RS_THREADS) k_os_hist(const uint64_t *__restrict__ key, int64_t n, uint64_t packed,
                                                         int npass, uint32_t *__restrict__ hist) {
    // warp-private counters per pass (conflicts only among a warp's own lanes):
    // dynamic shared memory [RS_WARPS][npass][256]
    extern __shared__ uint32_t h_dyn[];
    pdl_trigger();
    pdl_wait();
    for (int i = threadIdx.x; i < RS_WARPS * npass * 256; i += RS_THREADS) h_dyn[i] = 0;
    __syncthreads();
    const int w = threadIdx.x >> 5;
    for (int64_t base = (int64_t)blockIdx.x * RS_TILE; base < n; base += (int64_t)gridDim.x * RS_TILE) {
        uint64_t k[RS_ITEMS];
#pragma unroll
        for (int r = 0; r < RS_ITEMS; r++) {
            const int64_t idx = base + r * RS_THREADS + threadIdx.x;
            k[r] = idx < n ? key[idx] : 0;
        }
#pragma unroll
        for (int p = 0; p < OS_MAX_PASSES; p++) {
            if (p >= npass) break;
            const int sh = (int)((packed >> (8 * p)) & 63);
#pragma unroll
            for (int r = 0; r < RS_ITEMS; r++)
                if (base + r * RS_THREADS + threadIdx.x < n)
                    atomicAdd(&h_dyn[(w * npass + p) * 256 + ((k[r] >> sh) & 255)], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < npass * 256; i += RS_THREADS) {
        uint32_t c = 0;
#pragma unroll
        for (int ww = 0; ww < RS_WARPS; ww++) c += h_dyn[ww * npass * 256 + i];
        if (c) atomicAdd(&hist[i], c);
    }
}

// One pass.  The tile's keys are ranked per warp, ordered by digit in shared
// memory (tile-local digit starts tstart[]), and written out in that order so
// that consecutive threads store consecutive positions of one digit's run.
// What bounds it: the ranking's ballots (8 per key and warp; the ALU pipe is busy
// 67% of a 4M-key pass), then latency.  Two blocks of 16 warps per SM: with 8 warps
// of twice the keys each the chain of a warp's ranking steps was exposed (4M keys
// and values: 73 us a pass, now 44 for words; 1M 23 -> 17.5, 300k 18.7 -> 10.6).
// Look-back words are 32 bits, and a block reads them with all its threads.
constexpr int OS_THREADS = 512;
constexpr int OS_WARPS = OS_THREADS / 32;
// what a pass carries: keys, (key, value) pairs, or words of a 32-bit key above a
// 32-bit value, which the last pass takes apart into a key (shifted up by
// `unpack`) and a value
enum { OS_KEYS, OS_PAIRS, OS_UNPACK };
template <int MODE, int ITEMS>
constexpr size_t os_pass_smem() {
    return (size_t)OS_THREADS * ITEMS * (sizeof(uint64_t) + (MODE == OS_PAIRS ? sizeof(int32_t) : 0));
}
template <int MODE, int ITEMS>
__global__ void __launch_bounds__(OS_THREADS, 2) k_os_pass(const uint64_t *__restrict__ key, const int32_t *__restrict__ val,
                                                           uint64_t *__restrict__ okey, int32_t *__restrict__ oval,
                                                           int64_t n, int shift, int unpack,
                                                           const uint32_t *__restrict__ ghist, uint32_t *status,
                                                           unsigned *tile_ctr, unsigned long long *err, long long limit) {
    constexpr int TILE = OS_THREADS * ITEMS;
    constexpr bool PAIRS = MODE == OS_PAIRS;
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) unsigned char os_sm[];
    uint64_t *skey = (uint64_t *)os_sm;                        // [TILE]
    int32_t *sval = (int32_t *)(os_sm + TILE * sizeof(uint64_t));
    __shared__ uint32_t wcnt[OS_WARPS][256];
    __shared__ uint32_t tstart[256];
    __shared__ uint32_t dbase[256];
    __shared__ uint32_t half[2][256];
    __shared__ uint32_t wsum[2][8];
    __shared__ unsigned tile_s;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) tile_s = atomicAdd(tile_ctr, 1u);
    for (int d = threadIdx.x; d < 256 * OS_WARPS; d += OS_THREADS) (&wcnt[0][0])[d] = 0;
    __syncthreads();
    const unsigned tile = tile_s;
    const int64_t tbase = (int64_t)tile * TILE;
    const int tn = (int)min((int64_t)TILE, n - tbase);
    const int i0 = w * (ITEMS * 32) + lane;  // this thread's keys: i0 + 32 r of the tile
    const bool full = tn == TILE;
    key += tbase;
    uint64_t k[ITEMS];
    int32_t v[ITEMS];
    uint32_t rank[ITEMS];
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const bool ok = full || i0 + r * 32 < tn;
        k[r] = ok ? key[i0 + r * 32] : 0;
        if (PAIRS) v[r] = ok ? val[tbase + i0 + r * 32] : 0;
    }
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const uint32_t d = (uint32_t)(k[r] >> shift) & 255u;
        unsigned peers = warp_match_bits<8>(d);
        if (!full) {  // lanes past the end stay out
            const bool ok = i0 + r * 32 < tn;
            const unsigned in = __ballot_sync(0xffffffffu, ok);
            peers = ok ? peers & in : 0;
        }
        const uint32_t before = wcnt[w][d];
        rank[r] = before + __popc(peers & lt);
        __syncwarp();
        if (peers && (peers & lt) == 0) wcnt[w][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    const int d = threadIdx.x & 255, hv = threadIdx.x >> 8;
    uint32_t tot = 0, g = 0, xt = 0, xg = 0;
    if (hv == 0) {
#pragma unroll
        for (int ww = 0; ww < OS_WARPS; ww++) {
            const uint32_t c = wcnt[ww][d];
            wcnt[ww][d] = tot;
            tot += c;
        }
        // this tile's digit counts, for the look-back of the later tiles
        st_relaxed_u32(status + (size_t)tile * 256 + d, OS_AGG | tot);
        // scans over the digits: tile-local starts, and the pass's global starts
        g = ghist[d];
        xt = tot;
        xg = g;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t yt = __shfl_up_sync(0xffffffffu, xt, o), yg = __shfl_up_sync(0xffffffffu, xg, o);
            if (lane >= o) {
                xt += yt;
                xg += yg;
            }
        }
        if (lane == 31) {
            wsum[0][w] = xt;
            wsum[1][w] = xg;
        }
    }
    __syncthreads();
    uint32_t ts = 0;
    if (hv == 0) {
        uint32_t wt = 0;
        for (int i = 0; i < w; i++) {
            wt += wsum[0][i];
            xg += wsum[1][i];
        }
        ts = wt + xt - tot;
        tstart[d] = ts;
    }
    __syncthreads();
    // the tile in digit order into shared memory, before the look-back, so
    // that the look-back has the registers for wide batches
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        if (full || i0 + r * 32 < tn) {
            const uint32_t dd = (uint32_t)(k[r] >> shift) & 255u;
            const uint32_t li = tstart[dd] + wcnt[w][dd] + rank[r];
            skey[li] = k[r];
            if (PAIRS) sval[li] = v[r];
        }
    }
    // Two-level look-back.  Tiles form groups of OS_GROUP: a tile sums the
    // counts of the earlier tiles of its group (one batch of loads); the last
    // tile of a group then publishes the group's total; a tile adds the totals
    // of the earlier groups (one batch per OS_GROUP groups).  Each half of the
    // block takes half of every batch.  Every wait is on a tile with a smaller
    // index, which started earlier and publishes without waiting on later tiles.
    // Polls are bounded; one that runs out sets *err.
    uint32_t *gbase = status + (size_t)gridDim.x * 256;  // [groups][256] group totals
    const unsigned grp = tile / OS_GROUP, tin = tile % OS_GROUP;
    bool ok = true;
    // the words of one digit at base + 256 q, q < cnt of this half's OS_GROUP / 2
    auto sum_published = [&](const uint32_t *base, int cnt, uint32_t &acc) {
        constexpr int B = OS_GROUP / 2;
        base += (size_t)hv * B * 256 + d;
        cnt -= hv * B;
        unsigned rem = cnt >= B ? (1u << B) - 1u : cnt > 0 ? (1u << cnt) - 1u : 0u;
        long long polls = 0;
        while (rem) {
            uint32_t sv[B];
#pragma unroll
            for (int q = 0; q < B; q++) sv[q] = ((rem >> q) & 1u) ? ld_relaxed_u32(base + (size_t)q * 256) : 0u;
#pragma unroll
            for (int q = 0; q < B; q++)
                if (sv[q] & OS_AGG) {
                    acc += sv[q] & ~OS_AGG;
                    rem &= ~(1u << q);
                }
            if (rem && ++polls > limit) {
                atomicOr(err, 1ull);
                return false;
            }
        }
        return true;
    };
    uint32_t acc = 0;
    if (tin > 0) ok = sum_published(status + (size_t)grp * OS_GROUP * 256, (int)tin, acc);
    if (tin == OS_GROUP - 1 || tile == gridDim.x - 1) {
        if (hv) half[0][d] = acc;
        __syncthreads();
        if (!hv) st_relaxed_u32(gbase + (size_t)grp * 256 + d, OS_AGG | (acc + half[0][d] + tot));
    }
    for (unsigned g0 = 0; ok && g0 < grp; g0 += OS_GROUP)
        ok = sum_published(gbase + (size_t)g0 * 256, (int)min((unsigned)OS_GROUP, grp - g0), acc);
    if (hv) half[1][d] = acc;
    // a look-back that ran out leaves the offsets unknown: write nothing (*err is set)
    if (__syncthreads_or(!ok)) return;
    if (!hv) dbase[d] = xg - g + acc + half[1][d] - ts;  // global position = dbase[digit] + tile-local index
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const int i = r * OS_THREADS + threadIdx.x;
        if (full || i < tn) {
            const uint64_t kk = skey[i];
            const uint32_t pos = dbase[(uint32_t)(kk >> shift) & 255u] + (uint32_t)i;
            okey[pos] = MODE == OS_UNPACK ? (kk >> 32) << unpack : kk;
            if (PAIRS) oval[pos] = sval[i];
            if (MODE == OS_UNPACK) oval[pos] = (int32_t)(uint32_t)kk;
        }
    }
}

template <int MODE, int ITEMS>
static void os_launch(kifmm_plan *P, int64_t ntiles, const uint64_t *key, const int32_t *val, uint64_t *okey,
                      int32_t *oval, int64_t n, int shift, int unpack, const uint32_t *hist, uint32_t *stat, unsigned *ctr) {
    constexpr size_t smem = os_pass_smem<MODE, ITEMS>();
    ensure_dyn_smem(k_os_pass<MODE, ITEMS>, smem);
    launch_pdl(k_os_pass<MODE, ITEMS>, dim3((unsigned)ntiles), dim3(OS_THREADS), smem, P->stream, key, val, okey, oval, n,
               shift, unpack, hist, stat, ctr, P->scal.p + KIFMM_SCAL_SORT_ERR, 1ll << 20);
}

// Sort by the 8-bit digits at the given shifts (ascending), stable.  `unpack` >= 0:
// the keys are words of a 32-bit key above a 32-bit value, taken apart by the last
// pass into key << unpack and val.
static void os_run(uint64_t *key, int32_t *val, uint64_t *key_tmp, int32_t *val_tmp, int64_t n, const int *shifts,
                   int npass, kifmm_plan *P, int mode, int unpack = 0) {
    KIFMM_REQUIRE(n < (1ll << 31), KIFMM_ERR_ARG, "radix sort: more than 2^31 keys");
    KIFMM_REQUIRE(npass <= OS_MAX_PASSES, KIFMM_ERR_ARG, "radix sort: too many passes");
    cudaStream_t s = P->stream;
    // keys per thread: 8 while two tiles per SM hold them all (1M: the tree 21 us
    // shorter than with 16), then 16 (4M: 18 us shorter than with 8).  4 keys make a
    // pass of 300k 9.2 instead of 10.6 us and no call shorter; at 4M they cost 52 us.
    // Pairs, which need more registers, stay at 8.
    const int items = n <= 16 * (int64_t)P->num_sms * OS_THREADS || mode == OS_PAIRS ? 8 : 16;
    const int64_t tile = OS_THREADS * items, ntiles = (n + tile - 1) / tile;
    OsShifts sh{};
    sh.n = npass;
    for (int p = 0; p < npass; p++) sh.s[p] = shifts[p];
    // scratch: digit counts [npass][256], tile counters [npass], look-back status
    // [npass][ntiles][256] (one pass's worth, cleared before each pass, when large)
    // per pass: the tiles' digit counts, then the groups' totals
    const size_t per_pass = (size_t)(ntiles + (ntiles + OS_GROUP - 1) / OS_GROUP) * 256;
    const bool all_at_once = (size_t)npass * per_pass * 4 <= ((size_t)32 << 20);
    const size_t nstat = all_at_once ? (size_t)npass * per_pass : per_pass;
    P->sort_hist.alloc((size_t)npass * 256 + npass);
    P->sort_status.alloc(nstat);
    uint32_t *hist = P->sort_hist.p;
    unsigned *ctr = P->sort_hist.p + (size_t)npass * 256;
    launch_fill(P, {{hist, (size_t)npass * 256 + npass, 0u}, {P->sort_status.p, nstat, 0u}});
    const unsigned hg = (unsigned)std::min<int64_t>((n + RS_TILE - 1) / RS_TILE, (int64_t)P->num_sms * 4);
    uint64_t packed = 0;
    for (int p = 0; p < npass; p++) packed |= (uint64_t)(shifts[p] & 63) << (8 * p);
    const size_t hsm = (size_t)RS_WARPS * npass * 256 * sizeof(uint32_t);
    ensure_dyn_smem(k_os_hist, hsm);
    launch_pdl(k_os_hist, dim3(hg), dim3(RS_THREADS), hsm, s, (const uint64_t *)key, n, packed, npass, hist);
    uint64_t *ka = key, *kb = key_tmp;
    int32_t *va = val, *vb = val_tmp;
    for (int p = 0; p < npass; p++) {
        uint32_t *stat = P->sort_status.p + (all_at_once ? (size_t)p * per_pass : 0);
        if (!all_at_once && p > 0) KIFMM_CUDA(cudaMemsetAsync(stat, 0, per_pass * sizeof(uint32_t), s));
        const bool last = p == npass - 1;
        auto go = [&](auto m, auto it) {
            os_launch<decltype(m)::value, decltype(it)::value>(P, ntiles, ka, va, kb, mode == OS_UNPACK ? val : vb, n,
                                                               sh.s[p], unpack, hist + 256 * p, stat, ctr + p);
        };
        auto size = [&](auto m) {
            constexpr int WIDE = decltype(m)::value == OS_PAIRS ? 8 : 16;
            if (items == 8) go(m, std::integral_constant<int, 8>{});
            else go(m, std::integral_constant<int, WIDE>{});
        };
        if (mode == OS_PAIRS) size(std::integral_constant<int, OS_PAIRS>{});
        else if (mode == OS_UNPACK && last) size(std::integral_constant<int, OS_UNPACK>{});
        else size(std::integral_constant<int, OS_KEYS>{});
        std::swap(ka, kb);
        std::swap(va, vb);
    }
    if (ka != key) {
        KIFMM_CUDA(cudaMemcpyAsync(key, ka, n * sizeof(uint64_t), cudaMemcpyDeviceToDevice, s));
        if (mode == OS_PAIRS) KIFMM_CUDA(cudaMemcpyAsync(val, va, n * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
    }
}

void radix_sort_pairs(uint64_t *key, int32_t *val, uint64_t *key_tmp, int32_t *val_tmp, int64_t n, int bits,
                      kifmm_plan *P) {
    int shifts[OS_MAX_PASSES];
    const int passes = (bits + 7) / 8;
    for (int p = 0; p < passes; p++) shifts[p] = 8 * p;
    if (n > 1) os_run(key, val, key_tmp, val_tmp, n, shifts, passes, P, OS_PAIRS);
}

// words (32-bit key << 32 | value) sorted stably by key; then key = (32-bit key)
// << up, and the values in val
void radix_sort_words(uint64_t *key, int32_t *val, uint64_t *key_tmp, int64_t n, int up, kifmm_plan *P) {
    const int shifts[4] = {32, 40, 48, 56};
    if (n > 0) os_run(key, val, key_tmp, nullptr, n, shifts, 4, P, OS_UNPACK, up);
}

// keys sorted by the digits at `shifts` only: the caller knows the other
// digits are equal for every key
void radix_sort_keys_shifts(uint64_t *key, uint64_t *key_tmp, int64_t n, const int *shifts, int npass,
                            kifmm_plan *P) {
    if (n > 1 && npass > 0) os_run(key, nullptr, key_tmp, nullptr, n, shifts, npass, P, OS_KEYS);
}

int64_t radix_sort_hist_words(int64_t n) { return (int64_t)256 * ((n + RS_TILE - 1) / RS_TILE) + 256; }

// Same passes as rs_run, on caller-provided scratch (histogram table of
// radix_sort_hist_words(n) words, ping-pong buffers of n entries); launches
// only, no allocation.  `bits` must give an even number of passes so the
// result ends in key/val.
void radix_sort_pairs_scratch(uint64_t *key, int32_t *val, uint64_t *key_tmp, int32_t *val_tmp, uint32_t *hist,
                              int64_t n, int bits, cudaStream_t stream) {
    if (n <= 1) return;
    int nb = (int)((n + RS_TILE - 1) / RS_TILE);
    int passes = (bits + 7) / 8;
    uint64_t *ka = key, *kb = key_tmp;
    int32_t *va = val, *vb = val_tmp;
    for (int p = 0; p < passes; p++) {
        int shift = 8 * p;
        k_rs_hist<<<nb, RS_THREADS, 0, stream>>>(ka, n, shift, hist, nb);
        KIFMM_LAUNCHED();
        k_rs_scan<<<256, 256, 0, stream>>>(hist, nb);
        KIFMM_LAUNCHED();
        k_rs_scatter<true><<<nb, RS_THREADS, 0, stream>>>(ka, va, kb, vb, n, shift, hist, nb);
        KIFMM_LAUNCHED();
        uint64_t *tk = ka; ka = kb; kb = tk;
        int32_t *tv = va; va = vb; vb = tv;
    }
}

}  // namespace kifmm
