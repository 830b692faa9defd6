// pair_f64.cuh -- FP64 kernel values for the pair loops (P2M, L2P, P2P).
//
// On sm_100a an SM issues 64 FP64 multiply-adds per clock (one warp instruction
// takes two issue slots of its scheduler) but only 16 FP64 conversions, and the
// CUDA math library's log, sqrt and Bessel functions cost 15 to 50 multiply-adds
// a call (measured, lane-operations per clock and SM: log 1.27, rsqrt 5.9, sqrt
// 4.4, int -> double 15.4, fma 60).  The values here take r^2 (no square root),
// one conflict-free table read and 8 FP64 instructions for the logarithm, and
// short power series beside it.
#pragma once
#include "kifmm_internal.cuh"

namespace kifmm {

// Natural logarithm of a positive normal number, table-driven (P. T. P. Tang,
// "Table-driven implementation of the logarithm function in IEEE
// floating-point arithmetic", ACM TOMS 16, 1990): x = 2^e m with m in
// [0.699, 1.398), so that e = 0 around 1 and nothing cancels there; v_i = 1/c_i
// rounded to FP64, c_i the midpoint of m's subinterval, r = m v_i - 1 (|r| <
// 2^-9), ln x = e ln2 - ln v_i + log1p(r).  The subinterval that holds 1 has v = 1,
// so its values are log1p(r) alone.  log1p(r) / r is its series to r^4 with the
// next term economised by the Chebyshev polynomial T5 (r^5 = h^5 (T5(r/h) + 20
// (r/h)^3 - 5 r/h) / 16, h = 2^-9).  Error against 113-bit values, 400,000
// samples a range: at most 4.0 ulp within 0.4% of 1 (mean 0.9), 1.6 elsewhere
// (mean 0.26 over 2^-30 .. 2^5).  With m in [1, 2) and half as many subintervals,
// at the same number of instructions but one, the error was 1e-16 absolutely, of
// any relative size beside 1.
// e is converted on the XU pipe, beside the FP64 pipe.
// The table is kept LOGTAB_COPIES times in shared memory, copy c in the 16-byte
// bank group c: a warp's 32 16-byte reads, eight to a phase, hit eight
// different groups whatever their entries (one copy measured 2-3 way
// conflicts, and the reads would then bound the loop instead of the FP64 pipe).
constexpr int LOGTAB_N = 256, LOGTAB_COPIES = 8;
constexpr double LOG_H2 = 1.0 / 262144.0;     // h^2
constexpr unsigned LOG_M_HI = 0x3fe65800u;    // high word of the least m: 1.0 lies in the middle of subinterval 154
constexpr unsigned LOG_STEP_HI = 0x00100000u / LOGTAB_N;  // high words of a subinterval
// the polynomial's coefficients r .. r^4 and ln 2, in constant memory, so
// that they are operands of the multiply-adds
enum { LOG_C2, LOG_C3, LOG_C4, LOG_C5, LOG_LN2 };
static __device__ __constant__ double LOG_K[] = {-0.5 + LOG_H2 * LOG_H2 * 5.0 / 96.0, 1.0 / 3.0,
                                                 -0.25 - LOG_H2 * 20.0 / 96.0, 0.2,
                                                 0.693147180559945309417232121458176568};

// log_table(device) holds [LOGTAB_N] (v_i, -ln v_i); stage its copies into
// tab[LOGTAB_N * LOGTAB_COPIES] (all threads of the block; the lanes of a warp write
// their copies in different bank groups)
__device__ __forceinline__ void stage_log_table(double2 *tab, const double2 *__restrict__ g) {
    for (int i = threadIdx.x; i < LOGTAB_N; i += blockDim.x) {
        const double2 v = g[i];
#pragma unroll
        for (int c = 0; c < LOGTAB_COPIES; c++) tab[i * LOGTAB_COPIES + ((c + i) & (LOGTAB_COPIES - 1))] = v;
    }
}

// ln(2^EADJ x); tl: this lane's copy, tab + (lane & 7).  x positive, normal,
// finite; anything else gives a finite or NaN value and reads inside the table.
template <int EADJ>
__device__ __forceinline__ double ln_tab(double x, const double2 *tl) {
    // t: e + EADJ above 20 bits of the distance from the least m
    const unsigned t = (unsigned)__double2hiint(x) - (LOG_M_HI - ((unsigned)EADJ << 20));
    constexpr unsigned ROW = LOGTAB_COPIES * sizeof(double2);  // bytes of an entry's copies
    static_assert(LOGTAB_N * ROW == 0x8000 && ROW == 0x80 && LOG_STEP_HI == 0x1000, "the shift and mask below");
    const double2 c = *(const double2 *)((const char *)tl + ((t >> 5) & 0x7f80u));
    const double m = __hiloint2double((int)((t & 0x000fffffu) + LOG_M_HI), __double2loint(x));
    const double e = (double)((int)t >> 20);
    const double r = fma(m, c.x, -1.0);
    double q = LOG_K[LOG_C5];
    q = fma(q, r, LOG_K[LOG_C4]);
    q = fma(q, r, LOG_K[LOG_C3]);
    q = fma(q, r, LOG_K[LOG_C2]);
    q = fma(q, r, 1.0);
    return fma(q, r, fma(e, LOG_K[LOG_LN2], c.y));
}

// Number of series terms that reach FP64 precision for t = (k r)^2 below
// 2^-4, 1 and 4: the terms are at most (H_n - gamma) t^n / (4^n (n!)^2).
constexpr int SERIES_NARROW = 7, SERIES_MID = 10, SERIES_WIDE = 13;
// high words of the bounds of t (t < bound iff hiword(t) < these)
constexpr unsigned SERIES_NARROW_HI = 0x3fb00000u, SERIES_MID_HI = 0x3ff00000u, SERIES_WIDE_HI = 0x40100000u;
template <int NT>
__device__ __forceinline__ double series(const double *c, double t) {
    double a = c[NT - 1];
#pragma unroll
    for (int i = NT - 2; i >= 0; i--) a = fma(a, t, c[i]);
    return a;
}

// The fast values are for t = r^2 (Laplace) or (k r)^2 that is a positive
// normal number below the bound whose high word is hi_end: those whose
// pair_rank is below hi_end - 2^20.
__device__ __forceinline__ unsigned pair_rank(double t) { return (unsigned)(__double2hiint(t) - 0x00100000); }
__device__ __forceinline__ bool pair_ordinary(double t, unsigned hi_end) { return pair_rank(t) < hi_end - 0x00100000u; }
constexpr unsigned LOG_HI_END = 0x7ff00000u;  // every finite number

// k^2 for (k r)^2.  Where it would lose bits (k below 1.5e-154) it is 0, which makes
// no pair ordinary: pair_value_any takes k r.
__device__ __forceinline__ double pair_k2(double k) {
    const double k2 = k * k;
    return k2 < 2.2250738585072014e-308 ? 0.0 : k2;
}

// Unscaled kernel value: re = ln r^2 (Laplace, times -1/(4 pi)), K0(k r) =
// P(t) - ln(t/4) I0(t)/2 (times 1/(2 pi)), or the real part of (i/4) H0(k r),
// ln(t/4) A(t) + R(t), whose imaginary part is -pi a with a = A(t).
struct PairValue {
    double re, a;
};
template <int KIND, int NT>
__device__ __forceinline__ PairValue pair_value(double t, const double2 *tl) {
    if (KIND == KIFMM_KERNEL_LAPLACE) return {ln_tab<0>(t, tl), 0.0};
    const double ln4 = ln_tab<-2>(t, tl);
    if (KIND == KIFMM_KERNEL_MOD_HELMHOLTZ) return {fma(ln4, series<NT>(K0_I0H_D, t), series<NT>(K0_P_D, t)), 0.0};
    const double a = series<NT>(H0_A_D, t);
    return {fma(ln4, a, series<NT>(H0_R_D, t)), a};
}
template <int KIND>
__device__ __forceinline__ double pair_scale() {
    return KIND == KIFMM_KERNEL_LAPLACE ? -0.07957747154594767
                                        : KIND == KIFMM_KERNEL_MOD_HELMHOLTZ ? 0.15915494309189535 : 1.0;
}
// K0(sqrt(t)) for t >= 4: exp(-x) / sqrt(x) F(4/x - 1), F as one polynomial
// (24 multiply-adds; Clenshaw's recurrence on its Chebyshev series takes 50),
// x = sqrt(t) and 1/x from one reciprocal square root
__device__ __forceinline__ double k0_far(double t) {
    const double y = rsqrt(t);
    double x = t * y;
    x = fma(0.5 * y, fma(-x, x, t), x);
    const double u = fma(4.0, y, -1.0);
    return exp(-x) * rsqrt(x) * series<K0_FAR_D_N>(K0_FAR_D, u);
}
// (i/4) H0(sqrt(t)) for 4 <= t < 64 (A and R as polynomials about t = 34) and
// for t >= 64 (Hankel's form).  CUDA's j0 and y0 are good to 5e-12 absolutely
// beyond 8; this is good to a few 1e-17, at about half the instructions of the
// two calls.
__device__ __forceinline__ PairValue h0_far(double t) {
    if (t < 64.0) {
        const double u = fma(t, 1.0 / 30.0, -34.0 / 30.0), a = series<H0_MID_A_D_N>(H0_MID_A_D, u);
        return {fma(log(0.25 * t), a, series<H0_MID_R_D_N>(H0_MID_R_D, u)), a};
    }
    const double y = rsqrt(t);
    double x = t * y;
    x = fma(0.5 * y, fma(-x, x, t), x);
    const double v = fma(128.0 * y, y, -1.0);
    const double p = series<H0_P_D_N>(H0_P_D, v), q = series<H0_Q_D_N>(H0_Q_D, v) * y;
    double s, c;
    sincos(x, &s, &c);
    const double m = 0.5641895835477563 * rsqrt(x), cs = c + s, sc = s - c;  // 1 / sqrt(pi x)
    return {-0.25 * m * fma(p, sc, q * cs), -0.07957747154594767 * m * fma(p, cs, -q * sc)};
}
// ... past the series, where the loops evaluate it in line: K0 for 4 <= t <
// 1e300, H0 for 4 <= t < 64 (h0_far's first form, with the table logarithm)
template <int KIND>
__device__ __forceinline__ PairValue pair_value_beyond(double t, const double2 *tl) {
    if (KIND == KIFMM_KERNEL_MOD_HELMHOLTZ) return {k0_far(t), 0.0};
    const double u = fma(t, 1.0 / 30.0, -34.0 / 30.0), a = series<H0_MID_A_D_N>(H0_MID_A_D, u);
    return {fma(ln_tab<-2>(t, tl), a, series<H0_MID_R_D_N>(H0_MID_R_D, u)), a};
}
template <int KIND>
__device__ __forceinline__ bool pair_beyond(double t) {
    return t >= 4.0 && t < (KIND == KIFMM_KERNEL_MOD_HELMHOLTZ ? 1e300 : 64.0);
}
// ... of any other pair (coincident points, underflow, k r >= 2); kept out of
// line, so that the pair loops stay small
template <int KIND>
__device__ __noinline__ PairValue pair_value_any(double r2, double k) {
    if (KIND == KIFMM_KERNEL_LAPLACE) return {log(r2), 0.0};
    if (KIND == KIFMM_KERNEL_MOD_HELMHOLTZ) {
        const double t = r2 * (k * k);
        return {t >= 4.0 && t < 1e300 ? k0_far(t) : k0_d(k * sqrt(r2)), 0.0};
    }
    const double t = r2 * (k * k);
    if (t >= 4.0 && t < 1e300) return h0_far(t);
    const double2 g = green_c(k, r2);
    return {g.x, -0.3183098861837907 * g.y};
}

}  // namespace kifmm
