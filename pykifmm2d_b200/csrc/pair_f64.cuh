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
// floating-point arithmetic", ACM TOMS 16, 1990): x = 2^e m with m in [1, 2),
// c_i = 1 + (i + 1/2)/128 the midpoint of m's subinterval, v_i = 1/c_i
// rounded to FP64, r = m v_i - 1 (|r| < 2^-8), ln x = e ln2 - ln v_i +
// log1p(r).  log1p is its series to r^6 with r^6 economised by the Chebyshev
// polynomial T6 (r^6 = h^6 (T6(r/h) + 48 (r/h)^4 - 18 (r/h)^2 + 1) / 32,
// h = 2^-8), so five coefficients leave 1.9e-17; the constant it leaves goes
// into the table.  Max error 1.6 ulp, mean 0.34 (against 60-digit values over
// 2^-30 .. 2^5).  e is converted on the XU pipe, beside the FP64 pipe.
// The table is kept LOGTAB_COPIES times in shared memory, copy c in the 16-byte
// bank group c: a warp's 32 16-byte reads, eight to a phase, hit eight
// different groups whatever their entries (one copy measured 2-3 way
// conflicts, and the reads would then bound the loop instead of the FP64 pipe).
constexpr int LOGTAB_N = 128, LOGTAB_COPIES = 8;
constexpr double LOG_H2 = 1.0 / 65536.0;  // h^2
// the polynomial's coefficients r^2 .. r^5 and ln 2, in constant memory, so
// that they are operands of the multiply-adds
enum { LOG_C2, LOG_C3, LOG_C4, LOG_C5, LOG_LN2 };
static __device__ __constant__ double LOG_K[] = {-0.5 + LOG_H2 * LOG_H2 * 18.0 / 192.0, 1.0 / 3.0,
                                                 -0.25 - LOG_H2 * 48.0 / 192.0, 0.2,
                                                 0.693147180559945309417232121458176568};

// log_table(device) holds [LOGTAB_N] (v_i, -ln v_i - h^6/192); stage its copies into tab[LOGTAB_N * LOGTAB_COPIES] (all threads of the block)
__device__ __forceinline__ void stage_log_table(double2 *tab, const double2 *__restrict__ g) {
    for (int i = threadIdx.x; i < LOGTAB_N * LOGTAB_COPIES; i += blockDim.x) tab[i] = g[i / LOGTAB_COPIES];
}

// ln(2^EADJ x); tl: this lane's copy, tab + (lane & 7).  x positive, normal,
// finite; anything else gives a finite or NaN value and reads inside the table.
template <int EADJ>
__device__ __forceinline__ double ln_tab(double x, const double2 *tl) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    constexpr unsigned ROW = LOGTAB_COPIES * sizeof(double2);  // bytes of an entry's copies
    static_assert(LOGTAB_N * ROW == 0x4000 && ROW == 0x80, "the shift and mask below");
    const double2 c = *(const double2 *)((const char *)tl + (((unsigned)hi >> 6) & 0x3f80u));
    const double m = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, lo);
    const double e = (double)((int)((unsigned)hi >> 20) - (1023 - EADJ));
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
