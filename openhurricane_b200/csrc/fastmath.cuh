// FP64 exponential, logarithm, reciprocal and fall-off forms of the chemistry kernels.
#pragma once

#include <cmath>

#include "rtc_base.cuh"

namespace hc {

// e^r and the integer n of x = n ln 2 + r, |r| <= ln 2 / 2, |x| <= 800 or NaN: the
// Taylor series to degree 13 (truncation 4e-18), even and odd terms apart, so that
// the chain of dependent FP64 operations is half that of one Horner scheme
__device__ __forceinline__ double exp_reduced(double x, int &n) {
    const double big = 6755399441055744.0;                 // 1.5 * 2^52: rounds to an integer in the low word
    const double t = fma(x, 1.4426950408889634074, big);
    const double k = t - big;
    double r = fma(-k, 0x1.62e42feep-1, x);                // ln 2 in two parts, k times the first exact
    r = fma(-k, 0x1.a39ef35793c76p-33, r);
    const double r2 = r * r;
    double od = fma(r2, 1.0 / 6227020800.0, 1.0 / 39916800.0), ev = fma(r2, 1.0 / 479001600.0, 1.0 / 3628800.0);
    od = fma(od, r2, 1.0 / 362880.0);
    ev = fma(ev, r2, 1.0 / 40320.0);
    od = fma(od, r2, 1.0 / 5040.0);
    ev = fma(ev, r2, 1.0 / 720.0);
    od = fma(od, r2, 1.0 / 120.0);
    ev = fma(ev, r2, 1.0 / 24.0);
    od = fma(od, r2, 1.0 / 6.0);
    ev = fma(ev, r2, 0.5);
#ifdef __CUDA_ARCH__
    n = __double2loint(t);
#else
    n = isnan(x) ? 0 : (int)k;
#endif
    return 1.0 + fma(r2, fma(od, r, ev), r);
}

// exp(x) without a branch, so that several interleave where a chain's latency counts
// (the library's exp takes 157 cycles on a B200, this one about 100). 2^n is applied
// in two exact factors: overflow gives infinity, results below the normal range round
// twice. Within 1 ulp of the exact value (test_fastmath_host.py compiles it for the host).
__device__ __forceinline__ double fast_exp(double x) {
    x = (x > 800.0) ? 800.0 : x;                           // NaN stays
    x = (x < -800.0) ? -800.0 : x;
    int n;
    const double e = exp_reduced(x, n);
    const int n1 = n >> 1;
#ifdef __CUDA_ARCH__
    return (e * __hiloint2double((n1 + 1023) << 20, 0)) * __hiloint2double((n - n1 + 1023) << 20, 0);
#else
    return ldexp(ldexp(e, n1), n - n1);
#endif
}

// the same value with fewer instructions, where throughput counts: 2^n goes into the
// exponent field, and arguments beyond +-700 and NaN branch to the long form
static __device__ HC_NOINLINE double exp_far(double x) { return fast_exp(x); }

__device__ __forceinline__ double lean_exp(double x) {
    if (!(fabs(x) < 700.0)) return exp_far(x);
    int n;
    const double e = exp_reduced(x, n);
#ifdef __CUDA_ARCH__
    return __hiloint2double(__double2hiint(e) + (n << 20), __double2loint(e));
#else
    return ldexp(e, n);
#endif
}

// 1/b for positive normal b: the hardware approximation and one cubic step
// r (1 + e + e^2), e = 1 - b r, which triples its correct bits (frcp, rtc_base.cuh)
__device__ __forceinline__ double fast_rcp(double b) {
#ifdef __CUDA_ARCH__
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    const double e = fma(-b, r, 1.0);
    return fma(r, fma(e, e, e), r);
#else
    return 1.0 / b;
#endif
}

// ln x = e ln 2 + ln(1 + f) with 1 + f in [sqrt 1/2, sqrt 2): with s = f / (2 + f),
// ln(1 + f) = f - (f^2/2 - s (f^2/2 + R)), R = 2/3 s^2 + 2/5 s^4 + ... (the series of
// 2 artanh s; ten terms, truncation 1e-18), in two chains like fast_exp and without a
// branch (the library's log takes 294 cycles on a B200). Within 1 ulp of the exact value.
// The reduction, ln 2 in two parts and the order of the last sum are those of fdlibm's log
// (K. C. Ng, SunSoft 1993); its fitted coefficients are not used.
__device__ __forceinline__ double fast_log(double x) {
    const bool low = x < 2.2250738585072014e-308;          // below the normal range (or not positive)
    const double xs = low ? x * 18014398509481984.0 : x;   // 2^54
#ifdef __CUDA_ARCH__
    const int hi = __double2hiint(xs), e0 = (hi - 0x3fe6a09e) >> 20;
    const double f = __hiloint2double(hi - (e0 << 20), __double2loint(xs)) - 1.0;
#else
    int e0;
    double mant = frexp(xs, &e0);                          // [1/2, 1)
    if (mant < 0.70710678118654752) {
        mant *= 2.0;
        --e0;
    }
    const double f = mant - 1.0;
#endif
    const double n = (double)(low ? e0 - 54 : e0);
    const double s = f * fast_rcp(2.0 + f), z = s * s, z2 = z * z;
    double od = fma(z2, 2.0 / 21.0, 2.0 / 17.0), ev = fma(z2, 2.0 / 19.0, 2.0 / 15.0);
    od = fma(od, z2, 2.0 / 13.0);
    ev = fma(ev, z2, 2.0 / 11.0);
    od = fma(od, z2, 2.0 / 9.0);
    ev = fma(ev, z2, 2.0 / 7.0);
    od = fma(od, z2, 2.0 / 5.0);
    ev = fma(ev, z2, 2.0 / 3.0);
    const double R = z * fma(od, z, ev);
    const double h = 0.5 * f * f;
    const double v = fma(n, 0x1.62e42feep-1, f - (h - fma(s, h + R, n * 0x1.a39ef35793c76p-33)));
    // +inf and NaN are their own logarithms; zero: -inf, negative: NaN
    const double special = (x == 0.0) ? -(double)INFINITY : (x < 0.0) ? (double)NAN : x;
    return (x > 0.0 && x <= 1.7976931348623157e308) ? v : special;
}

// Fall-off rates (unimolecularFallOffRR.cpp:37-91, fallOffFunctions.cpp:81-157), k =
// kinf w with w = F Pr / (1 + Pr), Pr = ratio M, ratio = k0 / kinf; q = w times the rest:
//   w, and for the Jacobian dq/dc_i = eff_i q gM (gM = d ln w / dM) and the part
//   q wT of dq/dT that comes through Pr and F (wT = d ln w / dT).
// The formulas are the reference's with F, Pr and their reciprocals cancelled where
// they divide themselves out, so that five independent reciprocals are left of a
// chain of a dozen. Both derivatives are zero when M <= tiny, as in the reference.
struct FallOff {
    double w, gM, wT;
};

// e1, e2, e3: the Troe centering exponentials exp(-T/T***), exp(-T/T*), exp(-T**/T)
// (e3 = 0 for three parameters); dlr = d ln ratio / dT.
template <bool JAC>
__device__ __forceinline__ FallOff fall_off(bool troe, double alpha, double iTsss, double iTs, double Tss, double e1,
                                            double e2, double e3, double ratio, double M, double dlr, double invT) {
    FallOff o;
    const double Pr = ratio * M, iP = frcp(1.0 + Pr);
    double F = 1.0, FP = 0.0, FT = 0.0;                    // d ln F / d ln Pr, d ln F / dT at fixed dlr
    if (troe) {
        const double ln10 = 2.302585092994045684, lg = 0.4342944819032518277;
        const double a1 = (1.0 - alpha) * e1, a2 = alpha * e2;
        const double Fc = hmax(a1 + a2 + e3, kTiny);
        const double lf = lg * fast_log(Fc), lp = lg * fast_log(hmax(Pr, kTiny));
        const double u = lp - 0.4 - 0.67 * lf, v = 0.75 - 1.27 * lf - 0.14 * u;
        const double iv = frcp(v), is = v * v * fast_rcp(fma(u, u, v * v));    // 1 / (1 + (u/v)^2)
        F = fast_exp(ln10 * lf * is);
        if (JAC) {
            const double dlf = (e3 * (Tss * invT * invT) - a1 * iTsss - a2 * iTs) * (lg * fast_rcp(Fc));
            const double x = u * iv, c = (2.0 * u * iv * iv) * (lf * is * is);
            const double t = lg * dlr - 0.67 * dlf;
            FP = -c * (1.0 + 0.14 * x);
            FT = ln10 * (dlf * is - c * (t - x * (-1.27 * dlf - 0.14 * t)));
        }
    }
    o.w = Pr * iP * F;
    o.gM = o.wT = 0.0;
    if (JAC) {
        const double gM = (iP + FP) * fast_rcp(hmax(M, kTiny)), wT = dlr * iP + FT;
        o.gM = (M > kTiny) ? gM : 0.0;
        o.wT = (M > kTiny) ? wT : 0.0;
    }
    return o;
}

}  // namespace hc
