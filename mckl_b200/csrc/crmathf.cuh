// crmathf.cuh -- log, exp, sin and cos of floats, evaluated in double and
// rounded once.
//
// A double library function is within an ULP or two of the exact value, and the
// float nearest to its result differs from the float nearest to any other value
// within 2^-40 relative only where a midpoint of two floats lies between them.
// So a short evaluation with an error below 2^-43 relative gives the same float
// whenever its 29 bits below the float's last one are further than 2^12 units
// (2^-40 relative) from that midpoint; one argument in 65,000 is not, and its
// caller takes the library function.  (The inputs are single: the reductions
// need no double-double, and there are no special cases in the ranges below.)
// About 13 (log), 12 (exp) and 24 (both of sin and cos) FP64 operations.
#pragma once

#include "crmath.cuh"

namespace mckl_b200 {
namespace dd {

#if defined(__CUDA_ARCH__)
#define MB_TO_FLOAT(y) __double2float_rn(y)
#define MB_FLOAT_BITS(a) __float_as_uint(a)
#else
#define MB_TO_FLOAT(y) static_cast<float>(y)
inline unsigned host_float_bits(float a)
{
    unsigned u;
    __builtin_memcpy(&u, &a, 4);
    return u;
}
#define MB_FLOAT_BITS(a) ::mckl_b200::dd::host_float_bits(a)
#endif

// *f = y rounded to float; false where a value within 2^12 units of y's last
// place may round to another float.  y is zero or rounds to a normal float.
MB_HD bool round_float(double y, float *f)
{
    const unsigned low = static_cast<unsigned>(MB_AS_BITS(y)) & 0x1fffffffu;
    *f = MB_TO_FLOAT(y);
    return low - (0x10000000u - 0x1000u) > 0x2000u;
}

// log of a positive normal float.  a = 2^e m; r = m inv_i - 1 from the table of
// log (exact, |r| <= 2^-7); log1p(r) to r^7 (truncation 2^-52 relative).  Near 1
// the table's entries (inv = 1 from above, 1/2 from below) make e ln2 - ln inv
// vanish exactly, so the sum is log1p(r) alone.  In the other cells the result is
// above 2^-8 and the sum's absolute error below 2^-51 max(1, |e|).
MB_HD bool log_float(float a, float *f)
{
    const unsigned u = MB_FLOAT_BITS(a);
    if (u - 0x00800000u >= 0x7f000000u) return false;  // zero, subnormal, negative, infinite, NaN
    const double e = MB_SUB(MB_FROM_BITS(0x4330000000000000ll | (u >> 23)), 0x1p52 + 127.0);
    const int i = static_cast<int>((u >> 16) & 127u);
    const double m = MB_FROM_BITS(static_cast<long long>(0x3ff0000000000000ull | static_cast<unsigned long long>(u & 0x7fffffu) << 29));
    const double r = MB_FMA(m, MB_LOGTAB(i, 0), -1.0);
    double P = 0x1.2492492492492p-3;         // 1/7
    P = MB_FMA(P, r, -0x1.5555555555555p-3);  // -1/6
    P = MB_FMA(P, r, 0x1.999999999999ap-3);   // 1/5
    P = MB_FMA(P, r, -0x1.0000000000000p-2);  // -1/4
    P = MB_FMA(P, r, 0x1.5555555555555p-2);   // 1/3
    P = MB_FMA(P, r, -0.5);
    const double q = MB_FMA(MB_MUL(r, r), P, r);
    const double t = MB_ADD(MB_FMA(e, kLn2Hi, MB_LOGTAB(i, 1)), MB_FMA(e, kLn2Lo, MB_LOGTAB(i, 2)));
    return round_float(MB_ADD(t, q), f);
}

// exp of a float in (-87, 87) (normal results): x = k ln2/64 + r, |r| <= ln2/128,
// 2^(j/64) (1 + r + ... + r^5/120) 2^m (truncation below 2^-54).
MB_HD bool exp_float(float a, float *f)
{
    if ((MB_FLOAT_BITS(a) & 0x7fffffffu) >= 0x42ae0000u) return false;
    const double x = static_cast<double>(a);
    int k;
    const double kd = round_int(MB_MUL(x, kExpInvL), &k);
    const double r = MB_FMA(-kd, kExpL2, MB_FMA(-kd, kExpL1, x));
    double P = 0x1.1111111111111p-7;         // 1/120
    P = MB_FMA(P, r, 0x1.5555555555555p-5);  // 1/24
    P = MB_FMA(P, r, 0x1.5555555555555p-3);  // 1/6
    P = MB_FMA(P, r, 0.5);
    const double T = MB_EXPTAB(k & 63, 0);
    const double y = MB_FMA(T, MB_FMA(MB_MUL(r, r), P, r), T);
    return round_float(MB_FROM_BITS(MB_AS_BITS(y) + (static_cast<long long>(k >> 6) << 52)), f);
}

// sin and cos of a float with 2^-60 <= |a| < 16 (an angle of a Box-Muller pair):
// r = a - k pi/2 in three parts, then the series to r^13 and r^14 (truncation
// below 2^-44.9 of sin and 2^-49 of cos for |r| <= pi/4).
MB_HD bool sincos_float(float a, float *sp, float *cp)
{
    if ((MB_FLOAT_BITS(a) & 0x7fffffffu) - 0x21800000u >= 0x41800000u - 0x21800000u) return false;
    const double x = static_cast<double>(a);
    int q;
    const double kd = round_int(MB_MUL(x, kTwoOverPi), &q);
    const double r = MB_FMA(-kd, kPio2P3, MB_FMA(-kd, kPio2P2, MB_FMA(-kd, kPio2P1, x)));
    const double w = MB_MUL(r, r);
    double S = 0x1.6124613a86d09p-33;            // 1/13!
    S = MB_FMA(S, w, -0x1.ae64567f544e4p-26);    // -1/11!
    S = MB_FMA(S, w, 0x1.71de3a556c734p-19);     // 1/9!
    S = MB_FMA(S, w, -0x1.a01a01a01a01ap-13);    // -1/7!
    S = MB_FMA(S, w, 0x1.1111111111111p-7);      // 1/5!
    S = MB_FMA(S, w, -0x1.5555555555555p-3);     // -1/3!
    const double s = MB_FMA(MB_MUL(r, w), S, r);
    double C = -0x1.93974a8c07c9dp-37;           // -1/14!
    C = MB_FMA(C, w, 0x1.1eed8eff8d898p-29);     // 1/12!
    C = MB_FMA(C, w, -0x1.27e4fb7789f5cp-22);    // -1/10!
    C = MB_FMA(C, w, 0x1.a01a01a01a01ap-16);     // 1/8!
    C = MB_FMA(C, w, -0x1.6c16c16c16c17p-10);    // -1/6!
    C = MB_FMA(C, w, 0x1.5555555555555p-5);      // 1/4!
    C = MB_FMA(C, w, -0.5);
    const double c = MB_FMA(w, C, 1.0);
    float fs, fc;
    const bool oks = round_float(s, &fs), okc = round_float(c, &fc);
    const bool swap = (q & 1) != 0;
    *sp = swap ? fc : fs;
    *cp = swap ? fs : fc;
    if (q & 2) *sp = -*sp;
    if ((q + 1) & 2) *cp = -*cp;
    return oks && okc;
}

}  // namespace dd

#if defined(__CUDACC__)
// log(u) < lr for u = (w + 1/2) 2^-32, as the double logarithm decides it.
// The single-precision logarithm of u is within 1e-5 of log u (rounding u:
// 2^-23 relative; __logf: 2^-21.4 absolute for u in [0.5, 1], 3 ulps of at most
// 23 below), so it decides whenever lr is further away than that (rounding lr
// to float is below 2e-6 for |lr| <= 32); a NaN goes to the double comparison.
__device__ __forceinline__ bool log_less(uint32_t w, double lr)
{
    const float u = __fmul_rn(__fadd_rn(__uint2float_rn(w), 0.5f), 0x1p-32f);
    const float d = __fsub_rn(__double2float_rn(lr), __logf(u));
    if (fabsf(d) > 1e-4f) return d > 0.0f;
    return ::log((static_cast<double>(w) + 0.5) * 0x1p-32) < lr;
}
#endif

}  // namespace mckl_b200
