// The escape values' logarithms without FP64: the smooth count and the distance
// are floats rounded from double expressions of log |z|^2 (mp.cpp:371-398), some
// 90 and 60 FP64 instructions on GB300, whose FP64 unit takes one warp
// instruction per 64 cycles. In pairs of floats (color_math.cuh) the logarithms
// come within 2^-42, which settles the rounding to float on all but about one
// smooth count in 2^17 and one distance in 2^15 (whose window is taken wider);
// those take the double expression. So the values are the same floats. Host and device; compiled without FMA contraction.
#pragma once
#include "color_math.cuh"
#include "floatexp.h"

namespace mbx {

// 1 / ln 2 and 1 / (2 ln 2) as pairs (hi = RN(v), lo = RN(v - hi))
constexpr float kInvLn2Hi = 0x1.715476p+0f, kInvLn2Lo = 0x1.4ae0c0p-26f;

// Natural log of a double in [2, 2^240): its top 24 bits by log_ff, the rest to
// first order (below 2^-23 of the argument: the second order is below 2^-47).
MBX_HD cm::ff log_pair(double x) {
    const uint64_t b = dbits(x);
    const int k = (int)(b >> 52) - 1023;
    const float mh = cm::from_bits(0x3f800000u | ((unsigned)(b >> 29) & 0x7fffffu));
    const float ml = cm::mul((float)(unsigned)(b & 0x1fffffffu), 0x1p-52f);
    const cm::ff lm = cm::ff_add_f(cm::log_ff(mh), cm::div(ml, mh));
    return cm::ff_add(cm::ff_mul_f(cm::ff{cm::kLn2Hi, cm::kLn2Lo}, (float)k), lm);
}

MBX_HD bool log_pair_takes(double x) { return (unsigned)(dbits(x) >> 32) - 0x40000000u < 0x0f000000u; } // [2, 2^241)

// (float)(n - log(log(zrad) / 2 / ln 2) / ln 2)
MBX_HD bool smooth_pair(int n, double zrad, float& out) {
    if (!log_pair_takes(zrad) || (unsigned)n > (1u << 24)) return false;
    const cm::ff inv{kInvLn2Hi, kInvLn2Lo};
    const cm::ff l = log_pair(zrad);
    const cm::ff t = cm::ff_mul(cm::ff{cm::mul(l.hi, 0.5f), cm::mul(l.lo, 0.5f)}, inv); // log2 |z| >= 1/2
    const cm::ff x = cm::ff_mul(cm::ff_add_f(cm::log_ff(t.hi), cm::div(t.lo, t.hi)), inv);
    cm::ff v = cm::ff_add_f(cm::ff{-x.hi, -x.lo}, (float)n);
    const bool neg = v.hi < 0.0f;
    if (neg) v = cm::ff{-v.hi, -v.lo};
    // |log2 t| < 8: its pair is within 2^-41 (log_ff's 2^-44 of it and of t)
    if (!cm::round_within(v, 0x1p-40f, out)) return false;
    if (neg) out = -out;
    return true;
}

// (float)(sqrt(zrad) log(zrad) / sqrt(a a + b b)) as zrad rsqrt(zrad d2) log zrad
MBX_HD bool distance_pair(double zrad, double a, double b, float& out) {
    const double d2 = a * a + b * b, q = zrad * d2;
    // q within [2^-900, 2^1000): no term of it left the normal range
    if (!log_pair_takes(zrad) || !((unsigned)(dbits(q) >> 32) - 0x07b00000u < 0x76c00000u) || !((unsigned)(dbits(d2) >> 32) - 0x07b00000u < 0x76c00000u)) return false;
    const cm::ff l = log_pair(zrad);
#ifdef __CUDA_ARCH__
    const double r = rsqrt(q);
#else
    const double r = 1.0 / __builtin_sqrt(q);
#endif
    const double y = (zrad * r) * ((double)l.hi + (double)l.lo);
    // the float nearest to y, unless y is within 2^-40 of a midpoint or below the
    // normal floats (from 2^128 on: infinity)
    const uint64_t u = dbits(y);
    const unsigned e = (unsigned)(u >> 52), rest = (unsigned)u & 0x1fffffffu;
    if (e < 900u || rest - (0x10000000u - 0x2000u) < 0x4000u) return false; // (2^-123)
    out = cm::from_bits(e < 1151u ? ((e - 896u) << 23 | ((unsigned)(u >> 29) & 0x7fffffu)) + (rest >> 28) : 0x7f800000u);
    return true;
}

} // namespace mbx
