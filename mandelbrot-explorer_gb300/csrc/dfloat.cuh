// Double-float arithmetic: a value is hi + lo with two floats, |lo| <= ulp(hi)/2,
// giving about 48 significant bits on the FP32 pipe. On GB300 FP64 issues at
// 1/64 of the FP32 rate and a single warp's FP64 dependency chain is long, so
// the lane that reruns the samples the FP32 pass cannot vouch for computes in
// this type. The error-free transformations are the published ones (Knuth's
// TwoSum, Dekker's Fast2Sum, the FMA-based TwoProd); addition is the "sloppy"
// variant (error bounded relative to |a| + |b|), multiplication and division
// follow the usual double-double construction reduced to float pairs.
#pragma once
#include <math.h>

#include <cuda_runtime.h>

#include "floatexp.h"

namespace mbx {

struct df32 {
    float hi, lo;
    df32() = default;
    MBX_HD constexpr df32(float h, float l) : hi(h), lo(l) {}
    MBX_HD constexpr df32(float x) : hi(x), lo(0.0f) {}
    MBX_HD constexpr df32(int x) : hi((float)x), lo(0.0f) {}
    MBX_HD df32(double x) : hi((float)x), lo((float)(x - (double)(float)x)) {}
    MBX_HD explicit operator double() const { return (double)hi + (double)lo; }
    MBX_HD explicit operator float() const { return hi + lo; }
};

struct df2 {
    df32 x, y;
};

MBX_HD float df_fma(float a, float b, float c) {
#ifdef __CUDA_ARCH__
    return __fmaf_rn(a, b, c);
#else
    return fmaf(a, b, c);
#endif
}
// s + e = a + b exactly (Knuth).
MBX_HD df32 df_two_sum(float a, float b) {
    const float s = a + b;
    const float bb = s - a;
    const float e = (a - (s - bb)) + (b - bb);
    return df32(s, e);
}
// s + e = a + b exactly for |a| >= |b| (Dekker).
MBX_HD df32 df_fast_two_sum(float a, float b) {
    const float s = a + b;
    return df32(s, b - (s - a));
}
MBX_HD df32 operator+(df32 a, df32 b) {
    const df32 s = df_two_sum(a.hi, b.hi);
    return df_fast_two_sum(s.hi, s.lo + (a.lo + b.lo));
}
MBX_HD df32 operator-(df32 a) { return df32(-a.hi, -a.lo); }
MBX_HD df32 operator-(df32 a, df32 b) { return a + (-b); }
MBX_HD df32 operator*(df32 a, df32 b) {
    const float p = a.hi * b.hi;
    float e = df_fma(a.hi, b.hi, -p);
    e = df_fma(a.hi, b.lo, df_fma(a.lo, b.hi, e));
    return df_fast_two_sum(p, e);
}
// (division and square root are called, not inlined: the lanes that use them are
// bound by instruction fetch, mixed_lane.cuh)
#ifdef __CUDACC__
#define MBX_DF_CALL __host__ __device__ __noinline__ inline
#else
#define MBX_DF_CALL inline
#endif
MBX_DF_CALL df32 operator/(df32 a, df32 b) {
    const float q1 = a.hi / b.hi;
    const df32 r = a - b * df32(q1);
    const float q2 = (r.hi + r.lo) / b.hi;
    return df_fast_two_sum(q1, q2);
}
MBX_HD df32& operator+=(df32& a, df32 b) { return a = a + b; }
MBX_HD df32& operator-=(df32& a, df32 b) { return a = a - b; }
MBX_HD df32& operator*=(df32& a, df32 b) { return a = a * b; }
MBX_HD bool operator<(df32 a, df32 b) { return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo); }
MBX_HD bool operator>(df32 a, df32 b) { return b < a; }
MBX_HD bool operator<=(df32 a, df32 b) { return !(b < a); }
MBX_HD bool operator>=(df32 a, df32 b) { return !(a < b); }
MBX_HD bool operator==(df32 a, df32 b) { return a.hi == b.hi && a.lo == b.lo; }
MBX_HD bool operator!=(df32 a, df32 b) { return !(a == b); }

// Complex double-floats, real and imaginary part side by side: Blackwell's paired
// FP32 instructions take both parts' operations at once. Each part goes through
// the operations of operator+ and operator* above in their order (a difference
// a - b as fma(b, -1, a), one rounding). The unit that uses them is compiled with
// contraction, which fuses products into sums of the scalar forms and leaves the
// paired ones as they are written: their last bits can differ, about one value of
// a frame in a hundred moved by a bit, and errors against the exact form stayed
// the same (mean, 99 % and largest over some 30 outputs of zoom, minibrot, 1e-300
// frames and tiles: ratios of 1.000). Half the instructions matter because the
// lanes that use them wait for instruction fetch.
struct cdf {
    float2 hi, lo;
};
MBX_HD cdf cd_make(df32 r, df32 i) { return cdf{make_float2(r.hi, i.hi), make_float2(r.lo, i.lo)}; }
MBX_HD df32 cd_re(cdf z) { return df32(z.hi.x, z.lo.x); }
MBX_HD df32 cd_im(cdf z) { return df32(z.hi.y, z.lo.y); }
MBX_HD float2 f2_add(float2 a, float2 b) {
#ifdef __CUDA_ARCH__
    return __fadd2_rn(a, b);
#else
    return make_float2(a.x + b.x, a.y + b.y);
#endif
}
MBX_HD float2 f2_mul(float2 a, float2 b) {
#ifdef __CUDA_ARCH__
    return __fmul2_rn(a, b);
#else
    return make_float2(a.x * b.x, a.y * b.y);
#endif
}
MBX_HD float2 f2_fma(float2 a, float2 b, float2 c) {
#ifdef __CUDA_ARCH__
    return __ffma2_rn(a, b, c);
#else
    return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
#endif
}
MBX_HD float2 f2_sub(float2 a, float2 b) { return f2_fma(b, make_float2(-1.0f, -1.0f), a); }
MBX_HD cdf cd_fast_two_sum(float2 a, float2 b) {
    const float2 s = f2_add(a, b);
    return cdf{s, f2_sub(b, f2_sub(s, a))};
}
MBX_HD cdf operator+(cdf a, cdf b) {
    const float2 s = f2_add(a.hi, b.hi), t = f2_sub(s, a.hi);
    const float2 e = f2_add(f2_sub(a.hi, f2_sub(s, t)), f2_sub(b.hi, t));
    return cd_fast_two_sum(s, f2_add(e, f2_add(a.lo, b.lo)));
}
// part by part
MBX_HD cdf cd_mul(cdf a, cdf b) {
    const float2 p = f2_mul(a.hi, b.hi);
    float2 e = f2_fma(a.hi, b.hi, f2_mul(p, make_float2(-1.0f, -1.0f)));
    e = f2_fma(a.hi, b.lo, f2_fma(a.lo, b.hi, e));
    return cd_fast_two_sum(p, e);
}
MBX_HD cdf cd_scale(df32 a, cdf b) { return cd_mul(cd_make(a, a), b); }
// (ar br - ai bi, ar bi + ai br)
MBX_HD cdf cd_cmul(df32 ar, df32 ai, cdf b) {
    const cdf i{make_float2(-b.hi.y, b.hi.x), make_float2(-b.lo.y, b.lo.x)};
    return cd_scale(ar, b) + cd_scale(ai, i);
}
MBX_HD cdf cd_twice(cdf a) { return cdf{f2_add(a.hi, a.hi), f2_add(a.lo, a.lo)}; }

MBX_DF_CALL df32 tsqrt(df32 a) {
    if (!(a.hi > 0.0f)) return df32(0.0f);
    const float x = sqrtf(a.hi);
    const df32 r = a - df32(x) * df32(x);
    return df_fast_two_sum(x, (r.hi + r.lo) / (2.0f * x));
}
MBX_HD df32 tabs(df32 a) { return a.hi < 0.0f ? -a : a; }
MBX_HD df32 tmin(df32 a, df32 b) { return a < b ? a : b; }

} // namespace mbx
