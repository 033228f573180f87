// Extended-exponent float (m * 2^e, 0.5 <= |m| < 1) and the complex helpers of
// the perturbation path, usable from host C++ and CUDA device code alike.
//
// Semantics follow the reference's src/engine/floatexp.h:17-107 operation by
// operation; frexp/ldexp are implemented on the IEEE bit patterns so that host
// and device produce identical bits (ldexp rounds to nearest-even in the
// subnormal range exactly like libm's). The exact form and the host compile it
// without FMA contraction (-ffp-contract=off / -fmad=false): there every
// operation's bits are part of the result. The lane passes compile it with
// contraction; the floatexp operations have no product that a sum could take in
// but exact ones (by powers of two), so theirs are the same.
#pragma once
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define MBX_HD __host__ __device__ __forceinline__
#else
#define MBX_HD inline
#endif

namespace mbx {

MBX_HD uint64_t dbits(double x) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    memcpy(&b, &x, 8);
    return b;
#endif
}
MBX_HD double bitsd(uint64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    memcpy(&x, &b, 8);
    return x;
#endif
}
MBX_HD double dabs(double x) { return bitsd(dbits(x) & 0x7fffffffffffffffull); }

// Comparisons on the bit patterns, with exactly the IEEE results (NaN
// included): integer compares, where an FP64 compare costs the latency of an
// FP64 add (64 cycles on GB300, against 4 for an FP32 FMA).
// x == 0.0 (either sign)
MBX_HD bool d_is_zero(double x) { return (dbits(x) << 1) == 0; }
// |a| < |b|; for a and b +0, positive or NaN (a sum of squares, a squared
// radius) this is a < b
MBX_HD bool d_abs_less(double a, double b) {
    const uint64_t ua = dbits(a) & 0x7fffffffffffffffull, ub = dbits(b) & 0x7fffffffffffffffull;
    return ua < ub && ub <= 0x7ff0000000000000ull;
}
// a == b (+0 equals -0, NaN equals nothing)
MBX_HD bool d_eq(double a, double b) {
    const uint64_t ua = dbits(a), ub = dbits(b);
    return (ua == ub && (ua & 0x7fffffffffffffffull) <= 0x7ff0000000000000ull) || ((ua | ub) << 1) == 0;
}
// x <= 0.0
MBX_HD bool d_le_zero(double x) {
    const uint64_t u = dbits(x);
    return (u << 1) == 0 || ((u >> 63) != 0 && (u & 0x7fffffffffffffffull) <= 0x7ff0000000000000ull);
}
// x + x, exactly as the FP64 add rounds it, on the bit pattern. (No FP64 add even
// for the rare cases: the compiler would execute it beside the common one.)
MBX_HD double d_twice(double x) {
    const uint64_t b = dbits(x);
    const uint64_t e = (b >> 52) & 0x7ff;
    if (e - 1 < 0x7fd) return bitsd(b + (1ull << 52)); // normal, result normal
    if (e == 0) // zero or subnormal: the magnitude shifts (a carry into the exponent gives the normal result)
        return bitsd((b & 0x8000000000000000ull) | ((b & 0x7fffffffffffffffull) << 1));
    if (e == 0x7fe) return bitsd((b & 0x8000000000000000ull) | 0x7ff0000000000000ull); // overflows to infinity
    return x; // infinity, NaN
}

// The floatexp operations run in the exact loop's serial chains, where an integer
// instruction costs its latency like an FP64 one (a BLA skip took some 750 of them
// beside 75 FP64 ones): each has one test for its common case (normal mantissas,
// in-range results) and leaves the others to a called function.
#ifdef __CUDACC__
#define MBX_COLD __host__ __device__ __noinline__ inline
#else
#define MBX_COLD inline
#endif

// frexp: x = r * 2^e with 0.5 <= |r| < 1; zero, inf and nan return x with e = 0.
struct FrexpOf {
    double m;
    int e;
};
MBX_COLD FrexpOf xfrexp_rare(double x) { // zero, subnormal, infinite, NaN
    uint64_t b = dbits(x);
    int ex = (int)((b >> 52) & 0x7ff);
    if (ex != 0 || (b << 1) == 0) return FrexpOf{x, 0};
    x = x * 18014398509481984.0; // 2^54, exact
    b = dbits(x);
    ex = (int)((b >> 52) & 0x7ff);
    return FrexpOf{bitsd((b & 0x800fffffffffffffull) | (1022ull << 52)), ex - 1022 - 54};
}
MBX_HD bool d_normal(uint64_t b) { return (unsigned)((b >> 52) & 0x7ff) - 1u < 0x7feu; }
MBX_HD double xfrexp(double x, int* e) {
    const uint64_t b = dbits(x);
    if (d_normal(b)) {
        *e = (int)((b >> 52) & 0x7ff) - 1022;
        return bitsd((b & 0x800fffffffffffffull) | (1022ull << 52));
    }
    const FrexpOf r = xfrexp_rare(x);
    *e = r.e;
    return r.m;
}

// Exact power of two 2^k for -1074 <= k <= 1023 (subnormal below -1022).
MBX_HD double pow2i(int k) {
    if (k >= -1022) return bitsd((uint64_t)(k + 1023) << 52);
    return bitsd(1ull << (k + 1074));
}

// ldexp for finite x, correctly rounded (one rounding in the subnormal range).
MBX_COLD double xldexp_rare(double x, int k) {
    if (d_is_zero(x)) return x;
    uint64_t b = dbits(x);
    if (((b >> 52) & 0x7ff) == 0x7ff) return x;
    int e;
    double m = xfrexp(x, &e); // |m| in [0.5,1)
    long long ne = (long long)e + k;   // value = m * 2^ne
    if (ne > 1024) return bitsd((b & 0x8000000000000000ull) | 0x7ff0000000000000ull);
    if (ne >= -1021) {                 // normal result, exact
        uint64_t mb = dbits(m);
        return bitsd((mb & 0x800fffffffffffffull) | ((uint64_t)(ne + 1022) << 52));
    }
    if (ne < -1074) return bitsd(b & 0x8000000000000000ull); // below half the smallest subnormal
    // 2^ne is exactly representable here; one multiply gives the one rounding.
    return m * pow2i((int)ne);
}
MBX_HD double xldexp(double x, int k) {
    const uint64_t b = dbits(x);
    // normal x, normal result: the exponent field moves
    if (d_normal(b) && (unsigned)((b >> 52) & 0x7ff) - 1u + (unsigned)k < 0x7feu) return bitsd(b + ((uint64_t)(int64_t)k << 52));
    return xldexp_rare(x, k);
}

// m 2^e. The exponent has 64 bits: a scale may be written 1e400000000, and |dz|^2
// of its frame is below 2^-(2^31). FEt<int> is for operands whose exponents are known
// to leave an int's range nowhere.
template <class E>
struct FEt {
    double m;
    E e;
};
using FE = FEt<int64_t>;

template <class E>
MBX_HD FEt<E> fe_make_as(double m, E e) {
    FEt<E> r;
    r.m = m;
    r.e = e;
    return r;
}
MBX_HD FE fe_make(double m, int64_t e) { return fe_make_as<int64_t>(m, e); }
template <class E>
MBX_HD FEt<E> fe_renorm_as(double m, E e) {
    const uint64_t b = dbits(m);
    if (d_normal(b)) return fe_make_as<E>(bitsd((b & 0x800fffffffffffffull) | (1022ull << 52)), e + (int)((b >> 52) & 0x7ff) - 1022);
    if (d_is_zero(m)) return fe_make_as<E>(0.0, 0);
    const FrexpOf r = xfrexp_rare(m);
    return fe_make_as<E>(r.m, e + r.e);
}
MBX_HD FE fe_renorm(double m, int64_t e) { return fe_renorm_as<int64_t>(m, e); }
MBX_HD FE fe_from(double x) { return fe_renorm(x, 0); }
template <class E>
MBX_COLD double fe_to_double_rare(FEt<E> a) {
    if (d_is_zero(a.m)) return 0.0;
    if (a.e > 1100) return bitsd(0x7ff0000000000000ull | (dbits(a.m) & 0x8000000000000000ull));
    if (a.e < -1100) return 0.0;
    return xldexp(a.m, (int)a.e);
}
template <class E>
MBX_HD double fe_to_double(FEt<E> a) {
    const uint64_t b = dbits(a.m);
    if (d_normal(b) && ((b >> 52) & 0x7ff) - 1u + (uint64_t)(int64_t)a.e < 0x7feu) return bitsd(b + ((uint64_t)(int64_t)a.e << 52));
    return fe_to_double_rare(a);
}
template <class E>
MBX_HD FEt<E> fe_mul(FEt<E> a, FEt<E> b) {
    if (d_is_zero(a.m) || d_is_zero(b.m)) return fe_make_as<E>(0.0, 0);
    return fe_renorm_as<E>(a.m * b.m, a.e + b.e);
}
template <class E>
MBX_HD FEt<E> fe_mul_d(FEt<E> a, double b) {
    if (d_is_zero(a.m) || d_is_zero(b)) return fe_make_as<E>(0.0, 0);
    return fe_renorm_as<E>(a.m * b, a.e);
}
template <class E>
MBX_HD FEt<E> fe_scale2(FEt<E> a, int64_t k) { return d_is_zero(a.m) ? a : fe_make_as<E>(a.m, a.e + (E)k); }
template <class E>
MBX_HD FEt<E> fe_add(FEt<E> a, FEt<E> b) {
    if (d_is_zero(a.m)) return b;
    if (d_is_zero(b.m)) return a;
    const E dw = a.e - b.e;
    if (dw > 54) return a;
    if (dw < -54) return b;
    const int d = (int)dw;
    // the smaller exponent's mantissa aligned to the larger (one add for both orders)
    const bool first = d >= 0;
    const double big = first ? a.m : b.m, small = xldexp(first ? b.m : a.m, first ? -d : d);
    return fe_renorm_as<E>(big + small, first ? a.e : b.e);
}
template <class E>
MBX_HD FEt<E> fe_neg(FEt<E> a) { return fe_make_as<E>(-a.m, a.e); }
template <class E>
MBX_HD FEt<E> fe_sub(FEt<E> a, FEt<E> b) { return fe_add(a, fe_neg(b)); }
// Quotient and square root on integers, correctly rounded, for normal operands
// and results. An FP64 division is some 9 FP64 instructions and a square root 10,
// each of which holds its SM quarter's FP64 unit for 64 cycles; a BLA skip of the
// exact loop took three divisions and a root, two thirds of its FP64
// instructions. These take some 35 integer ones each. Long division by digits: a
// 30-bit reciprocal (of b, of sqrt(x)) from a single-precision seed and one Newton
// step, a first digit of 30 bits, the exact remainder modulo 2^64 (its magnitude
// stays below 2^57), a second of 23 bits, and the rounding decided by the last
// remainder. The exact loop takes them (its pass over the 1,276 leftovers of the
// 1080p minibrot frame 24.5 -> 22.5 ms, over the 1080p frame at 1e-300 41.9 ->
// 39.8); the lanes' called functions keep the plain operations (with these the
// 1080p zoom frame took 24.7 ms instead of 23.4: more instructions to fetch).
MBX_COLD double div_rare(double a, double b) { return a / b; }
MBX_HD double int_div(double a, double b) {
    const uint64_t ua = dbits(a), ub = dbits(b), kOne = 1ull << 52, kFrac = kOne - 1;
    uint64_t A = (ua & kFrac) | kOne;
    const uint64_t B = (ub & kFrac) | kOne;
    const int below = A < B ? 1 : 0;
    const int e = (int)((ua >> 52) & 0x7ff) - (int)((ub >> 52) & 0x7ff) + 1023 - below;
    if (!(d_normal(ua) && d_normal(ub) && (unsigned)(e - 1) < 2046u)) return div_rare(a, b);
    A <<= below; // A / B in [1, 2)
    const uint32_t b32 = (uint32_t)(B >> 21);
    // r = 2^83 / B within 2.5: 30 bits
#ifdef __CUDA_ARCH__
    uint32_t r = (uint32_t)__fdividef(0x1p62f, (float)b32);
#else
    uint32_t r = (uint32_t)(0x1p62f / (float)b32);
#endif
    const int64_t d = (int64_t)((1ull << 62) - (uint64_t)r * b32); // |d| < 2^41
    r += (uint32_t)(int32_t)(((int64_t)(int32_t)(d >> 30) * (int64_t)r) >> 32);
    // A / B in units of 2^-29 within 5, the remainder below 5 B
    const uint32_t q0 = (uint32_t)(((A >> 22) * (uint64_t)r) >> 32);
    const int64_t r1 = (int64_t)((A << 29) - (uint64_t)q0 * B);
    // the next 23 bits: (R1 / B) 2^23 less c1 lies in (-0.3, 1.3)
    const int32_t c1 = (int32_t)(((int64_t)(int32_t)(r1 >> 25) * (int64_t)r) >> 35);
    const int64_t r2 = (int64_t)(((uint64_t)r1 << 23) - (uint64_t)(int64_t)c1 * B);
    // no quotient of two doubles lies halfway between two normal ones
    const uint64_t q = ((uint64_t)q0 << 23) + (uint64_t)(int64_t)c1 + (2 * r2 > (int64_t)B ? 1 : 0);
    return bitsd(((ua ^ ub) & 0x8000000000000000ull) | (((uint64_t)e << 52) + (q - kOne)));
}
MBX_COLD double sqrt_rare(double x) {
#ifdef __CUDA_ARCH__
    return __dsqrt_rn(x);
#else
    return __builtin_sqrt(x);
#endif
}
MBX_HD double int_sqrt(double x) {
    const uint64_t u = dbits(x), kOne = 1ull << 52;
    if (!(d_normal(u) && (int64_t)u > 0)) return sqrt_rare(x);
    const int e = (int)(u >> 52) - 1023, odd = e & 1;
    const uint64_t V = ((u & (kOne - 1)) | kOne) << odd; // v = V 2^-52 in [1, 4)
    const uint32_t v32 = (uint32_t)(V >> 22);
    // y = 2^31 / sqrt(v) to 28 bits
#ifdef __CUDA_ARCH__
    uint32_t y = (uint32_t)(0x1p46f * rsqrtf((float)v32));
#else
    uint32_t y = (uint32_t)(0x1p46f / __builtin_sqrtf((float)v32));
#endif
    const uint32_t t = (uint32_t)(((uint64_t)y * y) >> 32);
    const int64_t d = (int64_t)((1ull << 60) - (uint64_t)v32 * t); // |d| < 2^40
    y += (uint32_t)(int32_t)(((int64_t)(int32_t)(d >> 29) * (int64_t)y) >> 32);
    // sqrt(v) in units of 2^-29 within 5, and the next 23 bits
    const uint32_t s0 = (uint32_t)(((uint64_t)v32 * y) >> 32);
    const int64_t r1 = (int64_t)((V << 6) - (uint64_t)s0 * s0);
    const int32_t c1 = (int32_t)(((int64_t)(int32_t)(r1 >> 3) * (int64_t)y) >> 35);
    uint64_t q = ((uint64_t)s0 << 23) + (uint64_t)(int64_t)c1; // sqrt(v) 2^52 - q in (-0.6, 1.4)
    const int64_t r2 = (int64_t)((V << 52) - q * q);
    // (q + 1/2)^2 = q^2 + q + 1/4: no tie
    q += r2 > (int64_t)q ? 1 : 0;
    q -= r2 <= -(int64_t)q ? 1 : 0;
    return bitsd(((uint64_t)((e - odd) / 2 + 1023) << 52) + (q - kOne));
}
template <bool INT = false, class E>
MBX_HD FEt<E> fe_div(FEt<E> a, FEt<E> b) {
    if (d_is_zero(a.m)) return fe_make_as<E>(0.0, 0);
    return fe_renorm_as<E>(INT ? int_div(a.m, b.m) : a.m / b.m, a.e - b.e);
}
template <class E>
MBX_HD bool fe_abs_less(FEt<E> a, FEt<E> b) {
    if (d_is_zero(a.m)) return !d_is_zero(b.m);
    if (d_is_zero(b.m)) return false;
    if (a.e != b.e) return a.e < b.e;
    return d_abs_less(a.m, b.m);
}
MBX_HD double xsqrt(double x) {
#ifdef __CUDA_ARCH__
    return __dsqrt_rn(x);
#else
    return __builtin_sqrt(x);
#endif
}
template <bool INT = false, class E>
MBX_HD FEt<E> fe_sqrt(FEt<E> a) {
    if (d_le_zero(a.m)) return fe_make_as<E>(0.0, 0);
    E e = a.e;
    double m = a.m;
    if (e & 1) {
        m = d_twice(m);
        --e;
    }
    return fe_renorm_as<E>(INT ? int_sqrt(m) : xsqrt(m), e / 2);
}

// Complex arithmetic as GCC evaluates std::complex<double> for finite operands
// (inline multiply; division through libgcc's scaled Smith algorithm, restated).
struct C2 {
    double re, im;
};
MBX_HD C2 c2(double r, double i) {
    C2 z;
    z.re = r;
    z.im = i;
    return z;
}
MBX_HD C2 c_add(C2 a, C2 b) { return c2(a.re + b.re, a.im + b.im); }
MBX_HD C2 c_mul(C2 x, C2 y) { return c2(x.re * y.re - x.im * y.im, x.re * y.im + x.im * y.re); }
MBX_HD C2 c_div(C2 num, C2 den) {
    double a = num.re, b = num.im, c = den.re, d = den.im;
    const double RBIG = 8.98846567431157953865e307; // DBL_MAX / 2
    const double RMIN = 2.2250738585072013831e-308;  // DBL_MIN
    const double RMIN2 = 2.2204460492503130808e-16;  // DBL_EPSILON
    const double RMINSCAL = 4503599627370496.0;      // 1 / DBL_EPSILON
    const double RMAX2 = RBIG * RMIN2;
    double ratio, denom, x, y;
    if (dabs(c) < dabs(d)) {
        if (dabs(d) >= RBIG) { a = a / 2; b = b / 2; c = c / 2; d = d / 2; }
        if (dabs(d) < RMIN2) {
            a = a * RMINSCAL; b = b * RMINSCAL; c = c * RMINSCAL; d = d * RMINSCAL;
        } else if ((dabs(a) < RMIN && dabs(b) < RMAX2 && dabs(d) < RMAX2) || (dabs(b) < RMIN && dabs(a) < RMAX2 && dabs(d) < RMAX2)) {
            a = a * RMINSCAL; b = b * RMINSCAL; c = c * RMINSCAL; d = d * RMINSCAL;
        }
        ratio = c / d;
        denom = (c * ratio) + d;
        if (dabs(ratio) > RMIN) {
            x = ((a * ratio) + b) / denom;
            y = ((b * ratio) - a) / denom;
        } else {
            x = ((c * (a / d)) + b) / denom;
            y = ((c * (b / d)) - a) / denom;
        }
    } else {
        if (dabs(c) >= RBIG) { a = a / 2; b = b / 2; c = c / 2; d = d / 2; }
        if (dabs(c) < RMIN2) {
            a = a * RMINSCAL; b = b * RMINSCAL; c = c * RMINSCAL; d = d * RMINSCAL;
        } else if ((dabs(a) < RMIN && dabs(b) < RMAX2 && dabs(c) < RMAX2) || (dabs(b) < RMIN && dabs(a) < RMAX2 && dabs(c) < RMAX2)) {
            a = a * RMINSCAL; b = b * RMINSCAL; c = c * RMINSCAL; d = d * RMINSCAL;
        }
        ratio = d / c;
        denom = (d * ratio) + c;
        if (dabs(ratio) > RMIN) {
            x = ((b * ratio) + a) / denom;
            y = (b - (a * ratio)) / denom;
        } else {
            x = (a + (d * (b / c))) / denom;
            y = (b - (d * (a / c))) / denom;
        }
    }
    return c2(x, y);
}

// c_div by one denominator many times (the series-approximation seeds: up to 30
// divisions a sample). The ratio and the scaled denominator of Smith's algorithm
// are formed once, and each quotient by the denominator comes from its correctly
// rounded reciprocal y: q = a y, then twice q += (a - q denom) y with fused
// operations; after the first q is faithful, and then the second rounds
// correctly (Markstein's theorem, "Computation of elementary functions on the
// IBM RISC System/6000 processor", 1990): the bits of c_div's division in 5 FP64
// instructions for about 9. Numerators or quotients near the ends of the range,
// or a denominator whose mantissa is all ones, take c_div.
struct CDivBy {
    C2 den;
    double ratio, denom, y;
    bool swap, scale, ok;
};
MBX_HD double d_fma(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return __builtin_fma(a, b, c);
#endif
}
// the exponent within [2^-400, 2^400]: no quotient or residual of two leaves the range
MBX_HD bool d_mid(double x) { return (unsigned)((dbits(x) >> 52) & 0x7ff) - 623u <= 800u; }
MBX_HD CDivBy c_div_by(C2 den) {
    CDivBy q;
    q.den = den;
    q.swap = d_abs_less(den.re, den.im);
    double c = den.re, d = den.im;
    const double big = q.swap ? d : c;
    q.scale = d_abs_less(big, 2.2204460492503130808e-16);
    if (q.scale) {
        c = c * 4503599627370496.0;
        d = d * 4503599627370496.0;
    }
    q.ratio = q.swap ? c / d : d / c;
    q.denom = q.swap ? (c * q.ratio) + d : (d * q.ratio) + c;
    q.y = 1.0 / q.denom;
    q.ok = d_mid(big) && d_mid(q.denom) && d_abs_less(2.2250738585072013831e-308, q.ratio) && (dbits(q.denom) & 0xfffffffffffffull) != 0xfffffffffffffull;
    return q;
}
MBX_HD double d_quotient(double a, double b, double y) {
    double q = a * y;
    q = d_fma(d_fma(-q, b, a), y, q);
    return d_fma(d_fma(-q, b, a), y, q);
}
MBX_COLD C2 c_div_rare(C2 num, C2 den) { return c_div(num, den); }
MBX_HD C2 c_div(C2 num, const CDivBy& by) {
    double a = num.re, b = num.im;
    if (by.ok && d_mid(a) && d_mid(b)) {
        if (by.scale) {
            a = a * 4503599627370496.0;
            b = b * 4503599627370496.0;
        }
        // the numerators of c_div's two quotients
        const double xn = by.swap ? (a * by.ratio) + b : (b * by.ratio) + a;
        const double yn = by.swap ? (b * by.ratio) - a : b - (a * by.ratio);
        if (d_mid(xn) && d_mid(yn)) return c2(d_quotient(xn, by.denom, by.y), d_quotient(yn, by.denom, by.y));
    }
    return c_div_rare(num, by.den);
}

} // namespace mbx
