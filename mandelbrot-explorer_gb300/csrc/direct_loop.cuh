// The direct iterations z -> z^2 + c of the shallow and Julia frames, in the
// reference's FP64 operations but with the fewest FP64 instructions: on GB300
// an SM quarter takes one FP64 warp instruction per 64 cycles (compares and
// float conversions included), and about thirty integer ones beside it for
// free. So a step keeps only the operations whose rounded results the next z
// needs — two squares, a product, three sums — and everything else is decided
// on the bit patterns or in FP32:
//   * doublings are exponent increments;
//   * the escape test forms |z|^2 only when a component's high word reaches
//     the bound below which |z|^2 cannot exceed the bailout^2;
//   * the interior test |D|^2 < 1e-9 (D = 2 prod 2z, mp.cpp:344-399) follows
//     |D|^2 in pairs of floats with an exponent, under a bound on its distance
//     from the FP64 recurrence's value; where the bound leaves the test open, the sample
//     is iterated again by the plain loop (kDirectOpen);
//   * counters are integers.
// Six FP64 instructions a step instead of 34 in the shallow loop (14 in the
// Julia loop). Measured with k_direct's packing (kernels_exact.cu): the whole
// set at 1280x720, maxiter 5,000, 24.5 -> 2.3 ms a frame, of which the longest
// sample's 5,000 steps alone take most; a 2560x1440 overlay image (dz/dc: 13
// instructions a step) 107 -> 36.8 ms, bound by the FP64 unit; a 160x120 Julia
// thumbnail, maxiter 2,000, 1.01 -> 0.11 ms (its interior samples end at the
// first repeated z).
// Host and device; compiled without FMA contraction.
#pragma once
#include "dfloat.cuh"
#include "floatexp.h"
#include "orbit_color.h"

namespace mbx {

MBX_HD unsigned hi_abs(double x) { return (unsigned)(dbits(x) >> 32) & 0x7fffffffu; }
MBX_HD unsigned umax_(unsigned a, unsigned b) { return a > b ? a : b; }
MBX_HD unsigned float_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    unsigned u;
    memcpy(&u, &x, 4);
    return u;
#endif
}
MBX_HD float bits_float(unsigned u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float x;
    memcpy(&x, &u, 4);
    return x;
#endif
}

// High word below which neither component lets |z|^2 exceed esc2: both below
// sqrt(esc2 / 2), by more than the sum's rounding. 0 (test every step) for a
// bailout that is not an ordinary number.
inline unsigned direct_escape_word(double esc2) {
    if (!(esc2 > 1e-30 && esc2 < 1e300)) return 0u;
    const double c = __builtin_sqrt(esc2 * 0.5) * (1.0 - 1.0 / (1 << 18));
    return (unsigned)(dbits(c) >> 32);
}
// Every |z| of an orbit inside the bailout, and its squares, must be in FP32's
// range for the interior test in pairs of floats.
MBX_HD bool direct_trackable(double esc2) { return esc2 <= 1.1e36; }
constexpr unsigned kDirectFarWord = 0x43b00000u;  // 2^60
constexpr unsigned kDirectTinyWord = 0x3e500000u; // 2^-26

// A positive double below 2^120 as hi + lo in floats, 47 bits (truncated); below
// 2^-100 something near 2^-100.
MBX_HD void split2f(double x, float& hi, float& lo) {
    const uint64_t b = dbits(x);
    unsigned h = (unsigned)(b >> 32);
    h = h > 0x39b00000u ? h : 0x39b00000u;
    const unsigned f = ((h << 3) | ((unsigned)b >> 29)) + 0x40000000u; // exponent bias 1023 -> 127
    hi = bits_float(f);
    // the next 23 bits under an implicit one 2^23 below, less that one
    const unsigned base = (h >> 20 << 23) + 0x40000000u - (23u << 23);
    lo = bits_float(base | (((unsigned)b >> 6) & 0x7fffffu)) - bits_float(base);
}

// |D|^2 as (gh + gl) 2^e, gh in [1, 2]. Each update multiplies by 4 |z|^2 in
// pairs of floats; relative error below 2^-42 a step (the split's 2^-46, the
// sum's and the product's roundings of 2^-46 to 2^-44). The FP64 recurrence
// itself stays within sqrt(5) 2^-53 a step of the product of its factors,
// normwise, which the same bound takes in.
struct InteriorTrack {
    float gh = 1.0f, gl = 0.0f;
    int e = 2, emax = 2; // |D_0|^2 = 4
    MBX_HD void step(double x2, double y2) { // the squares of z's parts
        float xh, xl, yh, yl;
        split2f(x2, xh, xl);
        split2f(y2, yh, yl);
        const float s = xh + yh, t = s - xh; // exact sum s + r
        const float r = ((xh - (s - t)) + (yh - t)) + (xl + yl);
        const float qh = s + r, ql = r - (qh - s);
        const float p = gh * qh;
        float d = df_fma(gh, qh, -p);
        d = df_fma(gh, ql, df_fma(gl, qh, d));
        const float v = p + d, w = d - (v - p);
        const unsigned b = float_bits(v);
        const int k = (int)(b >> 23) - 127;
        e += k + 2;
        gh = bits_float((b & 0x007fffffu) | 0x3f800000u);
        gl = w * bits_float((unsigned)(127 - k) << 23);
        emax = e > emax ? e : emax;
    }
    // Called with e <= -30 after n steps: 1 |D|^2 < 1e-9, 0 not, 2 open.
    // emax: an FP64 component overflows at 2^1024, after which D is never
    // finite again; it cannot have while |D|^2 stayed below 2^1990.
    MBX_HD int below(int n) const {
        if (emax > 2060) return 0;
        // |D|^2 2^30 - 1e-9 2^30 (1.073741824), against the error bound
        const float m = (float)n * 2.5e-13f + 1e-12f;
        const float d = e < -30 ? -0.07f : (gh - 0x1.12e0bep+0f) + (gl - 0x1.04dad2p-25f);
        if (d > 1.1f * m) return 0;
        if (emax >= 1990) return 2;
        return d < -1.1f * m ? 1 : 2;
    }
};

// How a step leaves a sample.
enum DirectEnd { kDirectRuns = 0, kDirectEscaped = 1, kDirectInterior = 2, kDirectOpen = 3 };

// One sample of z -> z^2 + c from z = c. LANE: the reference's lane kernel
// (mp.cpp:416-532) takes a step before it looks at maxiter and doubles the
// product zr zi; its scalar loop (mp.cpp:330-399) looks first and doubles zr.
// DERIV: dz/dc as well. visit(zr, zi, zr^2, zi^2) sees every z.
template <bool LANE, bool DERIV>
struct DirectLane {
    double zr, zi, x2, y2, cr, ci;
    double dcr, dci;
    InteriorTrack track;
    int n; // iterations taken plus one; at the escape, the escape iteration
    unsigned hm;

    MBX_HD int start(double c_re, double c_im, int mxit, double esc2) {
        zr = cr = c_re;
        zi = ci = c_im;
        dcr = 1.0;
        dci = 0.0;
        n = 1;
        track = InteriorTrack();
        if (!LANE && mxit <= 1) return kDirectInterior;
        hm = umax_(hi_abs(zr), hi_abs(zi));
        if (hm >= kDirectFarWord || hm < kDirectTinyWord || !direct_trackable(esc2)) return kDirectOpen;
        x2 = zr * zr;
        y2 = zi * zi;
        return kDirectRuns;
    }
    // One step, without its tests: true when one of them may apply (one branch a
    // step: the tests' own would hold up a lone sample's chain). hm: the larger
    // part's high word.
    template <class Visit>
    MBX_HD bool advance(int mxit, unsigned esc_word, Visit&& visit) {
        const double s = x2 - y2, m = LANE ? d_twice(zr * zi) : d_twice(zr) * zi;
        track.step(x2, y2);
        if (DERIV) {
            const double t = d_twice(dcr * zr - dci * zi) + 1.0;
            dci = d_twice(dcr * zi + dci * zr);
            dcr = t;
        }
        zr = s + cr;
        zi = m + ci;
        x2 = zr * zr;
        y2 = zi * zi;
        visit(zr, zi, x2, y2);
        hm = umax_(hi_abs(zr), hi_abs(zi));
        ++n;
        return hm >= esc_word || hm < kDirectTinyWord || track.e <= -30 || n >= mxit;
    }
    // The tests of that step, in the reference's order.
    MBX_HD int resolve(int mxit, double esc2, unsigned esc_word) const {
        if (hm >= esc_word && d_abs_less(esc2, x2 + y2)) return kDirectEscaped; // |z|^2 > esc2
        if (track.e <= -30) {
            const int b = track.below(n - 1);
            if (b) return b == 1 ? kDirectInterior : kDirectOpen;
        }
        if (n >= mxit) return kDirectInterior;
        return hm < kDirectTinyWord ? kDirectOpen : kDirectRuns; // (|z|^2 near split2f's floor)
    }
    template <class Visit>
    MBX_HD int step(int mxit, double esc2, unsigned esc_word, Visit&& visit) {
        return advance(mxit, esc_word, visit) ? resolve(mxit, esc2, esc_word) : kDirectRuns;
    }
};

// One Julia sample of z -> z^2 + c (solveJuliaShallowSimdList, mp.cpp:534-636;
// D' = 2 z D from D_0 = 1 under DERIV). A z that repeats an earlier one bit for
// bit cycles for ever: the orbit never escapes (Brent's doubling window).
template <bool DERIV>
struct JuliaLane {
    double zr, zi, x2, y2;
    double dcr, dci; // D
    uint64_t sr, si;
    int n, next, win; // n: iterations taken

    MBX_HD int start(double z_re, double z_im, double esc2) {
        zr = z_re;
        zi = z_im;
        x2 = zr * zr;
        y2 = zi * zi;
        dcr = 1.0;
        dci = 0.0;
        n = 0;
        sr = si = ~0ull; // (a NaN: no finite z equals it)
        next = win = 8;
        return d_abs_less(esc2, x2 + y2) ? kDirectEscaped : kDirectRuns;
    }
    // (as DirectLane::advance and resolve; the repeat is looked for on one low word)
    MBX_HD bool advance(double cr, double ci, int mxit, unsigned esc_word) {
        const double s = x2 - y2, m = zr * zi;
        if (DERIV) {
            const double t = d_twice(dcr * zr - dci * zi);
            dci = d_twice(dcr * zi + dci * zr);
            dcr = t;
        }
        zr = s + cr;
        zi = d_twice(m) + ci;
        x2 = zr * zr;
        y2 = zi * zi;
        ++n;
        return umax_(hi_abs(zr), hi_abs(zi)) >= esc_word || n >= mxit || n == next || (unsigned)dbits(zr) == (unsigned)sr;
    }
    MBX_HD int resolve(int mxit, double esc2) {
        if (d_abs_less(esc2, x2 + y2)) return kDirectEscaped;
        if (n >= mxit || (dbits(zr) == sr && dbits(zi) == si)) return kDirectInterior;
        if (n == next) {
            sr = dbits(zr);
            si = dbits(zi);
            next = n > (1 << 29) ? 0x7fffffff : n + win;
            win += win > (1 << 29) ? 0 : win;
        }
        return kDirectRuns;
    }
    MBX_HD int step(double cr, double ci, int mxit, double esc2, unsigned esc_word) {
        return advance(cr, ci, mxit, esc_word) ? resolve(mxit, esc2) : kDirectRuns;
    }
};

// OrbitTrap over the direct iteration's finite z: the same minima, with the
// comparisons on bit patterns and |z|^2, sqrt |z|^2 in FP64 only where a
// smaller value is possible (for the circle an FP32 screen with a margin well
// above its error).
struct DirectTrap {
    double point2, circle;
    uint64_t cross; // bits of a non-negative double
    float circle_hi; // above circle

    MBX_HD void init() {
        point2 = circle = 1e300;
        cross = dbits(1e300);
        circle_hi = 3e38f;
    }
    MBX_HD void push(double zr, double zi, double x2, double y2) {
        const uint64_t ar = dbits(zr) & 0x7fffffffffffffffull, ai = dbits(zi) & 0x7fffffffffffffffull;
        const uint64_t c = ar < ai ? ar : ai;
        if (c < cross) cross = c;
        // |z|^2 >= both squares, rounded too
        if (umax_(hi_abs(x2), hi_abs(y2)) <= hi_abs(point2)) {
            const double m2 = x2 + y2;
            if (d_abs_less(m2, point2)) point2 = m2;
        }
        const bool near = umax_(hi_abs(zr), hi_abs(zi)) < kDirectFarWord;
        if (near) {
            float xh, yh, t;
            split2f(x2, xh, t);
            split2f(y2, yh, t);
            const float r = sqrtf(xh + yh); // |z| to 3e-7 relative
            if (fabsf(r - 0.5f) - 1e-6f * (r + 1.0f) > circle_hi) return;
        }
        const double r = fabs(xsqrt(x2 + y2) - 0.5);
        if (d_abs_less(r, circle)) {
            circle = r;
            if (r < 1e30) circle_hi = (float)r * 1.000001f;
        }
    }
};

} // namespace mbx
