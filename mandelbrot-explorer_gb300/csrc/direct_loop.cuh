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
// Julia loop), still bound by them. Measured: the whole set at 1280x720,
// maxiter 5,000, 24.5 -> 5.7 ms a frame; a 160x120 Julia thumbnail, maxiter
// 2,000, 1.00 -> 0.11 ms (its interior samples end at the first repeated z).
// Host and device; compiled without FMA contraction.
#pragma once
#include "dfloat.cuh"
#include "floatexp.h"
#include "orbit_color.h"

namespace mbx {

MBX_HD unsigned hi_abs(double x) { return (unsigned)(dbits(x) >> 32) & 0x7fffffffu; }
MBX_HD unsigned umax_(unsigned a, unsigned b) { return a > b ? a : b; }
// x + x: an exponent increment for normal x with a normal result
MBX_HD double twice(double x) {
    const unsigned h = hi_abs(x);
    if (h - 0x00100000u < 0x7fd00000u) return bitsd(dbits(x) + (1ull << 52));
    return x + x;
}
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

enum DirectEnd { kDirectEscaped = 1, kDirectInterior = 2, kDirectOpen = 3 };

struct DirectState {
    double zr, zi, zrad;   // the escaped z and |z|^2
    double dcr, dci;       // dz/dc (DERIV)
    int n;                 // iterations taken
};

// Iterate z from c at most until n reaches mxit (n starts at 1). LANE: the
// reference's lane kernel (mp.cpp:416-532) takes a step before it looks at
// maxiter and doubles the product zr zi; its scalar loop (mp.cpp:330-399) looks
// first and doubles zr. DERIV: dz/dc as well. visit(zr, zi) sees every z.
template <bool LANE, bool DERIV, class Visit>
MBX_HD int direct_iterate(double cr, double ci, int mxit, double esc2, unsigned esc_word, DirectState& s, Visit&& visit) {
    double zr = cr, zi = ci, dcr = 1, dci = 0;
    s.n = 1;
    if (!LANE && mxit <= 1) return kDirectInterior;
    unsigned hm = umax_(hi_abs(zr), hi_abs(zi));
    if (hm >= kDirectFarWord || hm < kDirectTinyWord || !direct_trackable(esc2)) return kDirectOpen;
    InteriorTrack track;
    double x2 = zr * zr, y2 = zi * zi;
    for (int n = 1;;) {
        track.step(x2, y2);
        if (DERIV) {
            const double t = twice(dcr * zr - dci * zi) + 1.0;
            dci = twice(dcr * zi + dci * zr);
            dcr = t;
        }
        const double nzi = (LANE ? twice(zr * zi) : twice(zr) * zi) + ci;
        zr = (x2 - y2) + cr;
        zi = nzi;
        x2 = zr * zr;
        y2 = zi * zi;
        visit(zr, zi, x2, y2);
        hm = umax_(hi_abs(zr), hi_abs(zi));
        if (hm >= esc_word) {
            const double zrad = x2 + y2;
            if (d_abs_less(esc2, zrad)) { // zrad > esc2
                s.zr = zr;
                s.zi = zi;
                s.zrad = zrad;
                s.dcr = dcr;
                s.dci = dci;
                s.n = n + 1;
                return kDirectEscaped;
            }
        }
        if (track.e <= -30) {
            const int b = track.below(n);
            if (b) return b == 1 ? kDirectInterior : kDirectOpen;
        }
        if (++n >= mxit) return kDirectInterior;
        if (hm < kDirectTinyWord) return kDirectOpen; // |z|^2 near split2f's floor
    }
}

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
    template <int OC>
    MBX_HD void give(OrbitColor<OC>& oc) const {
        if constexpr ((OC & kOcTrap) != 0) {
            oc.trap.point2 = point2;
            oc.trap.cross = bitsd(cross);
            oc.trap.circle = circle;
        }
    }
};

// The Julia iteration z -> z^2 + c from z (solveJuliaShallowSimdList,
// mp.cpp:534-636; D' = 2 z D from D_0 = 1 under DERIV). A z that repeats an
// earlier one bit for bit cycles for ever: the orbit never escapes (Brent's
// doubling window). Returns 1 escaped, 2 not.
template <bool DERIV>
MBX_HD int julia_iterate(double zr, double zi, double cr, double ci, int mxit, double esc2, unsigned esc_word, DirectState& s) {
    double dr = 1.0, di = 0.0;
    double x2 = zr * zr, y2 = zi * zi;
    s.zr = zr;
    s.zi = zi;
    s.zrad = x2 + y2;
    s.dcr = 1.0;
    s.dci = 0.0;
    s.n = 0;
    if (d_abs_less(esc2, s.zrad)) return kDirectEscaped;
    uint64_t sr = ~0ull, si = ~0ull; // (a NaN: equals no finite z)
    int next = 8, win = 8;
    for (int n = 0;;) {
        if (DERIV) {
            const double t = twice(dr * zr - di * zi);
            di = twice(dr * zi + di * zr);
            dr = t;
        }
        const double nzi = twice(zr * zi) + ci;
        zr = (x2 - y2) + cr;
        zi = nzi;
        x2 = zr * zr;
        y2 = zi * zi;
        ++n;
        if (umax_(hi_abs(zr), hi_abs(zi)) >= esc_word) {
            const double zrad = x2 + y2;
            if (d_abs_less(esc2, zrad)) {
                s.zr = zr;
                s.zi = zi;
                s.zrad = zrad;
                s.dcr = dr;
                s.dci = di;
                s.n = n;
                return kDirectEscaped;
            }
        }
        if (n >= mxit || (dbits(zr) == sr && dbits(zi) == si)) return kDirectInterior;
        if (n == next) {
            sr = dbits(zr);
            si = dbits(zi);
            next = n > (1 << 29) ? 0x7fffffff : n + win;
            win += win > (1 << 29) ? 0 : win;
        }
    }
}

} // namespace mbx
