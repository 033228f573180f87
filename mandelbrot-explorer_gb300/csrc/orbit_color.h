// Orbit colourings of the delta loops (host and device): the stripe average
// (ColoringMethod::STRIPE_AVERAGE, "SAC") and the orbit traps
// (ColoringMethod::ORBIT_TRAP), as src/engine/orbit_coloring.h:21-132 defines
// them and the loops use them (mp.cpp:338-398 shallow, 2359-2378, 2422-2427,
// 2471-2472, 2497-2500 double path, 3338-3346, 3389-3397, 3503-3504, 3524-3529
// floatexp path, 764-882 arbitrary-precision point).
//
// Stripe average: every iteration's z adds the term t = 1/2 + sin(7 arg z) / 2;
// the value is the average of the last W terms under a triangular weight (the
// newest weighs W, the oldest 1), interpolated at escape between the average
// with and without the last term by the smooth-iteration fraction. A BLA skip
// breaks the run of terms, so it restarts the window. W = 256, the
// reference's default window.
// Orbit traps: the orbit's closest approach to the point 0 (|z|), the cross
// (min(|Re z|, |Im z|), weighted 1.5) and the circle |z| = 1/2; the value is
// 0.17 (-log10 distance) + 0.025 mu, mu the smooth escape count (0 interior).
// Operation order follows the reference's, in double; the device forms a
// stripe term by stripe_sin7, and log and log10 are the platform's.
#pragma once
#include <math.h>
#include <string.h>

#ifndef MBX_OC_HD
#ifdef __CUDACC__
#define MBX_OC_HD __host__ __device__ __forceinline__
#else
#define MBX_OC_HD inline
#endif
#endif

namespace mbx {

// coloring bits of the orbit colourings (mbx_request.coloring_method)
constexpr int kOcStripe = 1, kOcTrap = 2;
constexpr int kStripeWindow = 256;

MBX_OC_HD unsigned long long oc_bits(double x) {
#ifdef __CUDA_ARCH__
    return (unsigned long long)__double_as_longlong(x);
#else
    unsigned long long b;
    memcpy(&b, &x, 8);
    return b;
#endif
}
MBX_OC_HD double oc_double(unsigned long long b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    memcpy(&x, &b, 8);
    return x;
#endif
}

// sin(7 arg z) as Im(z^7) / |z|^7: z scaled to [1, 2) by its larger part's binade,
// four complex products and a reciprocal square root, about 40 FP64 operations
// where atan2 and sin take over 150. Its error is below theirs (on the device at
// most 1.2e-15 against 4.5e-15 over 2.1e6 points in quadruple precision, 1.8e-16
// against 4.7e-16 in the mean: theirs begins with the rounding of 7 arg z). For a larger part in
// [2^-900, 2^900]; the plain form otherwise.
MBX_OC_HD double stripe_sin7(double zr, double zi) {
    const double ar = fabs(zr), ai = fabs(zi), m = ar > ai ? ar : ai;
    if (!(m >= 0x1p-900 && m <= 0x1p900)) return sin(7.0 * atan2(zi, zr));
    const unsigned long long me = oc_bits(m) >> 52;
    const double s = oc_double((2046ull - me) << 52); // 2^(1023 - me)
    const double a = zr * s, b = zi * s;
    const double aa = a * a, bb = b * b, r2 = aa + bb;
    const double p2r = aa - bb, p2i = 2.0 * a * b;
    const double p4r = p2r * p2r - p2i * p2i, p4i = 2.0 * p2r * p2i;
    const double p6r = p4r * p2r - p4i * p2i, p6i = p4r * p2i + p4i * p2r;
    const double p7i = p6r * b + p6i * a;
    const double r4 = r2 * r2, r6 = r4 * r2, r14 = r6 * r6 * r2;
#ifdef __CUDA_ARCH__
    return p7i * rsqrt(r14);
#else
    return p7i / sqrt(r14);
#endif
}

struct StripeAvg {
    double ring[kStripeWindow];
    double run;     // sum of the window's terms
    double tri;     // triangular-weighted sum (newest term weight W)
    double last;    // the latest term
    int pos, fill;

    MBX_OC_HD void init() {
        run = tri = last = 0.0;
        pos = fill = 0;
    }
    MBX_OC_HD void restart() { // a BLA skip: the window starts again
        run = tri = 0.0;
        pos = fill = 0;
    }
    MBX_OC_HD void push(double zr, double zi) {
#ifdef __CUDA_ARCH__
        const double t = 0.5 + 0.5 * stripe_sin7(zr, zi);
#else
        const double t = 0.5 + 0.5 * sin(7.0 * atan2(zi, zr));
#endif
        last = t;
        double out = 0.0;
        if (fill == kStripeWindow) out = ring[pos];
        else ++fill;
        // every older term loses one unit of weight, the new one enters at W
        tri += (double)kStripeWindow * t - run;
        run += t - out;
        ring[pos] = t;
        pos = pos + 1 == kStripeWindow ? 0 : pos + 1;
    }
    // value at escape: |z|^2 = zrad, escape radius R
    MBX_OC_HD float value(double zrad, double R) const {
        double frac = 1.0 - log(log(zrad) * 0.5 / log(R)) / log(2.0);
        const double weight = (double)fill * kStripeWindow - (double)fill * (fill - 1) / 2.0;
        const double with_last = weight > 0.0 ? tri / weight : 0.0;
        const double wl = (double)kStripeWindow;
        const double without_last = weight > wl ? (tri - wl * last) / (weight - wl) : with_last;
        frac -= floor(frac);
        return (float)(without_last + (with_last - without_last) * frac);
    }
};

// The stripe average of a run of at most W terms: the same sums while no term
// has left the window (every term still in it, `out` above always 0), without
// the ring.
struct StripeTail {
    double run, tri, last;
    int fill;

    MBX_OC_HD void init() {
        run = tri = last = 0.0;
        fill = 0;
    }
    MBX_OC_HD void push(double zr, double zi) {
        const double t = 0.5 + 0.5 * stripe_sin7(zr, zi);
        last = t;
        ++fill;
        tri += (double)kStripeWindow * t - run;
        run += t;
    }
    MBX_OC_HD float value(double zrad, double R) const {
        StripeAvg a;
        a.tri = tri;
        a.last = last;
        a.fill = fill;
        return a.value(zrad, R);
    }
};

struct OrbitTrap {
    double point2;  // min |z|^2
    double cross;   // min min(|Re z|, |Im z|)
    double circle;  // min ||z| - 1/2|

    MBX_OC_HD void init() { point2 = cross = circle = 1e300; }
    MBX_OC_HD void push(double zr, double zi) {
        const double m2 = zr * zr + zi * zi;
        if (m2 < point2) point2 = m2;
        const double c = fmin(fabs(zr), fabs(zi));
        if (c < cross) cross = c;
        const double r = fabs(sqrt(m2) - 0.5);
        if (r < circle) circle = r;
    }
    // mu: the smooth escape count (0 for interior samples)
    MBX_OC_HD float value(double mu) const {
        double d = fmin(fmin(sqrt(point2), cross * 1.5), circle);
        if (d > 1.0) d = 1.0;
        const double trap = -log10(fmax(d, 1e-14));
        if (mu < 0.0) mu = 0.0;
        return (float)(0.17 * trap + 0.025 * mu);
    }
};

// The accumulators of one sample; OC selects which exist (kOcStripe, kOcTrap).
template <int OC>
struct OrbitColor {
    StripeAvg sac;
    OrbitTrap trap;
    MBX_OC_HD void init() {
        if (OC & kOcStripe) sac.init();
        if (OC & kOcTrap) trap.init();
    }
    MBX_OC_HD void push(double zr, double zi) {
        if (OC & kOcStripe) sac.push(zr, zi);
        if (OC & kOcTrap) trap.push(zr, zi);
    }
    MBX_OC_HD void skipped() {
        if (OC & kOcStripe) sac.restart();
    }
    // escape value when no DE / normal-map / overlay colouring takes precedence
    MBX_OC_HD float escaped(double mu, double zrad, double R) const {
        if (OC & kOcTrap) return trap.value(mu);
        return sac.value(zrad, R);
    }
    MBX_OC_HD float interior() const { return (OC & kOcTrap) ? trap.value(0.0) : -2.0f; }
};
template <>
struct OrbitColor<kOcTrap> { // the traps alone: no stripe window to carry
    OrbitTrap trap;
    MBX_OC_HD void init() { trap.init(); }
    MBX_OC_HD void push(double zr, double zi) { trap.push(zr, zi); }
    MBX_OC_HD void skipped() {}
    MBX_OC_HD float escaped(double mu, double, double) const { return trap.value(mu); }
    MBX_OC_HD float interior() const { return trap.value(0.0); }
};
template <>
struct OrbitColor<0> { // no orbit colouring: nothing to carry
    MBX_OC_HD void init() {}
    MBX_OC_HD void push(double, double) {}
    MBX_OC_HD void skipped() {}
    MBX_OC_HD float escaped(double, double, double) const { return 0.0f; }
    MBX_OC_HD float interior() const { return -2.0f; }
};

} // namespace mbx
