"""The direct iterations with few FP64 operations (csrc/direct_loop.cuh) against
the reference's loops written out (mp.cpp:330-399, 416-532, 534-636), on the
host: outcome, count, every bit of z, |z|^2 and the derivative, and the trap's
minima, over whole frames, axes, tiny and huge numbers and odd bailouts."""
import os
import subprocess
import tempfile

from conftest import PKG

PROGRAM = r"""
#include "direct_loop.cuh"
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
using namespace mbx;
struct DirectState { double zr, zi, zrad, dcr, dci; int n; };
template <bool LANE, bool DERIV, class Visit>
static int direct_iterate(double cr, double ci, int mxit, double esc2, unsigned w, DirectState& s, Visit&& visit) {
    DirectLane<LANE, DERIV> l;
    int st = l.start(cr, ci, mxit, esc2);
    while (st == kDirectRuns) st = l.step(mxit, esc2, w, visit);
    if (st == kDirectEscaped) s = DirectState{l.zr, l.zi, l.x2 + l.y2, l.dcr, l.dci, l.n};
    return st;
}
template <bool DERIV>
static int julia_iterate(double zr, double zi, double cr, double ci, int mxit, double esc2, unsigned w, DirectState& s) {
    JuliaLane<DERIV> l;
    int st = l.start(zr, zi, esc2);
    while (st == kDirectRuns) st = l.step(cr, ci, mxit, esc2, w);
    if (st == kDirectEscaped) s = DirectState{l.zr, l.zi, l.x2 + l.y2, l.dcr, l.dci, l.n};
    return st;
}
struct Ref { int st, n; double zr, zi, zrad, dcr, dci; OrbitTrap trap; };
static Ref plain(bool lane, double cr, double ci, int mxit, double esc2) {
    Ref r{};
    r.trap.init();
    double zr = cr, zi = ci, dr = 2, di = 0, dcr = 1, dci = 0;
    r.st = 2;
    if (!lane && mxit <= 1) return r;
    for (int n = 1;; ++n) {
        const double ndr = 2.0 * (dr * zr - di * zi), ndi = 2.0 * (dr * zi + di * zr);
        const double ndcr = 2.0 * (dcr * zr - dci * zi) + 1.0, ndci = 2.0 * (dcr * zi + dci * zr);
        const double nzr = zr * zr - zi * zi + cr;
        const double nzi = (lane ? 2.0 * (zr * zi) : 2.0 * zr * zi) + ci;
        zr = nzr; zi = nzi; dr = ndr; di = ndi; dcr = ndcr; dci = ndci;
        r.trap.push(zr, zi);
        const double zrad = zr * zr + zi * zi;
        if (zrad > esc2) { r.st = 1; r.n = n + 1; r.zr = zr; r.zi = zi; r.zrad = zrad; r.dcr = dcr; r.dci = dci; return r; }
        if (dr * dr + di * di < 1e-9) return r;
        if (n + 1 >= mxit) return r;
    }
}
static Ref plain_julia(double zr, double zi, double cr, double ci, int mxit, double esc2) {
    Ref r{};
    double dr = 1, di = 0, zrad = zr * zr + zi * zi;
    r.st = 1; r.n = 0; r.zr = zr; r.zi = zi; r.zrad = zrad; r.dcr = 1; r.dci = 0;
    if (zrad > esc2) return r;
    for (int n = 0;; ++n) {
        const double ndr = 2.0 * (dr * zr - di * zi), ndi = 2.0 * (dr * zi + di * zr);
        const double nzr = zr * zr - zi * zi + cr, nzi = 2.0 * (zr * zi) + ci;
        zr = nzr; zi = nzi; dr = ndr; di = ndi;
        zrad = zr * zr + zi * zi;
        if (zrad > esc2) { r.st = 1; r.n = n + 1; r.zr = zr; r.zi = zi; r.zrad = zrad; r.dcr = dr; r.dci = di; return r; }
        if (n + 1 >= mxit) { r.st = 2; return r; }
    }
}
static bool same(double a, double b) { return dbits(a) == dbits(b) || (a != a && b != b); }
int main() {
    std::mt19937_64 g(5);
    std::uniform_real_distribution<double> u(-1, 1);
    long bad = 0, open = 0, open_frame = 0, total = 0, frame = 0;
    auto esc_of = [](double r) { const float f = (float)r; return (double)(f * f); };
    const double radii[] = {1e8, 256.0, 2.0, 1e18, 0.5, 1e-3, 1e-25, 1e25};
    auto check = [&](double cr, double ci, int mxit, double esc2, bool in_frame) {
        const unsigned w = direct_escape_word(esc2);
        for (int lane = 0; lane < 2; ++lane) {
            const Ref r = plain(lane, cr, ci, mxit, esc2);
            DirectTrap t;
            t.init();
            auto visit = [&](double zr, double zi, double x2, double y2) { t.push(zr, zi, x2, y2); };
            DirectState s{};
            const int st = lane ? direct_iterate<true, true>(cr, ci, mxit, esc2, w, s, visit) : direct_iterate<false, true>(cr, ci, mxit, esc2, w, s, visit);
            ++total;
            frame += in_frame;
            if (st == kDirectOpen) { ++open; open_frame += in_frame; continue; }
            bool ok = st == r.st;
            if (ok && st == 1) ok = s.n == r.n && same(s.zr, r.zr) && same(s.zi, r.zi) && same(s.zrad, r.zrad) && same(s.dcr, r.dcr) && same(s.dci, r.dci);
            if (ok && (st == 1 || mxit > 1 || lane)) ok = same(t.point2, r.trap.point2) && same(bitsd(t.cross), r.trap.cross) && same(t.circle, r.trap.circle);
            DirectState s2{};
            auto none = [](double, double, double, double) {};
            const int st2 = lane ? direct_iterate<true, false>(cr, ci, mxit, esc2, w, s2, none) : direct_iterate<false, false>(cr, ci, mxit, esc2, w, s2, none);
            ok = ok && st2 == st && s2.n == s.n && same(s2.zrad, s.zrad);
            if (!ok && ++bad < 10) printf("c %.17g %.17g mxit %d esc2 %g lane %d: %d/%d n %d/%d\n", cr, ci, mxit, esc2, lane, st, r.st, s.n, r.n);
        }
    };
    auto check_j = [&](double zr, double zi, double cr, double ci, int mxit, double esc2) {
        const Ref r = plain_julia(zr, zi, cr, ci, mxit, esc2);
        DirectState s{};
        const int st = julia_iterate<true>(zr, zi, cr, ci, mxit, esc2, direct_escape_word(esc2), s);
        bool ok = st == r.st && (st != 1 || (s.n == r.n && same(s.zr, r.zr) && same(s.zi, r.zi) && same(s.zrad, r.zrad) && same(s.dcr, r.dcr) && same(s.dci, r.dci)));
        DirectState s2{};
        const int st2 = julia_iterate<false>(zr, zi, cr, ci, mxit, esc2, direct_escape_word(esc2), s2);
        ok = ok && st2 == st && (st != 1 || (s2.n == s.n && same(s2.zrad, s.zrad)));
        if (!ok && ++bad < 10) printf("julia z %.17g %.17g c %.17g %.17g mxit %d esc2 %g: %d/%d n %d/%d\n", zr, zi, cr, ci, mxit, esc2, st, r.st, s.n, r.n);
    };
    // the whole set, and windows on its edge
    for (int i = 0; i < 97; ++i)
        for (int j = 0; j < 131; ++j) {
            check(-2.1 + 2.8 * j / 130, -1.2 + 2.4 * i / 96, 1500, esc_of(1e8), true);
            check(-0.75 + 0.05 * j / 130, 0.1 + 0.04 * i / 96, 800, esc_of(256.0), true);
        }
    // random centres, depths, bailouts and limits
    for (int k = 0; k < 20000; ++k) {
        const double sc = std::ldexp(1.0, -(int)(g() % 40));
        check(-0.7436438870371587 + sc * u(g), 0.131825904205312 + sc * u(g), 1 + (int)(g() % 400), esc_of(radii[g() % 8]), false);
        check(-1.75 + sc * u(g), sc * u(g), 1 + (int)(g() % 400), esc_of(radii[g() % 8]), false);
    }
    // axes, zeros, tiny, huge and special values
    const double sp[] = {0.0, -0.0, 1e-300, -1e-310, 5e-324, 1e-160, 1e-20, -2.0, -1.0, 0.25, -0.75, 2.0, 1e9, 1e40, 1e155, -1e300, 1.7e308, INFINITY, NAN};
    for (double a : sp)
        for (double b : sp)
            for (double r : radii)
                for (int m : {1, 2, 3, 50, 700}) {
                    check(a, b, m, esc_of(r), false);
                    check(a, b, m, INFINITY, false);
                    check(a + 1e-9 * u(g), b, m, esc_of(r), false);
                    for (double c : {0.0, -2.0, -0.123, 1e-200, 0.3}) check_j(a, b, c, 0.0, m, esc_of(r)), check_j(a, b, c, 0.745, m, esc_of(r));
                }
    for (int i = 0; i < 90; ++i)
        for (int j = 0; j < 120; ++j) {
            check_j(-1.6 + 3.2 * j / 119, -1.2 + 2.4 * i / 89, -0.123, 0.745, 900, esc_of(256.0));
            check_j(-1.6 + 3.2 * j / 119, -1.2 + 2.4 * i / 89, 0.0, 1.0, 900, esc_of(1e8));
            check_j(-1.6 + 3.2 * j / 119, -1.2 + 2.4 * i / 89, -0.390540870218399, -0.586787907346969, 900, esc_of(2.0));
            check_j(-2.0 + 4.0 * j / 119, 1e-200 * i, -2.0, 0.0, 900, esc_of(1e8));
        }
    // the plain loop must take few of a frame's samples
    printf("%ld bad of %ld, open %ld, in frames %ld of %ld\n", bad, total, open, open_frame, frame);
    return bad != 0 || open_frame * 1000 > frame;
}
"""


def test_direct_loops_match_the_plain_ones():
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        open(src, "w").write(PROGRAM)
        subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I" + os.path.join(PKG, "csrc"), "-I/usr/local/cuda/include", src, "-o", exe])
        out = subprocess.run([exe], capture_output=True, text=True)
        assert out.returncode == 0, out.stdout + out.stderr


STRIPE_PROGRAM = r"""
#include "orbit_color.h"
#include <cmath>
#include <cstdio>
#include <random>
using namespace mbx;
int main() {
    std::mt19937_64 g(3);
    std::uniform_real_distribution<double> u(-1, 1);
    double worst = 0;
    for (long i = 0; i < 2000000; ++i) {
        const double sc = std::ldexp(1.0, (int)(g() % 2000) - 1000);
        const double a = u(g) * sc, b = u(g) * sc * (i % 7 ? 1.0 : std::ldexp(1.0, -(int)(g() % 80)));
        worst = std::fmax(worst, (double)fabsl(stripe_sin7(a, b) - sinl(7.0L * atan2l(b, a))));
    }
    const double exact[] = {stripe_sin7(0, 0), stripe_sin7(0, 3), stripe_sin7(0, -2), stripe_sin7(5, 0)};
    printf("%g\n", worst);
    return !(worst < 4e-15 && exact[0] == 0 && exact[1] == -1 && exact[2] == 1 && exact[3] == 0);
}
"""


def test_stripe_term_is_as_accurate_as_the_trigonometry():
    """sin(7 arg z) from powers of z against 64-bit long double trigonometry,
    over 600 decades: within 4e-15, what atan2 and sin in double are off by
    (7 arg z up to 22 is itself rounded by 1.8e-15)."""
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        open(src, "w").write(STRIPE_PROGRAM)
        subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I" + os.path.join(PKG, "csrc"), src, "-o", exe])
        out = subprocess.run([exe], capture_output=True, text=True)
        assert out.returncode == 0, out.stdout + out.stderr
