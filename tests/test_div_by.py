"""Division by one complex denominator many times (csrc/floatexp.h CDivBy) against
the plain division (libgcc's scaled Smith algorithm, c_div), bit for bit, on the
host: random and special mantissas, all magnitudes, numerators of both parts."""
import os
import subprocess
import tempfile

from conftest import PKG

PROGRAM = r"""
#include "floatexp.h"
#include <cmath>
#include <cstdio>
#include <random>
using namespace mbx;
int main() {
    std::mt19937_64 g(4);
    std::uniform_real_distribution<double> u(-1, 1);
    long bad = 0, fast = 0, n = 0;
    auto num = [&](int span) {
        const uint64_t r = g();
        double m = u(g);
        if (r % 5 == 0) m = bitsd((dbits(m) & 0xfff0000000000000ull) | (g() & 0xf)); // few bits at the bottom
        if (r % 7 == 0) m = bitsd((dbits(m) | 0x000fffffffffffffull) ^ (g() & 0xf)); // nearly all ones
        if (r % 11 == 0) m = std::ldexp((double)(1 + (int)(g() % 64)), -6) * (r & 64 ? 1 : -1);
        if (r % 997 == 0) m = 0;
        return std::ldexp(m, span ? (int)(g() % (2 * span)) - span : 0);
    };
    for (int k = 0; k < 4000; ++k) {
        const int span = k % 4 == 0 ? 0 : k % 4 == 1 ? 60 : k % 4 == 2 ? 400 : 1070;
        const C2 den = c2(num(span), num(span));
        const CDivBy by = c_div_by(den);
        for (int i = 0; i < 1000; ++i, ++n) {
            const C2 a = c2(num(span), num(span)), p = c_div(a, den), q = c_div(a, by);
            const bool same = (dbits(p.re) == dbits(q.re) || (p.re != p.re && q.re != q.re)) && (dbits(p.im) == dbits(q.im) || (p.im != p.im && q.im != q.im));
            if (!same && ++bad < 8) printf("(%a,%a)/(%a,%a): %a %a, %a %a\n", a.re, a.im, den.re, den.im, p.re, p.im, q.re, q.im);
            fast += by.ok && d_mid(a.re) && d_mid(a.im);
        }
    }
    printf("%ld bad of %ld, %ld on the short path\n", bad, n, fast);
    return bad != 0 || fast * 2 < n;
}
"""


def test_division_by_one_denominator_is_the_plain_division():
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        open(src, "w").write(PROGRAM)
        subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I" + os.path.join(PKG, "csrc"), src, "-o", exe])
        out = subprocess.run([exe], capture_output=True, text=True)
        print(out.stdout)
        assert out.returncode == 0, out.stdout + out.stderr
