"""The integer quotient and square root (csrc/floatexp.h int_div, int_sqrt) against
the host's correctly rounded FP64 operations, bit for bit: random mantissas, few
or nearly all bits set, quotients and roots next to a rounding boundary, all
exponents, and the operands that they leave to the plain operation."""
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
    std::mt19937_64 g(11);
    long bad = 0, n = 0;
    auto same = [](double p, double q) { return dbits(p) == dbits(q) || (p != p && q != q); };
    auto check_div = [&](double a, double b) {
        ++n;
        if (!same(int_div(a, b), a / b) && ++bad < 8) printf("%a / %a: %a %a\n", a, b, int_div(a, b), a / b);
    };
    auto check_sqrt = [&](double x) {
        ++n;
        if (!same(int_sqrt(x), std::sqrt(x)) && ++bad < 8) printf("sqrt %a: %a %a\n", x, int_sqrt(x), std::sqrt(x));
    };
    auto num = [&]() {
        const uint64_t r = g();
        uint64_t f = g() & 0xfffffffffffffull;
        if (r % 5 == 0) f = g() & 0xf;
        if (r % 5 == 1) f = 0xfffffffffffffull ^ (g() & 0xf);
        if (r % 5 == 2) f = (g() & 0xff) << 44;
        if (r % 13 == 0) f = 1ull << (g() % 52);
        const uint64_t e = r & 64 ? 1023 + (r >> 8) % 3 - 1 : (r >> 8) % 2048;
        return bitsd(((r >> 63) << 63) | (e << 52) | f);
    };
    for (long k = 0; k < 6000000; ++k) {
        const double a = num(), b = num();
        check_div(a, b);
        check_sqrt(dabs(a));
        check_sqrt(a);
        // products, one ulp either side: quotients and roots beside a representable one
        for (int d = -1; d <= 1; ++d) {
            check_div(bitsd(dbits(a * b) + (uint64_t)(int64_t)d), b);
            check_sqrt(bitsd((dbits(a * a) + (uint64_t)(int64_t)d) & 0x7fffffffffffffffull));
        }
        // beside a halfway point: (a + half an ulp)^2 and (a + half an ulp) b
        const double h = std::fma(a, a, a * std::ldexp(1.0, -52));
        check_sqrt(dabs(h));
    }
    printf("%ld bad of %ld\n", bad, n);
    return bad != 0;
}
"""


def test_integer_quotient_and_root_round_correctly():
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        open(src, "w").write(PROGRAM)
        subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I" + os.path.join(PKG, "csrc"), src, "-o", exe])
        out = subprocess.run([exe], capture_output=True, text=True)
        print(out.stdout)
        assert out.returncode == 0, out.stdout + out.stderr
