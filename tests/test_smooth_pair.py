"""The escape values' logarithms in pairs of floats (csrc/smooth.cuh) against the
double expressions (mp.cpp:371-398), on the host: the same float wherever they
are accepted, accepted nearly everywhere, refused outside their range."""
import os
import subprocess
import tempfile

from conftest import PKG

PROGRAM = r"""
#include "smooth.cuh"
#include <cstdio>
#include <random>
using namespace mbx;
int main() {
    std::mt19937_64 g(21);
    std::uniform_real_distribution<double> u(0, 1);
    const double ln2 = 0x1.62e42fefa39efp-1;
    long bad = 0, no_s = 0, no_d = 0, n = 3000000;
    for (long i = 0; i < n; ++i) {
        const double zrad = i % 3 ? std::exp2(1.0 + 239.0 * u(g)) : std::exp2(std::exp2(1.0 + 6.0 * u(g)));
        const int k = 1 + (int)std::exp2(24.0 * u(g)) % (1 << 24);
        float out;
        if (!smooth_pair(k, zrad, out)) ++no_s;
        else if (out != (float)((double)k - std::log(std::log(zrad) / 2 / ln2) / ln2)) ++bad;
        const double s = std::exp2(60.0 * (u(g) - 0.3)), a = (2 * u(g) - 1) * s, b = (2 * u(g) - 1) * s * (i % 5 ? 1.0 : 1e-9);
        if (!distance_pair(zrad, a, b, out)) ++no_d;
        else if (out != (float)(std::sqrt(zrad) * std::log(zrad) / std::sqrt(a * a + b * b))) ++bad;
    }
    float out;
    const double odd[] = {0.0, -4.0, 1.0, 1.999, 1e80, 1e300, INFINITY, NAN};
    for (double x : odd) bad += smooth_pair(7, x, out) + distance_pair(x, 1.0, 2.0, out);
    const double far[] = {0.0, 1e-200, 1e200, INFINITY, NAN};
    for (double x : far) bad += distance_pair(1e10, x, 0.0, out);
    bad += smooth_pair(1 << 25, 1e10, out);
    printf("%ld bad, refused %ld and %ld of %ld\n", bad, no_s, no_d, n);
    return bad != 0 || no_s * 200 > n || no_d * 2000 > n;
}
"""


def test_smooth_count_and_distance_in_pairs_of_floats():
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        open(src, "w").write(PROGRAM)
        subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I" + os.path.join(PKG, "csrc"), src, "-o", exe])
        out = subprocess.run([exe], capture_output=True, text=True)
        print(out.stdout)
        assert out.returncode == 0, out.stdout + out.stderr
