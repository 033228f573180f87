"""dz/dc through a BLA skip in pairs of floats (csrc/mixed_lane.cuh lane_j_bla_df),
J' = A J + B, against extended precision. A product of pairs is within 2^-45 and a
sum within 2^-46 of its size, so the two products, their sum and B's are within
2^-43 (|A| |J| + |B|) together; the FP32 lane adds one rounding to float, half a
unit of the last place."""
import os
import subprocess
import tempfile

from conftest import PKG

PROGRAM = r"""
#include <cuda_runtime.h>
#include "mixed_lane.cuh"
#include <cmath>
#include <cstdio>
#include <random>
using namespace mbx;
static std::mt19937_64 g(4);
static std::uniform_real_distribution<double> u(-1, 1);
template <class T> T num();
template <> float num<float>() { return (float)u(g); }
template <> df32 num<df32>() {
    const double x = u(g);
    const float h = (float)x;
    return df32(h, (float)(x - (double)h));
}
static long double val(float x) { return x; }
static long double val(df32 x) { return (long double)x.hi + (long double)x.lo; }
template <class T>
static long run(bool single) {
    long bad = 0;
    for (int n = 0; n < 1000000; ++n) {
        const T ar = num<T>(), ai = num<T>(), br = num<T>(), bi = num<T>(), jr = num<T>(), ji = num<T>();
        const int ea = (int)(40 * u(g)), ej = (int)(40 * u(g)), eb = n % 4 ? ea + ej + (int)(30 * u(g)) : (int)(200 * u(g));
        const JBla<T> v = lane_j_bla_df<T>(ar, ai, ea, br, bi, eb, jr, ji, ej);
        const long double sa = ldexpl(1, ea + ej - v.e), sb = ldexpl(1, eb - v.e);
        const long double wr = (val(ar) * val(jr) - val(ai) * val(ji)) * sa + val(br) * sb, wi = (val(ar) * val(ji) + val(ai) * val(jr)) * sa + val(bi) * sb;
        const long double size = hypotl(val(ar), val(ai)) * hypotl(val(jr), val(ji)) * sa + hypotl(val(br), val(bi)) * sb;
        const long double tol = ldexpl(size, -43);
        auto half_ulp = [&](long double w) { return single && w != 0 ? ldexpl(1, (int)ilogbl(w) - 24) * (1 + 1e-6L) : 0.0L; };
        if (fabsl(val(v.r) - wr) > tol + half_ulp(wr) || fabsl(val(v.i) - wi) > tol + half_ulp(wi)) ++bad;
    }
    return bad;
}
int main() {
    const long f = run<float>(true), d = run<df32>(false);
    printf("%ld and %ld bad\n", f, d);
    return f || d;
}
"""


def test_derivative_through_a_skip():
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        open(src, "w").write(PROGRAM)
        subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wno-deprecated-declarations", "-I" + os.path.join(PKG, "csrc"), "-I/usr/local/cuda/include", src, "-o", exe])
        out = subprocess.run([exe], capture_output=True, text=True)
        print(out.stdout)
        assert out.returncode == 0, out.stdout + out.stderr
