"""The relief shade and shaded sums in pairs of floats (csrc/color_math.cuh)
against the reference's double expressions (render.cpp:47-69, 263-292), on the
host: equal wherever they are accepted, and accepted nearly everywhere."""
import os
import subprocess
import tempfile

from conftest import PKG

PROGRAM = r"""
#include "color_math.cuh"
#include <cstdio>
#include <random>
using namespace mbx::cm;
int main() {
    std::mt19937_64 g(9);
    std::uniform_real_distribution<double> u(-1, 1), u01(0, 1);
    long bad = 0, acc_no = 0, rel_no = 0, n = 3000000;
    for (long i = 0; i < n; ++i) {
        const float acc = i % 11 ? (float)(u01(g) * std::pow(2.0, (double)(i % 7))) : 0.0f;
        const float c = i % 13 ? (float)(u01(g) * std::pow(2.0, -(double)(g() % 30))) : 0.0f, sh = (float)(0.25 + 0.85 * u01(g));
        float out;
        if (!acc_shaded_ff(acc, c, sh, out)) ++acc_no;
        else if (out != (float)((double)acc + (double)c * (double)sh)) ++bad;
        const double az = 4 * u(g), el = 1.6 * u(g), strength = i % 5 ? std::pow(10.0, 2 * u(g)) : 1.0;
        const double lx = std::cos(el) * std::cos(az), ly = std::cos(el) * std::sin(az), lz = std::sin(el);
        const ReliefParams p{ff_from(strength), ff_from(lx), ff_from(ly), ff_from(lz)};
        const double size = std::pow(10.0, 6 * u(g));
        const float sx = i % 17 ? (float)(u(g) * size) : 0.0f, sy = i % 19 ? (float)(u(g) * size) : 0.0f;
        const double nx = (double)(-sx) * strength, ny = (double)(-sy) * strength;
        double d = (nx * lx + ny * ly + lz) * (1.0 / std::sqrt(nx * nx + ny * ny + 1.0));
        if (d < 0) d = 0;
        if (!relief_ff(sx, sy, p, out)) ++rel_no;
        else if (out != (float)(0.25 + 0.85 * d)) ++bad;
    }
    // outside their range both leave the value to the double path
    float out;
    const ReliefParams p{ff_from(1.0), ff_from(0.6), ff_from(0.0), ff_from(0.8)};
    if (relief_ff(NAN, 0.0f, p, out) || relief_ff(INFINITY, 1.0f, p, out) || relief_ff(1e12f, 1.0f, p, out)) ++bad;
    if (acc_shaded_ff(NAN, 0.5f, 0.5f, out) || acc_shaded_ff(0.5f, NAN, 0.5f, out) || acc_shaded_ff(0.0f, NAN, 0.5f, out)) ++bad;
    printf("%ld %ld %ld of %ld\n", bad, acc_no, rel_no, n);
    return bad != 0 || acc_no * 1000 > n || rel_no * 1000 > n;
}
"""


def test_shading_in_pairs_of_floats():
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        open(src, "w").write(PROGRAM)
        subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I" + os.path.join(PKG, "csrc"), src, "-o", exe])
        out = subprocess.run([exe], capture_output=True, text=True)
        assert out.returncode == 0, out.stdout + out.stderr
