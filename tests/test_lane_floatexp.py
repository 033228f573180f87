"""The lanes' rare floatexp steps (csrc/mixed_lane.cuh lane_rebase_fe,
lane_j_step_fe) take int exponents where those cannot leave an int's range and
64-bit ones elsewhere: the same bits as with 64 bits throughout, for orbit entries
and scales on both sides of the line (2^28), zeros and a missing entry among them."""
import os
import subprocess
import tempfile

from conftest import PKG

PROGRAM = r"""
#include <cuda_runtime.h>
#include "mixed_lane.cuh"
#include <cstdio>
#include <random>
using namespace mbx;
int main() {
    std::mt19937_64 g(9);
    std::uniform_real_distribution<double> u(-1, 1);
    long bad = 0, mid = 0, far = 0;
    const int line = 1 << 28, bases[] = {0, -900, -70000, -line + 40, -line - 40, line - 40, -2 * line, -1800000000};
    auto num = [&](int64_t e) { return g() % 29 == 0 ? fe_make(0.0, 0) : fe_renorm(u(g), e); };
    for (int n = 0; n < 400000; ++n) {
        const int b = bases[g() % 8], near = (int)(80 * u(g));
        const TE<double> S{0.5 + 0.49 * std::fabs(u(g)), b + near};
        FE2 X{num(b + (int64_t)(60 * u(g))), num(g() % 3 ? b + (int64_t)(60 * u(g)) : (int64_t)(60 * u(g)))};
        const FE2* at = g() % 7 ? &X : nullptr;
        const FE zero = fe_make(0.0, 0), Xr = at ? X.re : zero, Xi = at ? X.im : zero;
        const double wr = u(g), wi = g() % 11 ? u(g) : 0.0;
        (te_mid(S.e) && te_mid(Xr.e) && te_mid(Xi.e) ? mid : far) += 1;
        const RebaseFe p = lane_rebase_fe(S, wr, wi, at, n & 1), q = lane_rebase_as(fe_make(S.m, S.e), wr, wi, Xr, Xi, n & 1);
        bad += p.take != q.take || dbits(p.S.m) != dbits(q.S.m) || p.S.e != q.S.e || dbits(p.wr) != dbits(q.wr) || dbits(p.wi) != dbits(q.wi);
        const int sje = n % 5 ? (int)(300 * u(g)) - b / 2 : b;
        const JVal j = lane_j_step_fe(at, S, wr, wi, sje, wi, wr), k = lane_j_step_as(Xr, Xi, fe_make(S.m, S.e), wr, wi, sje, wi, wr);
        bad += dbits(j.r) != dbits(k.r) || dbits(j.i) != dbits(k.i) || j.e != k.e;
    }
    printf("%ld bad, %ld by int, %ld by 64 bits\n", bad, mid, far);
    return bad != 0 || mid < 50000 || far < 50000;
}
"""


def test_int_exponents_give_the_same_bits():
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        open(src, "w").write(PROGRAM)
        subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wno-deprecated-declarations", "-I" + os.path.join(PKG, "csrc"), "-I/usr/local/cuda/include", src, "-o", exe])
        out = subprocess.run([exe], capture_output=True, text=True)
        print(out.stdout)
        assert out.returncode == 0, out.stdout + out.stderr
