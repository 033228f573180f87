"""Exponents beyond 32 bits in the floatexp arithmetic (csrc/floatexp.h): a scale
may be written 1e400000000, whose |dz|^2 lies below 2^-(2^31).

* on the host: an operation on operands shifted by 2^k gives the unshifted
  operation's mantissa bits, its exponent shifted, at shifts past 2^31 and 2^32;
* on the GPU: at such a scale every sample of a frame is the centre's own orbit,
  whose count and value plain arithmetic gives.
"""
import math
import os
import subprocess
import tempfile

import numpy as np
import pytest

import mbx
from conftest import PKG

PROGRAM = r"""
#include "floatexp.h"
#include <cstdio>
#include <random>
using namespace mbx;
int main() {
    std::mt19937_64 g(5);
    std::uniform_real_distribution<double> u(-1, 1);
    long bad = 0;
    auto same = [&](FE got, FE want, int64_t k) {
        const bool zero = d_is_zero(want.m);
        if (dbits(got.m) != dbits(want.m) || (!zero && got.e != want.e + k)) ++bad;
    };
    const int64_t shifts[] = {0, 2000000000, -2000000000, 2658000000, -2658000000, -(1ll << 33), (1ll << 40)};
    for (int n = 0; n < 200000; ++n) {
        const FE a = fe_renorm(u(g), (int64_t)(60 * u(g))), b = fe_renorm(u(g), (int64_t)(60 * u(g)));
        for (int64_t k : shifts) {
            const FE A = fe_make(a.m, a.e + k), B = fe_make(b.m, b.e + k);
            same(fe_mul(A, B), fe_mul(a, b), 2 * k);
            same(fe_mul_d(A, b.m), fe_mul_d(a, b.m), k);
            same(fe_add(A, B), fe_add(a, b), k);
            same(fe_sub(A, B), fe_sub(a, b), k);
            same(fe_add(A, b), k > 200 ? A : (k < -200 ? b : fe_add(a, b)), 0);
            same(fe_div<true>(A, b), fe_div<true>(a, b), k);
            same(fe_div(b, A), fe_div(b, a), -k);
            same(fe_sqrt(fe_mul(A, A)), fe_sqrt(fe_mul(a, a)), k);
            same(fe_scale2(a, k), a, k);
            bad += fe_abs_less(A, B) != fe_abs_less(a, b);
            if (k > 200) bad += fe_abs_less(A, b) || !std::isinf(fe_to_double(A));
            if (k < -200) bad += !fe_abs_less(A, b) || fe_to_double(A) != 0.0;
        }
    }
    printf("%ld bad\n", bad);
    return bad != 0;
}
"""


def test_exponents_past_32_bits():
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        open(src, "w").write("#include <cmath>\n" + PROGRAM)
        subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I" + os.path.join(PKG, "csrc"), src, "-o", exe])
        out = subprocess.run([exe], capture_output=True, text=True)
        assert out.returncode == 0, out.stdout + out.stderr


def _orbit(c, maxiter, bailout):
    """The reference's count and smooth value of one point."""
    z = c
    for n in range(2, maxiter + 1):
        z = z * z + c
        if abs(z) > bailout:
            return n, n - math.log(math.log(abs(z) ** 2) / 2 / math.log(2)) / math.log(2)
    return -1, -2.0


@pytest.mark.gpu
@pytest.mark.parametrize("scale", ["1e300000000", "1e400000000", "1e640000000"])
@pytest.mark.parametrize("mode", [mbx.PRECISION_EXACT, mbx.PRECISION_MIXED])
def test_frames_past_2_to_the_31st(scale, mode):
    be = mbx.create_compute_backend("cuda")
    try:
        for c in (1 + 0j, 0.3 + 0.6j, -0.1 + 0.7j):
            n, v = _orbit(c, 300, 256.0)
            r = mbx.ComputeRequest(repr(c.real), repr(c.imag), scale, 24, 16, 300, bailout=256.0, precision_mode=mode)
            assert be.compute_status(r) == mbx.OK, be.last_error()
            assert np.all(r.escape_iteration == n), (c, np.unique(r.escape_iteration))
            np.testing.assert_allclose(r.iterations, v, rtol=1e-6)
    finally:
        be.close()
