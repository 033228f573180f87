"""The arithmetic that takes other operations on the device than on the host
(approximate seeds, rsqrt), on the device: the integer quotient and square root
(csrc/floatexp.h) bit for bit beside the FP64 unit's correctly rounded ones; the
escape values and shadings in pairs of floats (csrc/smooth.cuh, color_math.cuh)
equal to the float of their double expression wherever they settle it; the
stripe term (csrc/orbit_color.h) within 2e-14 of sin(7 arg z): 7 times two units
of atan2's last place (6.2e-15), the product's rounding (1.8e-15), sin's own and
the term's (below 3e-15)."""
import os
import subprocess
import tempfile

import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include "smooth.cuh"
#include "orbit_color.h"
#include <cstdio>
using namespace mbx;
struct Rng {
    unsigned long long s;
    __device__ unsigned long long next() { // splitmix64
        unsigned long long z = (s += 0x9e3779b97f4a7c15ull);
        z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
        z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
        return z ^ (z >> 31);
    }
    __device__ double u() { return (double)(next() >> 11) * 0x1p-53; }
};
enum { kDiv, kSqrt, kSmooth, kDistance, kRelief, kShaded, kSin7, kKinds };
__device__ unsigned long long bad[kKinds], left[kKinds], seen[kKinds];
__device__ void check(int k, bool settled, bool same) {
    atomicAdd(&seen[k], 1ull);
    if (!settled) atomicAdd(&left[k], 1ull);
    else if (!same) atomicAdd(&bad[k], 1ull);
}
__device__ double num(Rng& g) { // few or nearly all bits set, all exponents
    const unsigned long long r = g.next();
    unsigned long long f = g.next() & 0xfffffffffffffull;
    if (r % 5 == 0) f = g.next() & 0xf;
    if (r % 5 == 1) f = 0xfffffffffffffull ^ (g.next() & 0xf);
    if (r % 5 == 2) f = (g.next() & 0xff) << 44;
    if (r % 13 == 0) f = 1ull << (g.next() % 52);
    if (r % 11 == 0) f = 0xfffffffffffffull ^ (g.next() & 0x1fffffffull); // a divisor whose top 32 bits round to 2^32 in a float
    if (r % 17 == 0) f = g.next() & 0x3fffffffull;                         // a radicand beside a power of two
    const unsigned long long e = r & 64 ? 1022 + (r >> 8) % 3 : (r >> 8) % 2048;
    return bitsd(((r >> 63) << 63) | (e << 52) | f);
}
__device__ bool eq(double p, double q) { return dbits(p) == dbits(q) || (p != p && q != q); }
__global__ void k_check(int rounds, cm::ReliefParams rp, double strength, double lx, double ly, double lz) {
    Rng g{(blockIdx.x * blockDim.x + threadIdx.x) * 0x2545f4914f6cdd1dull};
    for (int i = 0; i < rounds; ++i) {
        const double a = num(g), b = num(g);
        check(kDiv, true, eq(int_div(a, b), __ddiv_rn(a, b)));
        check(kSqrt, true, eq(int_sqrt(a), __dsqrt_rn(a)) && eq(int_sqrt(dabs(b)), __dsqrt_rn(dabs(b))));
        for (int d = -1; d <= 1; ++d) { // beside representable quotients and roots
            const double p = bitsd(dbits(a * b) + (unsigned long long)(long long)d), q = bitsd((dbits(a * a) + (unsigned long long)(long long)d) & 0x7fffffffffffffffull);
            check(kDiv, true, eq(int_div(p, b), __ddiv_rn(p, b)));
            check(kSqrt, true, eq(int_sqrt(q), __dsqrt_rn(q)));
        }
        const double h = dabs(__fma_rn(a, a, a * 0x1p-52)); // beside a halfway root
        check(kSqrt, true, eq(int_sqrt(h), __dsqrt_rn(h)));

        float out;
        const double ln2 = 0x1.62e42fefa39efp-1;
        const double zrad = i % 3 ? exp2(1.0 + 239.0 * g.u()) : exp2(exp2(1.0 + 6.0 * g.u()));
        const int n = 1 + (int)exp2(24.0 * g.u()) % (1 << 24);
        bool ok = smooth_pair(n, zrad, out);
        check(kSmooth, ok, out == (float)((double)n - log(log(zrad) / 2 / ln2) / ln2));
        const double s = exp2(60.0 * (g.u() - 0.3)), da = (2 * g.u() - 1) * s, db = (2 * g.u() - 1) * s * (i % 5 ? 1.0 : 1e-9);
        if (log_pair_takes(zrad)) {
            ok = distance_pair(zrad, da, db, out);
            check(kDistance, ok, out == (float)(sqrt(zrad) * log(zrad) / sqrt(da * da + db * db)));
        }
        const float sc = (float)exp2(40.0 * g.u() - 20.0), sx = (float)(2 * g.u() - 1) * sc, sy = (float)(2 * g.u() - 1) * (i % 4 ? sc : 0.0f);
        ok = cm::relief_ff(sx, sy, rp, out);
        const double nx = __dmul_rn((double)(-sx), strength), ny = __dmul_rn((double)(-sy), strength);
        const double inv = __ddiv_rn(1.0, __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(nx, nx), __dmul_rn(ny, ny)), 1.0)));
        double dd = __dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(nx, lx), __dmul_rn(ny, ly)), lz), inv);
        if (dd < 0) dd = 0;
        const float shade = (float)__dadd_rn(0.25, __dmul_rn(0.85, dd));
        check(kRelief, ok, out == shade);
        const float acc = (float)(9.0 * g.u()), c = (float)g.u();
        ok = cm::acc_shaded_ff(acc, c, shade, out);
        check(kShaded, ok, out == (float)__dadd_rn((double)acc, __dmul_rn((double)c, (double)shade)));
        const double zr = (2 * g.u() - 1) * exp2(30.0 * (g.u() - 0.5)), zi = (2 * g.u() - 1) * exp2(30.0 * (g.u() - 0.5));
        check(kSin7, true, fabs(stripe_sin7(zr, zi) - sin(7.0 * atan2(zi, zr))) < 2e-14);
    }
}
int main() {
    unsigned long long b[kKinds] = {}, l[kKinds] = {}, s[kKinds] = {}, total = 0;
    const char* name[kKinds] = {"int_div", "int_sqrt", "smooth_pair", "distance_pair", "relief_ff", "acc_shaded_ff", "stripe_sin7"};
    const double strengths[] = {1.0, 0.03, 47.0};
    for (double st : strengths) {
        const double az = 2.3, el = 0.55, lx = cos(el) * cos(az), ly = cos(el) * sin(az), lz = sin(el);
        const cm::ReliefParams rp{cm::ff_from(st), cm::ff_from(lx), cm::ff_from(ly), cm::ff_from(lz)};
        k_check<<<152, 128>>>(200, rp, st, lx, ly, lz);
    }
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    cudaMemcpyFromSymbol(b, bad, sizeof(b));
    cudaMemcpyFromSymbol(l, left, sizeof(l));
    cudaMemcpyFromSymbol(s, seen, sizeof(s));
    for (int k = 0; k < kKinds; ++k) {
        printf("%s: %llu bad, %llu left to the double expression of %llu\n", name[k], b[k], l[k], s[k]);
        total += b[k];
        if (!s[k] || l[k] * 20 > s[k]) total += 1; // settled nearly everywhere
    }
    return total != 0;
}
"""


def test_device_forms_round_as_the_double_expressions():
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cu"), os.path.join(d, "t")
        open(src, "w").write(PROGRAM)
        nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
        subprocess.check_call([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2", "-fmad=false", "--expt-relaxed-constexpr", "-Xcompiler", "-ffp-contract=off",
                               "-I" + os.path.join(PKG, "csrc"), src, "-o", exe])
        out = subprocess.run([exe], capture_output=True, text=True)
        print(out.stdout)
        assert out.returncode == 0, out.stdout + out.stderr
