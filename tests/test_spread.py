"""The order in which a small pass of the double path takes its entries
(csrc/kernels.h spread_entry): on the host, every entry exactly once for every
number of warp turns; on the GPU, frames around the rule's line (16 warp turns an
SM: 77,824 entries on 152 SMs), of less than a warp and with a part of one, a key
list and the derivative, equal to the oracle (class and escape iteration at every
sample, values within 1e-6 relative: the logarithm's library differs)."""
import os
import subprocess
import tempfile

import numpy as np
import pytest

import mbx
from conftest import PKG, load_cases

PROGRAM = r"""
#include <cuda_runtime.h>
#include "kernels.h"
#include <cstdio>
#include <vector>
int main() {
    for (int tickets : {1, 2, 3, 7, 31, 32, 33, 608, 2431, 2432, 70001}) {
        std::vector<int> seen((size_t)tickets * 32, 0);
        for (int t = 0; t < tickets; ++t)
            for (int l = 0; l < 32; ++l) {
                const int i = mbx::spread_entry(t, l, tickets);
                if (i < 0 || i >= tickets * 32) return 1;
                ++seen[(size_t)i];
            }
        for (int c : seen)
            if (c != 1) return 2;
    }
    return 0;
}
"""


def test_every_entry_once():
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        open(src, "w").write(PROGRAM)
        subprocess.check_call(["g++", "-std=c++17", "-O2", "-I" + os.path.join(PKG, "csrc"), "-I/usr/local/cuda/include", src, "-o", exe])
        assert subprocess.run([exe]).returncode == 0


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,cm,sub", [(5, 3, 0, 1), (33, 31, 2, 1), (48, 104, 0, 1), (304, 256, 0, 1), (389, 200, 0, 1), (311, 251, 64, 1), (120, 67, 1, 3)])
def test_double_path_frames(w, h, cm, sub):
    import oracle

    c = load_cases()["c1"]
    args = (c["center_re"], c["center_im"], c["scale"], w, h, c["max_iterations"])
    be = mbx.create_compute_backend("cuda")
    try:
        r = mbx.ComputeRequest(*args, sub=sub, coloring_method=cm, bailout=c["bailout"])
        assert be.compute_status(r) == mbx.OK, be.last_error()
        assert be.last_stats.as_dict()["used_floatexp"] == 0
    finally:
        be.close()
    it, _, en, _ = oracle.render(*args, sub=sub, coloring_method=cm, bailout=c["bailout"])
    assert np.array_equal(r.escape_iteration, en) and np.array_equal(r.iterations < -1.5, it < -1.5)
    np.testing.assert_allclose(r.iterations, it, rtol=1e-6, atol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,cm,sub", [(5, 3, 0, 1), (48, 104, 0, 1), (304, 256, 0, 1), (311, 251, 64, 1), (60, 33, 1, 3)])
def test_frames_with_interior(w, h, cm, sub):
    """Frames whose probe finds interior take the order in the main pass: the cusp
    of the period-3 minibrot on the needle."""
    import oracle

    args = ("-1.7499996", "0.0000001", "2000000", w, h, 20000)
    be = mbx.create_compute_backend("cuda")
    try:
        r = mbx.ComputeRequest(*args, sub=sub, coloring_method=cm, bailout=256.0)
        assert be.compute_status(r) == mbx.OK, be.last_error()
        assert be.last_stats.as_dict()["used_floatexp"] == 0
    finally:
        be.close()
    it, _, en, _ = oracle.render(*args, sub=sub, coloring_method=cm, bailout=256.0)
    assert (en < 0).any() and np.array_equal(r.escape_iteration, en) and np.array_equal(r.iterations < -1.5, it < -1.5)
    np.testing.assert_allclose(r.iterations, it, rtol=1e-6, atol=0)
