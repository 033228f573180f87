"""The direct kernel (kernels_exact.cu k_direct) where it takes blocks of 512
threads: from 512 samples per SM (77,824 on 152 SMs) on, with more than 48 KB of
dynamic shared memory, lanes refilled from the work counter and last samples
packed over the block. Every form, the last size below, the first of them and
ragged ones, against the oracle: class and escape iteration equal at every
sample, values within 1e-6 relative (the logarithm's library differs). Normal
angles are differences of two arguments up to pi, each within 2^-51: 1e-13 beside
the relative bound."""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

import mbx
import oracle
from test_zz_no_alloc import trunc53

pytestmark = pytest.mark.gpu

SS, EDE, SAC, NORMAL, TRAP, OVERLAY = 1, 2, 8, 16, 32, 64
RTOL, ANGLE = 1e-6, 1e-13


@pytest.fixture(scope="module")
def be():
    b = mbx.create_compute_backend("cuda")
    yield b
    b.close()


def _same(r, it, nr, en, angles):
    assert np.array_equal(r.escape_iteration, en)
    assert np.array_equal(r.iterations < -1.5, it < -1.5)
    np.testing.assert_allclose(r.iterations, it, rtol=RTOL, atol=0)
    if angles:
        np.testing.assert_allclose(r.normal, nr, rtol=RTOL, atol=ANGLE)


@pytest.mark.parametrize("w,h", [(304, 255), (304, 256), (311, 251), (607, 389)])
@pytest.mark.parametrize("cm", [0, EDE, OVERLAY, NORMAL, SAC, TRAP, SAC | EDE, TRAP | OVERLAY, SAC | TRAP])
def test_shallow_forms(be, w, h, cm):
    args = ("-0.6", "0.01", "1", w, h, 1500)
    r = mbx.ComputeRequest(*args, coloring_method=cm, bailout=1e8)
    if cm & (NORMAL | OVERLAY):
        r.normal = np.full(w * h, 7.0, np.float32)
    assert be.compute_status(r) == mbx.OK, be.last_error()
    it, nr, en, _ = oracle.render(*args, coloring_method=cm, bailout=1e8)
    # (under a trap the oracle leaves the overlay's distances out)
    _same(r, it, nr, en, bool(cm & (NORMAL | OVERLAY)) and not cm & TRAP)


@pytest.mark.parametrize("cm", [0, EDE, SAC, TRAP])
def test_supersampled_key_lists(be, cm):
    """sub 3: the second pass takes a list of the sub-samples near the set, here
    of more than 77,824 entries."""
    args = ("-0.6", "0.01", "1", 1401, 933, 1000)
    r = mbx.ComputeRequest(*args, sub=3, coloring_method=cm | SS, bailout=1e8)
    assert be.compute_status(r) == mbx.OK, be.last_error()
    assert be.last_stats.as_dict()["samples"] > 1401 * 933 + 77824
    it, nr, en, _ = oracle.render(*args, sub=3, coloring_method=cm | SS, bailout=1e8)
    _same(r, it, nr, en, False)


def test_strip(be):
    args = ("-0.6", "0.01", "1", 512, 203, 1000)
    r = mbx.ComputeRequest(*args, bailout=1e8, full_height=512, row_base=131)
    assert be.compute_status(r) == mbx.OK, be.last_error()
    it, nr, en, _ = oracle.render(*args, bailout=1e8, full_height=512, row_base=131)
    _same(r, it, nr, en, False)


@pytest.mark.parametrize("w,h", [(304, 255), (304, 256), (353, 251), (807, 461)])
@pytest.mark.parametrize("cm", [0, EDE])
@pytest.mark.parametrize("c", [("-0.123", "0.745"), ("0", "1")])
def test_julia_forms(be, w, h, cm, c):
    r = mbx.ComputeRequest("0.01", "-0.02", "1.1", w, h, 2000, coloring_method=cm, bailout=256.0, compute_mode=mbx.MODE_JULIA, fixed_c_re=c[0], fixed_c_im=c[1])
    assert be.compute_status(r) == mbx.OK, be.last_error()
    it, en = oracle.julia("0.01", "-0.02", "1.1", c[0], c[1], w, h, 2000, cm, 256.0)
    _same(r, it, None, en, False)


def test_noalloc_entry_point():
    """The allocation-free entry point at 512 x 257 (centre (-0.5, 0), scale 1:
    half-width 2, half-height 257/256) against the regular one, bit for bit."""
    torch = pytest.importorskip("torch")
    w, h, mxit = 512, 257, 2000
    for cm in (0, EDE, OVERLAY):
        b = mbx.create_compute_backend("cuda")
        r = mbx.ComputeRequest("-0.5", "0", "1", w, h, mxit, coloring_method=cm, bailout=1e8)
        if cm & OVERLAY:
            r.normal = np.empty(w * h, np.float32)
        assert b.compute_status(r) == mbx.OK, b.last_error()
        b.close()
        it = torch.full((w * h,), 123.0, dtype=torch.float32, device="cuda")
        en = torch.full((w * h,), 7, dtype=torch.int32, device="cuda")
        nr = torch.full((w * h,), 55.0, dtype=torch.float32, device="cuda") if cm & OVERLAY else None
        rc = mbx.load_library().mbx_render_shallow_noalloc(-2.5, -float(Fraction(257, 256)), 2.0 * trunc53(Fraction(2, 511)), float(2 * Fraction(257, 256) / 256), w, h, mxit, 1e8, cm,
                                                           ctypes.c_void_p(it.data_ptr()), ctypes.c_void_p(en.data_ptr()), ctypes.c_void_p(nr.data_ptr()) if nr is not None else None, None)
        assert rc == mbx.OK
        assert np.array_equal(it.cpu().numpy().view(np.uint32), r.iterations.view(np.uint32))
        assert np.array_equal(en.cpu().numpy(), r.escape_iteration)
        if nr is not None:
            assert np.array_equal(nr.cpu().numpy().view(np.uint32), r.normal.view(np.uint32))
