"""Batches whose frames render on their own threads beside the shared passes, and
batches in the learned order (calls of 32 lane budgets): the outputs of frames
rendered alone; and the error that a batch reports."""
import numpy as np
import pytest

import mbx
import order_train
import views

pytestmark = pytest.mark.gpu


@pytest.fixture()
def be():
    b = mbx.create_compute_backend("cuda")
    yield b
    b.close()


def _deep(depth, w, h):
    v = views.deep_view(depth)
    return mbx.ComputeRequest(v["center_re"], v["center_im"], v["scale"], w, h, v["max_iterations"], bailout=v["bailout"], precision_mode=mbx.PRECISION_MIXED)


def _shallow(w, h, cm=0):
    return mbx.ComputeRequest("-0.6", "0.01", "1", w, h, 2000, coloring_method=cm)


def _check(be, make, repeats=2):
    alone = []
    for f in make:
        r = f()
        assert be.compute_status(r) == mbx.OK, be.last_error()
        alone.append((r.iterations.copy(), r.escape_iteration.copy()))
    for _ in range(repeats):
        reqs = [f() for f in make]
        assert be.compute_batch(reqs) == mbx.OK, be.last_error()
        for r, (it, en) in zip(reqs, alone):
            assert np.array_equal(r.escape_iteration, en) and np.array_equal(r.iterations, it)


# frames of at least 20,000 pixels render on their own here
@pytest.mark.parametrize("make", [
    [lambda: _shallow(200, 150)],                                                                    # one frame
    [lambda: _shallow(200, 150), lambda: _deep(300, 240, 135), lambda: _shallow(222, 111, mbx.DE_OVERLAY)], # large ones only
    [lambda: _deep(1000, 240, 135)] * 6 + [lambda: _deep(300, 96, 54)],                              # more large ones than threads
    [lambda: _deep(300, 96, 54)] * 5 + [lambda: _deep(1000, 240, 135)] + [lambda: _shallow(60, 40)], # one large one
], ids=["one", "large", "many", "mixed"])
def test_own_frames_are_those_rendered_alone(be, make):
    assert be.set_batch_direct(20000) == mbx.OK
    _check(be, make)


def test_first_frame_that_failed_is_reported(be):
    assert be.set_batch_direct(20000) == mbx.OK
    def own_bad():
        r = _deep(300, 222, 111)
        r.reference_re, r.reference_im, r.reference_period = "x", "0", 3  # "unparsable reference nucleus"
        return r
    def shared_bad():
        r = _deep(300, 96, 54)
        r.scale = "x"  # "unparsable centre or scale"
        return r
    good = [lambda: _deep(300, 96, 54), lambda: _shallow(200, 150)]
    for make, want in (([good[0], own_bad, shared_bad, good[1]], "reference nucleus"), ([good[1], shared_bad, good[0], own_bad], "centre or scale"), ([good[0], own_bad, good[1]], "reference nucleus"),
                       ([own_bad], "reference nucleus"), ([good[1], shared_bad], "centre or scale")):
        assert be.compute_batch([f() for f in make]) == mbx.E_INVALID
        assert want in be.last_error(), (want, be.last_error())
        assert be.compute_batch([f() for f in good]) == mbx.OK, be.last_error()


def test_calls_of_32_budgets_change_no_output(be):
    """As many samples as take long calls (more than twice 152 x 768 lanes), in the
    order of the untrained model."""
    sizes = [(400, 256), (384, 288), (480, 200)]
    alone = []
    for w, h in sizes:
        r = _deep(300, w, h)
        assert be.compute_status(r) == mbx.OK, be.last_error()
        alone.append((r.iterations.copy(), r.escape_iteration.copy()))
    be.schedule_params(order_train.initial_params(None))
    assert be.set_batch_scheduling(2) == mbx.OK, be.last_error()
    reqs = [_deep(300, w, h) for w, h in sizes]
    assert be.compute_batch(reqs) == mbx.OK, be.last_error()
    for r, (it, en) in zip(reqs, alone):
        assert np.array_equal(r.escape_iteration, en) and np.array_equal(r.iterations, it)
