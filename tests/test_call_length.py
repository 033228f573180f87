"""Lane calls of two lengths: a pass over more than twice its resident lanes takes
eight lane budgets a call. Where calls end changes no result: frames rendered
alone (short calls) equal the same frames in a batch (long calls, one pass over
all of them), and a frame with long calls is the same at another budget."""
import numpy as np
import pytest

import mbx
import views

pytestmark = pytest.mark.gpu

COUNTERS = ("iterations_total", "interior", "bla_applies", "bla_skipped", "rebases", "effective_iterations")


def _req(depth, w, h, coloring=0):
    v = views.deep_view(depth)
    return mbx.ComputeRequest(v["center_re"], v["center_im"], v["scale"], w, h, v["max_iterations"], bailout=v["bailout"], precision_mode=mbx.PRECISION_MIXED,
                              coloring_method=coloring)


@pytest.mark.parametrize("depth", [300, 1000])
def test_batch_of_long_calls_matches_short_calls(depth):
    sizes = [(400, 256), (384, 288), (480, 200)]  # each below twice 152 x 768 lanes, together above it
    be = mbx.create_compute_backend("cuda")
    singles = []
    for w, h in sizes:
        r = _req(depth, w, h)
        assert be.compute_status(r) == mbx.OK, be.last_error()
        singles.append((r.iterations.copy(), r.escape_iteration.copy()))
    reqs = [_req(depth, w, h) for w, h in sizes]
    assert be.compute_batch(reqs) == mbx.OK, be.last_error()
    for r, (it, en) in zip(reqs, singles):
        assert np.array_equal(r.escape_iteration, en)
        assert np.array_equal(r.iterations, it)
    be.close()


@pytest.mark.parametrize("depth,coloring", [(1000, 0), (300, 2)])
def test_long_calls_at_another_budget(depth, coloring):
    be = mbx.create_compute_backend("cuda")
    out = []
    for budget in (256, 17):
        be.set_lane_budget(budget)
        r = _req(depth, 700, 400, coloring)
        assert be.compute_status(r) == mbx.OK, be.last_error()
        s = be.last_stats.as_dict()
        out.append((r.iterations.copy(), r.escape_iteration.copy(), {k: s[k] for k in COUNTERS if k in s}))
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][0], out[1][0], equal_nan=True)
    assert out[0][2] == out[1][2]
    be.close()
