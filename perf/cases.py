"""The renderer's work, as timed cases: what a user has it do, through its public
entry points, from an interactive thumbnail to a batch of deep-zoom tiles.

Sizes and views are those of the repository's benchmark, view generators and
tests (views.py, zoom.py, tests/golden). Every frame is a whole call on a
backend that the program keeps: geometry, reference, passes, outputs. Seeds
move the view's centre, the Julia constant or the chosen tiles, so that each
state is another frame of the same kind.
"""
import math
import os
import random
import sys
from decimal import Decimal, getcontext
from fractions import Fraction

import numpy as np
import torch

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mandelbrot-explorer_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import mbx  # noqa: E402
import views  # noqa: E402
import zoom  # noqa: E402

SS, EDE, SAC, NORMAL, TRAP, OVERLAY = 1, 2, 8, 16, 32, 64
LN2 = math.log(2.0)

# Julia constants of the test fixtures: the rabbit (an interior with period 3),
# the dendrite (all exterior, long escapes near it) and a Siegel disk's boundary.
JULIA_C = {"rabbit": (-0.123, 0.745), "dendrite": (0.0, 1.0), "siegel": (-0.390540870218399, -0.586787907346969)}


def listed():
    return [
        # The smallest call: a Julia thumbnail redrawn as the constant follows the
        # mouse. Launches, copies and waits count here, not the loop.
        {"name": "julia_thumbnail", "kind": "julia", "c": "rabbit", "width": 160, "height": 120, "scale": 1.0, "maxiter": 2000, "coloring": 0, "device": False, "steps": 220},
        # A full-screen Julia frame with distance estimation, left on the GPU for display.
        {"name": "julia_1080p_ede", "kind": "julia", "c": "dendrite", "width": 1920, "height": 1080, "scale": 1.2, "maxiter": 3000, "coloring": EDE, "device": True, "steps": 7},
        # The first view of every session: the whole set, in a window, read back by the GUI.
        {"name": "shallow_720p", "kind": "shallow", "width": 1280, "height": 720, "scale": 1.0, "maxiter": 5000, "coloring": 0, "sub": 1, "device": False, "steps": 100},
        # The stripe-average colouring with adaptive 3x3 supersampling (the tests'
        # shallow_sac_ss3 at preview size): the scalar loop with its window, then the key-list pass.
        {"name": "shallow_stripe_ss3", "kind": "shallow", "width": 601, "height": 399, "scale": 1.0, "maxiter": 5000, "coloring": SAC | SS, "sub": 3, "device": False, "steps": 150},
        # The render tool: values, distance overlay and the colour pass in one call,
        # 4 samples a pixel, the RGB image read back.
        {"name": "image_overlay_ss2", "kind": "image", "width": 2560, "height": 1440, "scale": 20.0, "maxiter": 2000, "coloring": OVERLAY, "ss": 2, "shading": 3, "steps": 100},
        # The plain FP64 workload's size, depth and maxiter (1280x720, half-width 1e-30,
        # 50,000) beside the zoom target, which has structure at every depth: the
        # default (exact) precision, reference orbits made anew each call.
        {"name": "double_path_720p", "kind": "double", "width": 1280, "height": 720, "depth": 30.0, "maxiter": 50000, "coloring": 0, "device": False, "steps": 400},
        # The 1e-300 benchmark frame in the default precision: the exact floatexp loop at 1080p.
        {"name": "floatexp_exact_1080p", "kind": "deep", "view": "1e-300", "width": 1920, "height": 1080, "maxiter": 1000000, "coloring": 0, "mixed": False, "device": False, "steps": 570},
        # The benchmark's target frame: a 1e-1000 minibrot and its surroundings at 1080p,
        # mixed precision, all tiers at work.
        {"name": "minibrot_mixed_1080p", "kind": "deep", "view": "1e-1000-minibrot", "width": 1920, "height": 1080, "maxiter": 1000000, "coloring": 0, "mixed": True, "device": False, "steps": 320},
        # One frame of the 600-frame zoom at 1080p with distance estimation: the program
        # keeps the backend, which keeps the shared reference orbit.
        {"name": "zoom_frame_1080p_ede", "kind": "zoom", "frame": 300, "width": 1920, "height": 1080, "coloring": EDE, "device": True, "steps": 900},
        # A storyboard of a zoom: views of uneven size, depth and maxiter in one call, half
        # of them with adaptive 3x3 supersampling (the batching workload at a quarter of its
        # linear sizes), all naming the zoom's nucleus as their reference.
        {"name": "batch_views", "kind": "batch", "views": 16, "shape_seed": 3, "size_div": 4, "steps": 1500},
        # 24 tiles of the 23040x12960 image at 1e-500, maxiter 2e6, in one call on one shared orbit.
        {"name": "batch_tiles", "kind": "tiles", "tiles": 24, "tile": 256, "steps": 1500},
        # Recolouring a supersampled frame that is on the GPU: the light or the density changed.
        {"name": "recolour_1080p_ss3", "kind": "colour", "width": 1920, "height": 1080, "ss": 3, "mapping": 0, "shading": 1, "steps": 0},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["julia", "shallow", "image", "double", "deep", "zoom", "batch", "tiles", "colour", "shallow", "zoom"])
    if kind == "julia":
        w = _logint(rng, 48, 1920)
        return {"kind": kind, "c": rng.choice(sorted(JULIA_C)), "width": w, "height": max(32, int(w * rng.uniform(0.4, 0.8))), "scale": round(math.exp(rng.uniform(-0.2, 3.0)), 4),
                "maxiter": _logint(rng, 200, 5000), "coloring": rng.choice([0, EDE]), "device": rng.random() < 0.5, "steps": 300}
    if kind == "shallow":
        w, cm = _logint(rng, 48, 1920), rng.choice([0, 0, EDE, NORMAL, OVERLAY, SAC, TRAP])
        sub = 3 if w <= 640 and cm in (0, EDE, SAC, TRAP) and rng.random() < 0.5 else 1
        return {"kind": kind, "width": w, "height": max(32, int(w * rng.uniform(0.4, 0.8))), "scale": round(math.exp(rng.uniform(0.0, math.log(1e5))), 4),
                "maxiter": _logint(rng, 500, 5000), "coloring": cm | (SS if sub > 1 else 0), "sub": sub, "device": rng.random() < 0.5, "steps": 500}
    if kind == "image":
        ss = rng.choice([1, 2, 3])
        w = _logint(rng, 64, 1280 // ss) * ss
        cm, sh = rng.choice([(0, 0), (0, 1), (NORMAL, 2), (OVERLAY, 3)])
        return {"kind": kind, "width": w, "height": max(16, int(w / ss * rng.uniform(0.4, 0.8))) * ss, "scale": round(math.exp(rng.uniform(0.0, math.log(1e4))), 4),
                "maxiter": _logint(rng, 500, 3000), "coloring": cm, "ss": ss, "shading": sh, "steps": 300}
    if kind == "double":
        w = _logint(rng, 48, 1280)
        return {"kind": kind, "width": w, "height": max(32, int(w * rng.uniform(0.4, 0.7))), "depth": round(rng.uniform(8.0, 30.0), 3), "maxiter": _logint(rng, 5000, 50000),
                "coloring": rng.choice([0, 0, EDE, NORMAL, OVERLAY, SAC]), "device": rng.random() < 0.5, "steps": 400}
    if kind == "deep":
        w = _logint(rng, 48, 800)
        mixed = rng.random() < 0.5
        return {"kind": kind, "view": rng.choice(["1e-300", "1e-1000-minibrot"]) if mixed else "1e-300", "width": w, "height": max(32, int(w * rng.uniform(0.4, 0.7))), "maxiter": 1000000,
                "coloring": rng.choice([0, 0, EDE]), "mixed": mixed, "device": rng.random() < 0.5, "steps": 1200}
    if kind == "zoom":
        w = _logint(rng, 48, 960)
        return {"kind": kind, "frame": rng.choice([rng.randint(8, 18), rng.randint(180, 480)]), "width": w, "height": max(32, int(w * rng.uniform(0.4, 0.7))), "coloring": rng.choice([0, EDE, EDE, NORMAL, OVERLAY]),
                "device": rng.random() < 0.5, "steps": 900}
    if kind == "batch":
        return {"kind": kind, "views": rng.randint(6, 12), "shape_seed": rng.randint(10, 9999), "size_div": 8, "steps": 1500}
    if kind == "tiles":
        return {"kind": kind, "tiles": rng.randint(6, 16), "tile": rng.choice([64, 96, 128, 160, 192]), "steps": 1500}
    return {"kind": "colour", "width": _logint(rng, 48, 1920), "height": _logint(rng, 32, 1080), "ss": rng.choice([1, 2, 3]), "mapping": rng.choice([0, 0, 1, 2, 3]),
            "shading": rng.choice([0, 1, 2, 3]), "steps": 0}


def _buffers(req, device):
    """The output buffers that a program keeps from frame to frame."""
    n = req.sample_count()
    if device:
        req.iterations = torch.empty(n, dtype=torch.float32, device="cuda")
        req.escape_iteration = torch.empty(n, dtype=torch.int32, device="cuda")
        if req.coloring_method & (NORMAL | OVERLAY):
            req.normal = torch.empty(n, dtype=torch.float32, device="cuda")
    else:
        req.iterations = np.empty(n, np.float32)
        req.escape_iteration = np.empty(n, np.int32)
        if req.coloring_method & (NORMAL | OVERLAY):
            req.normal = np.empty(n, np.float32)
    return req


def _julia_numbers(case, seed):
    rng = random.Random(seed)
    cr, ci = JULIA_C[case["c"]]
    cr, ci = cr + rng.uniform(-1e-3, 1e-3), ci + rng.uniform(-1e-3, 1e-3)
    return repr(rng.uniform(-0.05, 0.05)), repr(rng.uniform(-0.05, 0.05)), repr(case["scale"]), repr(cr), repr(ci)


def _shallow_numbers(case, seed):
    rng = random.Random(seed)
    re, im = (-0.5, 0.0) if case["scale"] < 4.0 else (-0.7436438870371587, 0.1318259042053120)
    step = 0.2 / case["scale"]
    return repr(re + rng.uniform(-step, step)), repr(im + rng.uniform(-step, step)), repr(case["scale"])


def _offset(re, im, half_width, share, rng):
    """The centre moved by `share` half-widths in a drawn direction (decimal strings)."""
    getcontext().prec = max(len(re), len(im)) + 20
    a = rng.uniform(0.0, 2.0 * math.pi)
    step = Decimal(repr(share)) * half_width
    return format(Decimal(re) + step * Decimal(repr(math.cos(a))), "f"), format(Decimal(im) + step * Decimal(repr(math.sin(a))), "f")


def _batch_requests(case, seed):
    """views.c3_views' workload with sizes, depths and maxiters (at least what the depth
    needs, about 30 a decade here) from the case and the views' centres from the seed."""
    d, shape, rng = views.nucleus()["zoom"], np.random.RandomState(case["shape_seed"]), random.Random(seed)
    n = case["views"]
    ss = set(shape.permutation(n)[: n // 2].tolist())
    out = []
    for i in range(n):
        size = int(shape.choice([256, 512, 1024, 2048, 4096])) // case["size_div"]
        depth, maxiter = float(shape.uniform(20.0, 600.0)), int(round(10 ** shape.uniform(4.0, 6.0)))
        maxiter = max(maxiter, int(60 * depth))
        half = Decimal(10) ** Decimal(repr(-depth))
        re, im = _offset(d["nucleus_re"], d["nucleus_im"], half, 0.3, rng)
        out.append(_buffers(mbx.ComputeRequest(re, im, format((Decimal(2) / half).normalize(), "E").replace("E+", "e"), size, size, maxiter, sub=3 if i in ss else 1,
                                               coloring_method=SS if i in ss else 0, bailout=256.0, precision_bits=zoom.ZOOM_PRECISION,
                                               precision_mode=mbx.PRECISION_MIXED, reference_re=d["nucleus_re"], reference_im=d["nucleus_im"],
                                               reference_period=d["period"]), False))
    return out


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "backend": mbx.create_compute_backend("cuda")}
    if kind == "julia":
        re, im, scale, cr, ci = _julia_numbers(case, seed)
        req = mbx.ComputeRequest(re, im, scale, case["width"], case["height"], case["maxiter"], coloring_method=case["coloring"], bailout=256.0, compute_mode=mbx.MODE_JULIA,
                                 fixed_c_re=cr, fixed_c_im=ci, precision_bits=64)
        state["request"] = _buffers(req, case["device"])
    elif kind in ("shallow", "image"):
        re, im, scale = _shallow_numbers(case, seed)
        req = mbx.ComputeRequest(re, im, scale, case["width"], case["height"], case["maxiter"], sub=case.get("sub", 1), coloring_method=case["coloring"], precision_bits=128)
        if kind == "image":
            req.want_escape_iteration = False
            state["params"] = mbx.ColorParams(supersample=case["ss"], shading=case["shading"])
            state["request"] = req
        else:
            state["request"] = _buffers(req, case["device"])
    elif kind == "double":
        d, half = views.nucleus()["zoom"], Decimal(10) ** Decimal(repr(-case["depth"]))
        re, im = _offset(d["nucleus_re"][:80], d["nucleus_im"][:80], half, 0.3, random.Random(seed))
        scale = format((Decimal(2) / half).normalize(), "f")
        req = mbx.ComputeRequest(re, im, scale, case["width"], case["height"], case["maxiter"], coloring_method=case["coloring"], bailout=256.0)
        state["request"] = _buffers(req, case["device"])
    elif kind == "deep":
        make = views.minibrot_view if case["view"].endswith("minibrot") else lambda **kw: views.deep_view(int(case["view"][3:]), **kw)
        v = make(seed=1 + seed % 4000000, width=case["width"], height=case["height"], max_iterations=case["maxiter"])
        req = mbx.ComputeRequest(v["center_re"], v["center_im"], v["scale"], v["width"], v["height"], v["max_iterations"], coloring_method=case["coloring"], bailout=v["bailout"],
                                 precision_mode=mbx.PRECISION_MIXED if case["mixed"] else mbx.PRECISION_EXACT)
        state["request"] = _buffers(req, case["device"])
    elif kind == "zoom":
        rng = random.Random(seed)
        req = zoom.request(case["frame"] + rng.randint(-2, 2), case["width"], case["height"], coloring_method=case["coloring"])
        req.center_re, req.center_im = _offset(req.center_re, req.center_im, Decimal(2) / Decimal(req.scale), 0.25, rng)
        state["request"] = _buffers(req, case["device"])
    elif kind == "batch":
        state["requests"] = _batch_requests(case, seed)
    elif kind == "tiles":
        state["requests"] = []
        for v in views.c4_tiles(seed, case["tiles"], case["tile"]):
            state["requests"].append(_buffers(mbx.ComputeRequest(
                v["center_re"], v["center_im"], v["scale"], v["width"], v["height"], v["max_iterations"], bailout=v["bailout"], precision_bits=v["precision_bits"],
                precision_mode=mbx.PRECISION_MIXED, reference_re=v["reference_re"], reference_im=v["reference_im"], reference_period=v["reference_period"]), False))
    else:
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = case["width"] * case["height"] * case["ss"] ** 2
        # what a frame holds: smooth counts over several decades and interior samples;
        # distances, stripe averages and trap values for their mappings
        if case["mapping"] == 0:
            values = torch.exp(torch.rand(n, generator=g, device="cuda") * 10.0) + 2.0
            values[torch.rand(n, generator=g, device="cuda") < 0.1] = -2.0
        elif case["mapping"] == 1:
            values = torch.exp(torch.rand(n, generator=g, device="cuda") * 12.0 - 6.0)
            values[torch.rand(n, generator=g, device="cuda") < 0.1] = -2.0
        else:
            values = torch.rand(n, generator=g, device="cuda")
        state["values"] = values
        state["aux"] = None
        if case["shading"] == 2:
            state["aux"] = (torch.rand(n, generator=g, device="cuda") - 0.5) * (4.0 * math.pi)
        elif case["shading"] == 3:
            state["aux"] = torch.exp(torch.rand(n, generator=g, device="cuda") * 12.0 - 6.0)
        state["params"] = mbx.ColorParams(supersample=case["ss"], mapping=case["mapping"], shading=case["shading"])
        state["size"] = (case["width"], case["height"])
    return state


def _outputs(req):
    out = {"values": req.iterations, "n": req.escape_iteration}
    if req.normal is not None:
        out["normal"] = req.normal
    return out


def run(state):
    be = state["backend"]
    if state["kind"] == "colour":
        return be.colorize(state["values"], *state["size"], state["params"], state["aux"])
    if state["kind"] == "image":
        return be.render_image(state["request"], state["params"])
    if "requests" in state:
        if be.compute_batch(state["requests"]) != mbx.OK:
            raise RuntimeError(be.last_error())
        return [_outputs(r) for r in state["requests"]]
    if not be.compute(state["request"]):
        raise RuntimeError(be.last_error())
    return _outputs(state["request"])


def work(case):
    """Outputs written once, inputs read once, and 25 operations (7 for a direct
    iteration) for each executed step; `steps` is the kind's usual mean per sample."""
    if case["kind"] == "colour":
        px, n = case["width"] * case["height"], case["width"] * case["height"] * case["ss"] ** 2
        return {"bytes": n * (4 + (4 if case["shading"] >= 2 else 0)) + 3 * px, "flops": n * 60}
    if case["kind"] == "batch":
        shape, n, out = np.random.RandomState(case["shape_seed"]), 0, 0
        ss = set(shape.permutation(case["views"])[: case["views"] // 2].tolist())
        for i in range(case["views"]):
            size = int(shape.choice([256, 512, 1024, 2048, 4096])) // case["size_div"]
            shape.uniform(20.0, 600.0), shape.uniform(4.0, 6.0)
            n += size * size
            out += size * size * (9 if i in ss else 1)
        return {"bytes": 8 * out, "flops": 25 * case["steps"] * n}
    if case["kind"] == "tiles":
        n = case["tiles"] * case["tile"] ** 2
        return {"bytes": 8 * n, "flops": 25 * case["steps"] * n}
    n = case["width"] * case["height"]
    if case["kind"] == "image":
        return {"bytes": 3 * n // case["ss"] ** 2, "flops": 7 * case["steps"] * n}
    out = n * case.get("sub", 1) ** 2
    per = 12 if case["coloring"] & (NORMAL | OVERLAY) else 8
    return {"bytes": per * out, "flops": (7 if case["kind"] in ("julia", "shallow") else 25) * case["steps"] * n}


def _iterate(zr, zi, cr, ci, dr, di, plus, first, maxiter, esc2):
    """z^2 + c from z with the derivative d' = 2 z d + plus, in 64 bits, in plain
    torch operations: (count, |z|^2, |d|^2) at the first iterate outside, count -1 inside."""
    n = zr.numel()
    count = torch.full((n,), -1, dtype=torch.int64, device=zr.device)
    rad, dmag = torch.zeros_like(zr), torch.ones_like(zr)
    at = torch.arange(n, device=zr.device)
    for k in range(first, maxiter):
        dr, di = 2 * (dr * zr - di * zi) + plus, 2 * (dr * zi + di * zr)
        zr, zi = (zr * zr - zi * zi) + cr, 2 * (zr * zi) + ci
        r = zr * zr + zi * zi
        out = r > esc2
        if bool(out.any()):
            w = at[out]
            count[w], rad[w], dmag[w] = k + 1, r[out], dr[out] * dr[out] + di[out] * di[out]
            keep = ~out
            zr, zi, cr, ci, dr, di, at = zr[keep], zi[keep], cr[keep], ci[keep], dr[keep], di[keep], at[keep]
            if at.numel() == 0:
                break
    return count, rad, dmag


def _toward_zero(q):
    x = float(q)
    return math.nextafter(x, 0.0) if abs(Fraction(x)) > abs(q) else x


def exact(case, seed):
    """Shallow and Julia values by plain 64-bit iteration (smooth count, or distance
    under EDE; -2 inside). Deep frames need arbitrary precision: no value here."""
    if case["kind"] not in ("julia", "shallow") or case.get("sub", 1) != 1 or case["coloring"] not in (0, EDE):
        return None
    w, h, dev = case["width"], case["height"], "cuda" if torch.cuda.is_available() else "cpu"
    if w * h * case["maxiter"] > 7e9:
        return None
    # corner and spacings as rationals, then the doubles nearest them towards zero,
    # which is how the engine takes a double from its arbitrary-precision numbers
    given = [Fraction(t) for t in (_julia_numbers if case["kind"] == "julia" else _shallow_numbers)(case, seed)]
    re, im, scale = given[:3]
    half = 2 / scale
    tall = half * h / w
    dx, dy = 2 * half / (w - 1), 2 * tall / (h - 1)
    i, j = torch.arange(h, device=dev, dtype=torch.float64), torch.arange(w, device=dev, dtype=torch.float64)
    x = (_toward_zero(re - half) + _toward_zero(dx) * j).repeat(h)
    y = (_toward_zero(im - tall) + _toward_zero(dy) * i).repeat_interleave(w)
    if case["kind"] == "julia":
        esc2 = 256.0 ** 2
        cr, ci = [torch.full_like(x, _toward_zero(t)) for t in given[3:]]
        count, rad, dmag = _iterate(x, y, cr, ci, torch.ones_like(x), torch.zeros_like(x), 0.0, 0, case["maxiter"], esc2)
    else:
        esc2 = float(np.float32(1e16))
        count, rad, dmag = _iterate(x, y, x, y, torch.ones_like(x), torch.zeros_like(x), 1.0, 1, case["maxiter"], esc2)
    inside = count < 0
    rad = torch.where(inside, torch.full_like(rad, 4.0), rad)
    if case["coloring"] == EDE:
        v = torch.sqrt(rad) * torch.log(rad) / torch.sqrt(dmag) / _toward_zero(dx)
    else:
        v = count.double() - torch.log(torch.log(rad) / 2 / LN2) / LN2
    return {"values": torch.where(inside, torch.full_like(v, -2.0), v), "n": None}
