"""The calls whose speed matters to a user of this engine, over the sizes and options they are made with.

Every case goes through the package's public entry points, in one of the ways programs use them:

  frame     the device path: lambda_device, minmax_device, normalize_device, colorize_device into buffers that stay on the GPU
  render    one blocking Engine.render, outputs in fresh host arrays (the web page's call: parameters in, pixels out)
  drop_in   compute_fractal and then normalize_data, both on host arrays (the call order of a program written for the
            reference's C++ header)
  zoom      a batch of frames through a kept Multi object, RGBA to page-locked host memory
  recolour  a kept lambda frame normalised and coloured again (another palette, no new orbits)
  glow      the glow pass on a host frame

A case names a parameter window; the seed cuts up to 1 % off each of its sides, so inputs of different seeds are
different frames of the same kind.
"""
import random

import numpy as np
import torch

import lyapunovfractalwasm_b200 as L

MODES = {"exact": L.MODE_EXACT, "fp64": L.MODE_FAST_FP64, "fp32": L.MODE_FAST_FP32, "orbit64": L.MODE_FAST_FP64_ORBIT}
# windows of the reference's page and of the benchmark frames: (min_x, max_x, min_y, max_y)
WINDOWS = {"page": (0.0, 4.0, 0.0, 4.0), "upper": (2.0, 4.0, 2.0, 4.0), "dense": (2.5, 4.0, 2.5, 4.0),
           "zircon": (3.4, 4.0, 2.5, 3.4)}
LETTERS_37 = "ABBABAABBBABAABABBBAABABAABBBABBAAABA"


def _case(name, kind, width, height, window, sequence, warmup, iterations, mode="exact", palette="cosmic", frames=0):
    return dict(name=name, kind=kind, width=width, height=height, window=window, sequence=sequence, warmup=warmup,
                iterations=iterations, mode=mode, palette=palette, frames=frames)


def listed():
    return [
        # a thumbnail for a parameter picker: the smallest call, latency and launches count
        _case("thumbnail 160x120", "render", 160, 120, "upper", "AB", 100, 1000),
        # the page's production call: 800 x 800 over [0,4]^2, orbits that leave the interval included
        _case("page 800x800", "render", 800, 800, "page", "AB", 100, 1000),
        # the reference struct's default parameters through the drop-in header's two calls
        _case("defaults 800x600", "drop_in", 800, 600, "page", "ABABABAB", 100, 10000),
        # the CPU-sized benchmark frame, on the device
        _case("frame 512x512", "frame", 512, 512, "upper", "AB", 100, 1000),
        # the headline benchmark frame, exact
        _case("frame 4096x4096", "frame", 4096, 4096, "dense", "AABAB", 200, 2000),
        # its fp32 preview
        _case("frame 4096x4096 fp32", "frame", 4096, 4096, "dense", "AABAB", 200, 2000, mode="fp32"),
        # a fast fp64 frame of odd size
        _case("frame 2731x1537 fp64", "frame", 2731, 1537, "upper", "ABB", 150, 1500, mode="fp64", palette="nebula"),
        # the 16384^2 frame with its six-and-six sequence: the largest
        _case("frame 16384x16384", "frame", 16384, 16384, "zircon", "BBBBBBAAAAAA", 500, 4000),
        # a zoom video: 1080p frames with a third parameter
        _case("zoom 1920x1080 x8", "zoom", 1920, 1080, "zoom", "ABC", 300, 3000, frames=8),
        # a sequence without a short period, on a ragged frame
        _case("37 letters 1277x719", "frame", 1277, 719, "dense", LETTERS_37, 100, 1000, palette="psychedelic"),
        # another palette on a kept frame
        _case("recolour 3840x2160", "recolour", 3840, 2160, "dense", "AABAB", 50, 250, palette="aurora"),
        # the glow pass on a finished 1080p picture
        _case("glow 1920x1080", "glow", 1920, 1080, "upper", "AB", 50, 250),
    ]


def _between(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "render", "render", "drop_in", "zoom", "recolour", "glow"])
    most = {"frame": 8192, "render": 2000, "drop_in": 2000, "zoom": 1920, "recolour": 8192, "glow": 3840}[kind]
    width = _between(rng, 128, most)
    height = max(96, min(most, int(width * rng.uniform(0.5, 1.3))))
    sequence = rng.choice(["AB", "AABAB", "BBBBBBAAAAAA", "ABB", LETTERS_37,
                           "AB" + "".join(rng.choice("AB") for _ in range(rng.randint(1, 9)))])
    iterations = _between(rng, 200, 5000)
    while width * height * iterations > 100_000_000_000:
        iterations = iterations * 2 // 3
    mode = rng.choice(["exact", "exact", "exact", "fp64", "fp32", "orbit64"]) if kind in ("frame", "render") else "exact"
    window = rng.choice(["page", "upper", "dense", "zircon"])
    frames = 0
    if kind == "zoom":
        sequence, window, frames = "ABC", "zoom", rng.randint(3, 12)
    if kind in ("recolour", "glow"):
        sequence, iterations = "AB", 250
    return {k: v for k, v in _case("", kind, width, height, window, sequence, iterations // 10, iterations, mode,
                                   rng.choice(L.PALETTES), frames).items() if k != "name"}


_kept = {}


def _engine():
    """The program's one engine, on a stream of its own that torch knows too."""
    if "engine" not in _kept:
        _kept["stream"] = torch.cuda.Stream()
        _kept["engine"] = L.Engine(0)
        _kept["engine"].set_stream(_kept["stream"].cuda_stream)
    return _kept["engine"]


def _multi():
    if "multi" not in _kept:
        _kept["multi"] = L.Multi([0])
    return _kept["multi"]


def _params(case, rng):
    x0, x1, y0, y1 = WINDOWS[case["window"]]
    cut = [rng.uniform(0.0, 0.01) for _ in range(4)]
    return L.make_params(min_x=x0 + cut[0] * (x1 - x0), max_x=x1 - cut[1] * (x1 - x0), min_y=y0 + cut[2] * (y1 - y0),
                         max_y=y1 - cut[3] * (y1 - y0), width=case["width"], height=case["height"],
                         sequence=case["sequence"], iterations=case["iterations"], warmup=case["warmup"],
                         mode=MODES[case["mode"]], palette=case["palette"])


def _zoom_params(case, rng):
    """Frames from all along the zoom of the benchmark batch: centre (3.82, 3.45), half-width 0.5 * 0.97^k, c = 3.7."""
    out = []
    for i in range(case["frames"]):
        half = 0.5 * 0.97 ** (256.0 * i / case["frames"] + rng.uniform(0.0, 1.0))
        out.append(L.make_params(min_x=3.82 - half, max_x=3.82 + half, min_y=3.45 - half, max_y=3.45 + half,
                                 width=case["width"], height=case["height"], sequence=case["sequence"],
                                 iterations=case["iterations"], warmup=case["warmup"], c=3.7, palette=case["palette"]))
    return out


def prepare(case, seed):
    rng = random.Random(seed)
    eng = _engine()
    kind, n = case["kind"], case["width"] * case["height"]
    state = dict(kind=kind, engine=eng, width=case["width"], height=case["height"], mode=case["mode"],
                 palette=L.PALETTES.index(case["palette"]))
    if kind == "zoom":
        state["multi"] = _multi()
        state["params"] = _zoom_params(case, rng)
        state["rgba"] = [torch.empty((case["height"], case["width"], 4), dtype=torch.uint8, pin_memory=True)
                         for _ in state["params"]]
        return state
    state["params"] = _params(case, rng)
    if kind == "glow":
        state["picture"] = eng.render(state["params"], want=("rgba",))["rgba"]
    if kind in ("frame", "recolour"):
        state["lambda"] = torch.empty(n, dtype=torch.float64, device="cuda")
        state["minmax"] = torch.empty(2, dtype=torch.float64, device="cuda")
        state["norm"] = torch.empty(n, dtype=torch.float64, device="cuda")
        state["rgba"] = torch.empty(4 * n, dtype=torch.uint8, device="cuda")
    if kind == "frame":
        state["lambda32"] = torch.empty(n, dtype=torch.float32, device="cuda")
    if kind == "recolour":
        eng.lambda_device(state["params"], d_lambda=state["lambda"].data_ptr())
        eng.sync()
    return state


def run(state):
    eng, kind = state["engine"], state["kind"]
    if kind == "render":
        out = eng.render(state["params"], want=("norm", "rgba"))
        return out["norm"], out["rgba"], out["stats"].executed_steps
    if kind == "drop_in":
        lam = eng.compute_fractal(state["params"])
        return lam, eng.normalize_data(lam)
    if kind == "zoom":
        stats = state["multi"].render_frames(state["params"], None, [t.data_ptr() for t in state["rgba"]])
        return state["rgba"], [s.executed_steps for s in stats]
    if kind == "glow":
        return eng.glow(state["picture"])
    n = state["width"] * state["height"]
    lam, mm, norm, rgba = (state[k].data_ptr() for k in ("lambda", "minmax", "norm", "rgba"))
    if kind == "frame":
        eng.lambda_device(state["params"], d_lambda=lam, d_lambda32=state["lambda32"].data_ptr())
    eng.minmax_device(lam, n, mm)
    eng.normalize_device(lam, n, mm, norm)
    eng.colorize_device(norm, state["width"], state["height"], 0, 0, state["palette"], rgba)
    if kind == "frame":
        return state["lambda"], state["lambda32"], state["minmax"], state["norm"], state["rgba"]
    return state["minmax"], state["norm"], state["rgba"]


def work(case):
    """Flops of the orbits walked step by step (fma = 2): a warm-up step is 3; an accumulated step 19 with its logarithm
    (exact), 6 with the derivative in a running product (fast).  An orbit that leaves (0,1) or comes back to an earlier
    value needs fewer; it is counted in full.  About 100 a pixel for the colour stage (pow, exp, sin, cos)."""
    n = case["width"] * case["height"]
    per_step = 19 if case["mode"] == "exact" else 6
    orbits = n * (3 * case["warmup"] + per_step * case["iterations"])
    kind = case["kind"]
    if kind == "frame":
        return {"bytes": n * (8 + 4 + 8 + 4), "flops": orbits + 100 * n}
    if kind == "render":
        return {"bytes": n * (8 + 4), "flops": orbits + 100 * n}
    if kind == "drop_in":
        return {"bytes": n * (8 + 8 + 8), "flops": orbits + 60 * n}
    if kind == "zoom":
        return {"bytes": case["frames"] * n * 4, "flops": case["frames"] * (orbits + 100 * n)}
    if kind == "recolour":
        return {"bytes": n * (8 + 8 + 4), "flops": 100 * n}
    # glow: two blurs (37 and 13 taps, rows and columns) of three channels and three blends
    return {"bytes": n * (4 + 4), "flops": n * 3 * (2 * 2 * (37 + 13) + 3 * 6)}


def tolerance(case):
    """Exact mode and the colour stage promise their bits.  A fast mode promises the orbit's bits and accumulates in its
    own order: against the same orbit's logarithms summed in extended precision, 20 000 pixels differ by at most 1.2e-16
    (fp64; largest 1.8e-15) and 3.3e-9 (fp32; largest 1.2e-7; rounding to float adds 3e-8) of the frame's rms.  A byte
    whose value sits on a step of the palette may go either way."""
    if case["mode"] == "exact":
        return "exact"
    if case["mode"] == "fp32":
        return {"rel": 1e-7, "max": 5e-7, "differ": 1e-4}
    return {"rel": 1e-14, "max": 1e-13, "differ": 1e-4}
