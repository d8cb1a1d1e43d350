"""GPU parity of the colour stage on the large benchmark frames: normalizeData's whole-frame min/max
(reference src/lyapunov_fractal.hpp:110-125), its map (:127-137) and the page's 3x3 mean + palette + byte store
(web/fractal_renderer.js:283-311,207-281,191-198), against the CPU oracle.  Bar: identical fp64 words and bytes."""
import time

import numpy as np
import pytest

import lyapunovfractalwasm_b200 as L
from conftest import CONFIGS, config5_frame

pytestmark = pytest.mark.gpu


def same_bits(a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    return a.shape == b.shape and np.array_equal(a.view(np.uint64), b.view(np.uint64))


def oracle_rows(port, kw, **rows):
    return port.lambda_rows(kw["min_x"], kw["max_x"], kw["min_y"], kw["max_y"], kw["width"], kw["height"],
                            kw["sequence"], kw["iterations"], kw["warmup"], c=kw.get("c"), **rows)


@pytest.mark.parametrize("k", [0, 33, 255])
def test_config5_frames_whole(engine, port, k):
    """Zoom-batch frames 0 (a third of the pixels escape), 33 (the last frame that still reaches a > 4) and 255, whole:
    lambda, executed steps, min/max, normalised grid and RGBA against the oracle."""
    kw = config5_frame(k)
    r = engine.render(L.make_params(**kw), want=("lambda", "norm", "rgba"))
    lam, steps = oracle_rows(port, kw)
    assert same_bits(r["lambda"], lam) and r["stats"].executed_steps == steps
    assert (r["stats"].lambda_min, r["stats"].lambda_max) == port.minmax(lam)
    norm = port.normalize(lam)
    assert same_bits(r["norm"], norm)
    assert np.array_equal(r["rgba"], port.colorize(norm, 0))


def check_blocks(port, kw, frame_mm, norm, rgba, blocks):
    """Row blocks [y0, y1) of a frame whose normalised grid and RGBA are in `norm` / `rgba`: the oracle renders lambda for
    the block plus one row either side, normalises it with the frame's min/max and colours it; the block's own rows of
    the 3x3 mean see exactly those rows."""
    lo, hi = frame_mm
    H = kw["height"]
    seen_lo, seen_hi = np.inf, -np.inf
    for y0, y1 in blocks:
        a, b = max(0, y0 - 1), min(H, y1 + 1)
        lam, _ = oracle_rows(port, kw, y0=a, y1=b)
        mn, mx = port.minmax(lam)
        seen_lo, seen_hi = min(seen_lo, mn), max(seen_hi, mx)
        want_norm = port.normalize(lam, lo, hi)
        assert same_bits(norm[a:b], want_norm), (y0, y1)
        want_rgba = port.colorize(want_norm, 0)
        # rows whose three neighbour rows are all inside [a, b), or cut by the image edge exactly as in the frame
        first = y0 - a if a > 0 else 0
        last = (y1 - a) if b < H else (b - a)
        assert np.array_equal(rgba[a + first:a + last], want_rgba[first:last]), (y0, y1)
    # the frame's extremes bound every sampled row's (they are equal only if the extreme pixel was sampled)
    assert lo <= seen_lo and hi >= seen_hi


def test_config3_colour_stage_one_device_and_two_bands(engine, port):
    """16384^2, "BBBBBBAAAAAA", 500 + 4000: the whole frame on the device, then sampled row blocks of the normalised grid
    and of the RGBA bytes against the oracle -- first, last, interior, and the rows either side of the band edge of a
    two-band render (lyap_multi_render, both bands on this device), whose bytes must equal the one-device frame's."""
    kw = CONFIGS[3]
    one = engine.render(L.make_params(**kw), want=("norm", "rgba"))
    mm = (one["stats"].lambda_min, one["stats"].lambda_max)
    blocks = [(0, 2), (5000, 5002), (8190, 8194), (16382, 16384)]
    check_blocks(port, kw, mm, one["norm"], one["rgba"], blocks)
    with L.Multi([0, 0]) as m:
        two = m.render(L.make_params(**kw), want=("norm", "rgba"))
    assert (two["stats"].lambda_min, two["stats"].lambda_max) == mm
    assert two["stats"].executed_steps == one["stats"].executed_steps
    assert same_bits(two["norm"], one["norm"])
    assert np.array_equal(two["rgba"], one["rgba"])


def test_fp32_lambda_on_config3_and_config4_bands(engine, port):
    """(float)lambda beside the fp64 value, on bands of the two largest frames."""
    for cfg, y0, y1 in ((3, 12287, 12290), (4, 49151, 49153)):
        kw = CONFIGS[cfg]
        r = engine.render(L.make_params(**kw, row_begin=y0, row_end=y1), want=("lambda", "lambda32"))
        want, steps = oracle_rows(port, kw, y0=y0, y1=y1)
        assert same_bits(r["lambda"], want) and r["stats"].executed_steps == steps
        assert r["lambda32"].dtype == np.float32 and np.array_equal(r["lambda32"], want.astype(np.float32))


def test_config4_colour_stage_on_a_band_with_given_minmax(engine, port):
    """65536-wide rows: the device entry points on a band (normalise with a supplied min/max, colour with neighbour rows
    present above and below) against the oracle on the same rows."""
    kw = CONFIGS[4]
    y0, y1 = 32766, 32770          # straddles the 2-, 4- and 8-band boundary at row 32768
    W = kw["width"]
    rows = y1 - y0
    lam, _ = oracle_rows(port, kw, y0=y0, y1=y1)
    mn, mx = -3.9, 1.0             # any fixed pair: the band path takes the frame's min/max from outside
    d_lam, d_norm = engine.alloc(rows * W * 8), engine.alloc(rows * W * 8)
    d_rgba, d_mm = engine.alloc((rows - 2) * W * 4), engine.alloc(16)
    engine.lambda_device(L.make_params(**kw, row_begin=y0, row_end=y1), d_lam.ptr)
    d_mm.from_host(np.array([mn, mx]))
    engine.normalize_device(d_lam.ptr, rows * W, d_mm.ptr, d_norm.ptr)
    engine.colorize_device(d_norm.ptr + W * 8, W, rows - 2, 1, 1, 0, d_rgba.ptr)
    engine.sync()
    want_norm = port.normalize(lam, mn, mx)
    assert same_bits(d_lam.to_host(np.float64).reshape(rows, W), lam)
    assert same_bits(d_norm.to_host(np.float64).reshape(rows, W), want_norm)
    assert np.array_equal(d_rgba.to_host(np.uint8).reshape(rows - 2, W, 4), port.colorize(want_norm, 0)[1:-1])
    for b in (d_lam, d_norm, d_rgba, d_mm):
        b.free()


# no more than 100: an angle's quadrant is a conversion to int, which CPU and GPU define differently from 2^31 on (the
# angle is at most 6 pi t; infinities and 1e300 gave other bytes than the CPU's before and after)
SPECIAL = [0.0, -0.0, 1.0, 0.5, 1e-310, 2.0 ** -301, 2.0 ** -300, 1.0 + 2.0 ** -52, 3.0, -0.25, 100.0, np.nan]


@pytest.mark.parametrize("shape", [(1, 5), (2, 4), (3, 6), (9, 7), (255, 9), (256, 4), (257, 5), (258, 12), (513, 6),
                                   (1, 2049), (2, 1030), (3, 700), (7, 297), (32, 65), (33, 57), (127, 22), (128, 18), (129, 13)])
def test_colour_kernel_edges_and_special_values(engine, port, shape):
    """Every palette at widths around a block's 256 columns, heights around a strip's 4 rows and, in narrow frames, around
    the strips of a block; half of the frames carry
    values a picture has none of, which take the general palette code: bytes equal the oracle's."""
    w, h = shape
    rng = np.random.default_rng(w * 100 + h)
    for special in (False, True):
        norm = rng.uniform(0.0, 1.0, size=(h, w))
        if special:
            at = rng.integers(0, h * w, size=max(1, h * w // 40))
            norm.flat[at] = rng.choice(SPECIAL, size=at.size)
        for palette in range(7):
            assert np.array_equal(engine.colorize(norm, palette), port.colorize(norm, palette)), (special, palette)


@pytest.mark.parametrize("n", [1, 2, 3, 31, 511, 512, 513, 303105])
def test_normalise_edges_and_special_values(engine, port, n):
    """Lengths around a block's round of pairs, values that are sentinels, special or the frame's own extremes."""
    rng = np.random.default_rng(n)
    for special in (False, True):
        values = rng.uniform(-3.0, 1.2, size=n)
        if special:
            at = rng.integers(0, n, size=max(1, n // 5))
            values[at] = rng.choice([-5.0, -4.0, -3.9999999, np.nan, np.inf, -np.inf, 0.0, 1e-310, -3.0, 1.2], size=at.size)
        assert same_bits(engine.normalize_data(values), port.normalize(values)), special


def test_minmax_of_an_unaligned_array_takes_no_longer(engine):
    """2^24 values from an address that is no multiple of 16 bytes against an aligned one: 1.8 times the time when their loop had
    one load in flight and its blocks did not all fit, 1.0 so."""
    n = 1 << 24
    d_v, d_mm = engine.alloc(8 * (n + 1)), engine.alloc(16)
    d_v.from_host(np.random.default_rng(2).uniform(-3.0, 1.2, n + 1))
    best = {}
    for offset in (0, 8):
        for _ in range(5):
            engine.sync()
            t0 = time.perf_counter()
            for _ in range(10):
                engine.minmax_device(d_v.ptr + offset, n, d_mm.ptr)
            engine.sync()
            best[offset] = min(best.get(offset, 1.0), time.perf_counter() - t0)
    assert best[8] < 1.4 * best[0]
    d_v.free()
    d_mm.free()


def test_normalise_of_a_flat_frame_takes_no_longer(engine, port):
    """Eight million values, all but the last 20 the minimum, against as many ordinary ones: 1.3 times the time when a warp of
    them went the common way and then put each right, 0.6 so.  Same bits as the oracle at the seam."""
    n = 1 << 23
    d_v, d_out, d_mm = engine.alloc(8 * n), engine.alloc(8 * n), engine.alloc(16)
    flat = np.full(n, 0.25)
    flat[-20:] = np.linspace(0.3, 0.5, 20)
    best = {}
    for name, values in (("ordinary", np.random.default_rng(1).uniform(-3.0, 1.2, n)), ("flat", flat)):
        d_v.from_host(values)
        engine.minmax_device(d_v.ptr, n, d_mm.ptr)
        for _ in range(5):
            engine.sync()
            t0 = time.perf_counter()
            for _ in range(10):
                engine.normalize_device(d_v.ptr, n, d_mm.ptr, d_out.ptr)
            engine.sync()
            best[name] = min(best.get(name, 1.0), time.perf_counter() - t0)
    assert same_bits(d_out.to_host(np.float64, 100, 8 * (n - 100)), port.normalize(flat)[-100:])
    assert best["flat"] < best["ordinary"]
    for b in (d_v, d_out, d_mm):
        b.free()


@pytest.mark.parametrize("n", [2, 3, 4, 5, 64, 4097, 700001])
def test_minmax_of_zeros_does_not_depend_on_their_order(engine, n):
    """Where the extreme is zero, the minimum is -0 and the maximum +0 if there is one, wherever it stands and however the
    array is aligned (a thread's loads, its block and the last block each choose between two)."""
    d_v, d_mm = engine.alloc(8 * (n + 1)), engine.alloc(16)
    rng = np.random.default_rng(n)
    for flip in (1.0, -1.0):
        for offset in (0, 8):
            for fill in (-1.0, 0.0, 1.0):
                values = rng.permutation(np.where(np.arange(n) < max(2, n // 2), 0.0, fill))
                at = np.flatnonzero(values == 0.0)
                values[at] = flip * 0.0
                values[rng.choice(at)] = -flip * 0.0
                d_v.from_host(values, offset)
                engine.minmax_device(d_v.ptr + offset, n, d_mm.ptr)
                lo, hi = d_mm.to_host(np.float64)
                assert lo == values.min() and hi == values.max()
                assert lo != 0.0 or np.signbit(lo), (flip, offset, fill)
                assert hi != 0.0 or not np.signbit(hi), (flip, offset, fill)
    d_v.free()
    d_mm.free()
