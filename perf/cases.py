"""The work that a user of the fill backend has it do, as cases to be timed.

Every case goes through the Python mirror of the C ABI (rrb) the way a page
renderer calls it: begin_page, the page set to white, one or more record_*
calls, submit_page, wait_page (or the one-call host form), with the seeded
page generators of the package as inputs. What comes back are the pages (or
coverage buffers) themselves: bytes, and the same bytes on every pass, so
there is no rounding to be judged and exact() has no value to give.

listed() has the cases; draw(rng) gives more of the same ranges.
"""

import math
import random
import statistics
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path("pdf-raster_b200").resolve()))

import rrb  # noqa: E402
from rrb.strokes import StrokePage  # noqa: E402

WHITE = 255


def listed():
    return [
        # The per-path form of the boundary (raster::fill replaced call by
        # call): one glyph onto a 150 dpi page. All latency and launches.
        dict(name="one_glyph", call="path_fill", scene="glyphs", paths=1, w=1240, h=1754, as_shipped=False),
        # A light page handed over whole from ordinary host arrays: a logo or a
        # small diagram on a screen-sized page.
        dict(name="small_page", call="batch", scene="polygons", paths=40, w=612, h=792, as_shipped=False),
        # An ordinary text page at 300 dpi from ordinary host arrays.
        dict(name="text_page", call="batch", scene="glyphs", paths=4000, w=2480, h=3508, as_shipped=False),
        # The polygon page of the benchmark, kept on the device and re-rendered.
        dict(name="polygon_page", call="resident", scene="polygons", paths=2000, w=2550, h=3300, as_shipped=False),
        # The glyph-dense page of the benchmark, kept on the device.
        dict(name="glyph_page", call="resident", scene="glyphs", paths=150000, w=2550, h=3300, as_shipped=False),
        # Uneven pages of glyphs, polygons and rectangles in one submission, a
        # good quarter of the benchmark's batch: the largest case.
        dict(name="mixed_batch", call="resident_mixed", pages=18, page_scale=1.0, paths_scale=1.0, as_shipped=False),
        # The same kind of pages from page-locked host memory and back to it, in
        # one call: what a serving process pays end to end.
        dict(name="mixed_host", call="host_mixed", pages=9, page_scale=1.0, paths_scale=1.0, as_shipped=False),
        # Colour pages of translucent shapes under clip rectangles, then the
        # luma page made from them: the renderer's RGB output.
        dict(name="colour_page", call="rgb_clip", scene="polygons", paths=900, w=1275, h=1651, as_shipped=False),
        # A page of rules, boxes, charts and dashes: strokes and fills in paint
        # order, outlines built by the call.
        dict(name="stroke_page", call="strokes", paths=1500, w=1700, h=2200, as_shipped=False),
        # The coverage operator with 64 samples a pixel, on a window of glyph
        # outlines already flattened and on the device.
        dict(name="aa_fill_glyphs", call="aa_fill", outlines=48, w=1024, h=1024, even_odd=False),
        # The same operator on a large window with few outlines, even-odd.
        dict(name="aa_fill_large", call="aa_fill", outlines=6, w=2047, h=2050, even_odd=True),
        # The analytic coverage operator from segments, records built on the way.
        dict(name="tile_fill_glyphs", call="tile_fill", outlines=48, w=1024, h=1024, even_odd=False),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    call = rng.choice(["path_fill", "batch", "batch", "resident", "resident", "resident_mixed", "host_mixed",
                       "rgb_clip", "strokes", "aa_fill", "aa_fill", "tile_fill"])
    w = _log(rng, 300, 3600)
    h = int(w * rng.uniform(0.7, 1.5))
    scene = rng.choice(["glyphs", "polygons"])
    if call == "path_fill":
        return dict(call=call, scene=scene, paths=1, w=w, h=h, as_shipped=False)
    if call == "batch":
        n = _log(rng, 2, 6000 if scene == "glyphs" else 1500)
        # The row map as shipped draws what lies near the top of a page.
        return dict(call=call, scene=scene, paths=n, w=w, h=h,
                    as_shipped=scene == "polygons" and n >= 200 and rng.random() < 0.5)
    if call == "resident":
        return dict(call=call, scene=scene, paths=_log(rng, 200, 150000 if scene == "glyphs" else 3000), w=w, h=h,
                    as_shipped=False)
    if call in ("resident_mixed", "host_mixed"):
        return dict(call=call, pages=rng.randint(1, 16 if call == "resident_mixed" else 9),
                    page_scale=round(rng.uniform(0.3, 1.0), 3), paths_scale=round(rng.uniform(0.05, 0.8), 3),
                    as_shipped=False)
    if call == "rgb_clip":
        return dict(call=call, scene=scene, paths=_log(rng, 20, 2500), w=w, h=h, as_shipped=False)
    if call == "strokes":
        return dict(call=call, paths=_log(rng, 20, 2000), w=max(w, 700), h=max(h, 500), as_shipped=False)
    side = _log(rng, 17, 2100)
    return dict(call=call, outlines=_log(rng, 1, 64), w=side, h=max(1, int(side * rng.uniform(0.5, 1.0))),
                even_odd=rng.random() < 0.5)


# One backend for what is uploaded call by call and one for what stays on the
# device, as two parts of a program hold them; made at first use and kept.
_backends = {}


def _backend(use):
    if use not in _backends:
        _backends[use] = rrb.B200Backend(0)
    return _backends[use]


class _Buffer:
    """Device memory of a backend, given back when nothing refers to it any more."""

    def __init__(self, be, size):
        self.be, self.buf = be, be.alloc_device(max(16, int(size)))

    def __del__(self):
        self.be.free_device(self.buf)

    def tensor(self, *shape):
        """The same memory for torch, not a copy; the tensor keeps the buffer."""
        return torch.as_tensor(_DeviceBytes(self, shape), device="cuda")


class _DeviceBytes:
    def __init__(self, owner, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "|u1", "data": (owner.buf.ptr, False), "version": 3}


class State:
    """Inputs, buffers and handles of one case."""

    def __init__(self, use):
        self.be = _backend(use)
        self.keep, self.batch = [], None

    def buffer(self, size):
        b = _Buffer(self.be, size)
        self.keep.append(b)
        return b

    def __del__(self):
        if self.batch is not None:
            self.batch.free()


def _page_locked(a):
    """A copy of a host array in page-locked memory."""
    v = torch.empty(max(1, a.nbytes), dtype=torch.uint8, pin_memory=True).numpy()[: a.nbytes].view(a.dtype)
    v[:] = a.reshape(-1)
    return v


# A4, Letter and A3 at 150, 300 and 600 dpi: the mixed pages' sizes at scale 1.
_SIZES = ((1240, 1754), (2480, 3508), (4961, 7016), (1275, 1650), (2550, 3300), (5100, 6600), (1754, 2480),
          (3508, 4961), (7016, 9921))


def _mixed_pages(case):
    """(width, height, paths) of each page: the nine sizes in turn, and the paths at evenly spaced quantiles of the
    generator's log-normal count (median 5,000, sigma 1.2, at most 50,000), in a fixed order."""
    n, scale = case["pages"], case["page_scale"]
    z = [statistics.NormalDist().inv_cdf((k + 0.5) / n) for k in range(n)]
    random.Random(n).shuffle(z)
    return [(max(16, round(_SIZES[k % 9][0] * scale)), max(16, round(_SIZES[k % 9][1] * scale)),
             max(1, min(50000, round(5000 * case["paths_scale"] * math.exp(1.2 * z[k]))))) for k in range(n)]


class _Mixed:
    """Mixed pages of the package's generator, one batch: every seed gives the same page sizes and path counts."""

    def __init__(self, case, seed):
        rng = random.Random(seed)
        parts = []
        for w, h, n in _mixed_pages(case):
            while True:  # the page size is the generator's first choice: a seed that takes this one
                sd = rng.getrandbits(48)
                probe = rrb.Scene(kind=2, seed=sd, n_pages=1, page_scale=case["page_scale"], path_cap=1)
                if abs(int(probe.page_width[0]) - w) <= 1 and abs(int(probe.page_height[0]) - h) <= 1:
                    break
            # A median far above the cap: the count is the cap.
            parts.append(rrb.Scene(kind=2, seed=sd, n_pages=1, page_scale=case["page_scale"], paths_scale=1e12,
                                   path_cap=n))
        cat = np.concatenate
        self.pts, self.flags = cat([s.pts for s in parts]), cat([s.flags for s in parts])
        ends = np.cumsum([s.n_pts for s in parts]) - [s.n_pts for s in parts]
        self.path_pt_off = cat([np.zeros(1, np.uint64)] +
                               [s.path_pt_off[1:] + np.uint64(e) for s, e in zip(parts, ends)])
        self.fill_rule, self.gray = cat([s.fill_rule for s in parts]), cat([s.gray for s in parts])
        self.alpha = cat([s.alpha for s in parts])
        self.path_page = cat([np.full(s.n_paths, k, np.uint32) for k, s in enumerate(parts)])
        self.page_width, self.page_height = cat([s.page_width for s in parts]), cat([s.page_height for s in parts])
        sizes = [(int(s.arena_bytes) + 255) // 256 * 256 for s in parts]
        self.page_offset = np.cumsum(sizes) - sizes
        self.arena_bytes, self.n_pages = int(sum(sizes)), len(parts)


def _scene(case, seed):
    if "pages" in case:
        return _Mixed(case, seed)
    return rrb.Scene(kind=1 if case["scene"] == "glyphs" else 0, seed=seed, n_paths=case["paths"], page_w=case["w"],
                     page_h=case["h"])


def _params(st, s, pages, case, copy=np.array):
    return rrb.batch_params(copy(s.pts.reshape(-1)), copy(s.flags), np.array(s.path_pt_off), np.array(s.fill_rule),
                            np.array(s.gray), np.array(s.alpha), np.array(s.path_page), np.array(s.page_width),
                            np.array(s.page_height), np.array(s.page_offset), pages, rowmap=int(case["as_shipped"]),
                            keep=st.keep)


def _outline_segments(case, seed):
    """Flattened glyph outlines spread over the window: f32 [n, 4], as a caller's own flattener leaves them."""
    w, h, n = case["w"], case["h"], case["outlines"]
    s = rrb.Scene(kind=1, seed=seed, n_paths=n, page_w=w, page_h=h)
    rng = np.random.default_rng(seed)
    cols = max(1, int(math.ceil(math.sqrt(n * w / h))))
    rows = max(1, -(-n // cols))
    t = np.linspace(0.0, 1.0, 5)[:, None]
    segs = []
    for i in range(n):
        a, b = int(s.path_pt_off[i]), int(s.path_pt_off[i + 1])
        p, f = s.pts[a:b], s.flags[a:b]
        lo, hi = p.min(0), p.max(0)
        cell = np.array([w / cols, h / rows])
        p = (p - lo) * (cell * rng.uniform(0.8, 1.1) / (hi - lo)) + np.array([i % cols, i // cols]) * cell
        k = 0
        while k < len(f):
            if f[k] & 1:
                k += 1
            elif f[k] & 8:  # a cubic from the point before
                c = [p[k - 1], p[k], p[k + 1], p[k + 2]]
                q = ((1 - t) ** 3 * c[0] + 3 * t * (1 - t) ** 2 * c[1] + 3 * t * t * (1 - t) * c[2] + t ** 3 * c[3])
                segs.append(np.concatenate([q[:-1], q[1:]], 1))
                k += 3
            else:
                segs.append(np.concatenate([p[k - 1], p[k]])[None])
                k += 1
    return np.ascontiguousarray(np.concatenate(segs), np.float32)


def prepare(case, seed):
    call = case["call"]
    if call in ("aa_fill", "tile_fill"):
        st = State("calls")
        segs = _outline_segments(case, seed)
        sb, cov = st.buffer(segs.nbytes), st.buffer(case["w"] * case["h"])
        st.be.wait_transfer(st.be.upload_async(sb.buf, segs.view(np.uint8).reshape(-1)))
        st.args = (sb.buf, len(segs), cov.buf, case["w"], case["h"], int(case["even_odd"]))
        st.out = cov.tensor(case["h"], case["w"])
        st.go = _go_aa_fill if call == "aa_fill" else _go_tile_fill
        return st
    st = State("resident" if call.startswith("resident") else "calls")
    s = st.scene = (StrokePage(seed=seed, n_paths=case["paths"], w=case["w"], h=case["h"]) if call == "strokes"
                    else _scene(case, seed))
    if call == "rgb_clip":
        # Colour pages of 3 bytes a pixel, translucent paint, and per path a
        # rectangle around a part of the page.
        rng = np.random.default_rng(seed)
        w, h, n = case["w"], case["h"], s.n_paths
        st.rgb = rng.integers(0, 256, (n, 3), np.uint8)
        x, y = rng.uniform(0, 0.5, n) * w, rng.uniform(0, 0.5, n) * h
        st.clip = np.stack([x, y, x + rng.uniform(0.2, 0.6, n) * w, y + rng.uniform(0.2, 0.6, n) * h], 1)
        s.alpha = rng.integers(64, 256, n).astype(np.uint8)
        pages, gray = st.buffer(3 * w * h), st.buffer(w * h)
        st.pages, st.gray, st.pixels = pages.buf, gray.buf, w * h
        st.params = _params(st, s, st.pages, case)
        st.out = (pages.tensor(h, w, 3), gray.tensor(h, w))
        st.go = _go_rgb
        return st
    pages = st.buffer(s.arena_bytes)
    st.pages = pages.buf
    if call == "host_mixed":
        st.params = _params(st, s, st.pages, case, copy=_page_locked)
        st.host = _page_locked(np.zeros(s.arena_bytes, np.uint8))
        st.out, st.go = st.host, _go_host
        return st
    st.out = pages.tensor(s.arena_bytes) if s.n_pages > 1 else pages.tensor(int(s.page_height[0]), int(s.page_width[0]))
    if call.startswith("resident"):
        params = _params(st, s, None, case)
        st.batch = st.be.batch_upload(params)
        st.rowmap = int(case["as_shipped"])
        st.go = _go_resident
        for _ in range(24):  # a batch that is kept is tuned by its first renders
            _go_resident(st)
            if st.be.last_batch_stats()["trials_left"] == 0:
                break
    elif call == "strokes":
        st.params = _params(st, s, st.pages, case)
        st.strokes = rrb.stroke_params(s.strokes, st.keep)
        st.go = _go_strokes
    elif call == "path_fill":
        st.path = (np.array(s.pts), np.array(s.flags), st.pages, case["w"], case["h"])
        st.opts = dict(fill_rule=int(s.fill_rule[0]), gray=int(s.gray[0]), alpha=int(s.alpha[0]),
                       rowmap=int(case["as_shipped"]))
        st.go = _go_path_fill
    else:
        st.params = _params(st, s, st.pages, case)
        st.go = _go_batch
    return st


def _go_path_fill(st):
    st.be.begin_page()
    st.be.record_fill_buffer(st.pages, WHITE)
    st.be.record_path_fill(*st.path, **st.opts)
    st.be.wait_page(st.be.submit_page())


def _go_batch(st):
    st.be.begin_page()
    st.be.record_fill_buffer(st.pages, WHITE)
    st.be.record_path_batch(st.params)
    st.be.wait_page(st.be.submit_page())


def _go_resident(st):
    st.be.begin_page()
    st.be.record_fill_buffer(st.pages, WHITE)
    st.batch.record(st.pages, st.rowmap)
    st.be.wait_page(st.be.submit_page())


def _go_host(st):
    st.be.render_pages_host(st.params, st.host, init=WHITE)


def _go_rgb(st):
    st.be.begin_page()
    st.be.record_fill_buffer(st.pages, WHITE)
    st.be.record_path_batch_ex(st.params, st.rgb, st.clip)
    st.be.record_rgb_to_gray(st.pages, st.gray, st.pixels)
    st.be.wait_page(st.be.submit_page())


def _go_strokes(st):
    st.be.begin_page()
    st.be.record_fill_buffer(st.pages, WHITE)
    st.be.record_stroke_batch(st.params, st.strokes)
    st.be.wait_page(st.be.submit_page())


def _go_aa_fill(st):
    st.be.begin_page()
    st.be.record_aa_fill(*st.args)
    st.be.wait_page(st.be.submit_page())


def _go_tile_fill(st):
    st.be.begin_page()
    st.be.record_tile_fill_segs(*st.args)
    st.be.wait_page(st.be.submit_page())


def run(state):
    state.go(state)
    return state.out


def exact(case, seed):
    """Pages and coverage are bytes that are the same on every pass: nothing here has a value in 64 bits."""
    return None


# Points of a path of each kind (the generators' averages): a polygon has two
# contours of 18 segments, half of them cubics, a glyph two of 36 cubics, a
# rectangle five points; a mixed page is 30% glyphs, 40% polygons, 30%
# rectangles.
_POINTS = {"glyphs": 217.0, "polygons": 76.0}
_MIXED_POINTS = 97.0
_PATH_BYTES = 15  # offset, rule, gray, alpha and page of a path


def work(case):
    """Every input read once (16 bytes a point and its flag, a path's words), every page written once."""
    call = case["call"]
    if call in ("aa_fill", "tile_fill"):
        segs = case["outlines"] * (_POINTS["glyphs"] / 3) * 4
        return {"bytes": 16 * segs + case["w"] * case["h"], "flops": 0}
    if "pages" in case:
        pages = _mixed_pages(case)
        paths, pixels = sum(n for _, _, n in pages), sum(w * h for w, h, _ in pages)
        return {"bytes": paths * (17 * _MIXED_POINTS + _PATH_BYTES) + pixels, "flops": 0}
    pixels = case["w"] * case["h"]
    if call == "strokes":
        return {"bytes": case["paths"] * (17 * 5 + _PATH_BYTES + 48) + pixels, "flops": 0}
    per_path = 17 * _POINTS[case["scene"]] + _PATH_BYTES
    if call == "rgb_clip":
        return {"bytes": case["paths"] * (per_path + 35) + 4 * pixels, "flops": 0}
    return {"bytes": case["paths"] * per_path + pixels, "flops": 0}
