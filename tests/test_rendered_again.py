"""Batches uploaded per call that are launched whole (their sizes checked behind
the launches) and rendered again by size where one did not fit: that a batch
rendered once fits from then on, whatever its edge count."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _record(be, rrb_lib, s, pages, rgb=None, clip=None):
    keep = []
    p = rrb_lib.batch_params(s.pts, s.flags, s.path_pt_off, s.fill_rule, s.gray, s.alpha, s.path_page, s.page_width,
                             s.page_height, s.page_offset, pages, keep=keep)
    be.begin_page()
    be.record_fill_buffer(pages, 255)
    be.record_path_batch_ex(p, rgb, clip)
    be.wait_page(be.submit_page())
    return be.last_batch_stats()


def _lines(n_edges, w, h):
    """One path of n_edges straight edges around the middle of a page."""

    class S:
        pass

    s, t = S(), np.linspace(0, 2 * np.pi, n_edges + 1)
    r = np.where(np.arange(n_edges + 1) % 2, 0.3, 0.45)
    s.pts = np.stack([w * (0.5 + r * np.cos(t)), h * (0.5 + r * np.sin(t))], 1)
    s.pts[-1] = s.pts[0]
    s.flags = np.array([5] + [0] * (n_edges - 1) + [6], np.uint8)
    s.path_pt_off, s.fill_rule = np.array([0, n_edges + 1], np.uint64), np.zeros(1, np.uint8)
    s.gray, s.alpha, s.path_page = np.array([20], np.uint8), np.array([140], np.uint8), np.zeros(1, np.uint32)
    s.page_width, s.page_height = np.array([w], np.uint32), np.array([h], np.uint32)
    s.page_offset, s.arena_bytes = np.zeros(1, np.uint64), w * h
    return s


# The first bounds buffer holds 32 groups of 32 edges, the last of them spare.
@pytest.mark.parametrize("n", [40, 928, 960, 961, 991, 992, 993, 1100])
def test_the_second_render_is_launched_whole(rrb_lib, oracle, n):
    first, s = _lines(4, 200, 150), _lines(n, 200, 150)
    exp = np.full(s.arena_bytes, 255, np.uint8)
    oracle.render_scene(s, exp)
    with rrb_lib.B200Backend(0) as be:
        pages = be.alloc_device(s.arena_bytes)
        by_size = _record(be, rrb_lib, first, pages)["host_syncs"]  # a context's first render
        _record(be, rrb_lib, s, pages)
        whole = [_record(be, rrb_lib, s, pages)["host_syncs"] for _ in range(3)]
        got = np.empty(s.arena_bytes, np.uint8)
        be.wait_download(be.download_async(pages, got))
        be.free_device(pages)
    assert np.array_equal(got, exp)
    assert max(whole) < by_size  # rendered again: more than by size


class _Paint:
    """A paint batch on one page: (points, stroke or None) per path; closed unless stroked."""

    def __init__(self, rng, paths, w, h):
        n = len(paths)
        self.pts = np.concatenate([p for p, _ in paths])
        self.flags = np.concatenate([np.array(([1] + [0] * (len(p) - 2) + [2]) if st else [5] + [0] * (len(p) - 2) + [6],
                                              np.uint8) for p, st in paths])
        self.path_pt_off = np.cumsum([0] + [len(p) for p, _ in paths]).astype(np.uint64)
        self.strokes = [st for _, st in paths]
        self.fill_rule, self.path_page = np.zeros(n, np.uint8), np.zeros(n, np.uint32)
        self.gray, self.alpha = rng.integers(0, 256, n).astype(np.uint8), rng.integers(60, 200, n).astype(np.uint8)
        self.page_width, self.page_height = np.array([w], np.uint32), np.array([h], np.uint32)
        self.page_offset, self.arena_bytes = np.zeros(1, np.uint64), w * h


def _comb(x0, x1, y0, y1, teeth):
    x = np.linspace(x0, x1, 2 * teeth)
    y = np.where(np.arange(2 * teeth) % 2, y1, y0)
    return np.vstack([np.stack([x, y], 1), [(x1, y1 + 1.5), (x0, y1 + 1.5), (x[0], y[0])]])


def _paint(be, rrb_lib, s, pages, rgb, clip):
    keep = []
    p = rrb_lib.batch_params(s.pts, s.flags, s.path_pt_off, s.fill_rule, s.gray, s.alpha, s.path_page, s.page_width,
                             s.page_height, s.page_offset, pages, keep=keep)
    be.begin_page()
    be.record_fill_buffer(pages, 255)
    be.record_stroke_batch(p, s.strokes, rgb, clip)
    be.wait_page(be.submit_page())
    return be.last_batch_stats()


def _growing(rng):
    """Batches each beyond the buffers of those before in one more count, named by it."""
    w, h = 900, 90
    hair = dict(line_width=0.0)

    def triangle(x, y, a, b):
        return np.array([(x, y), (x + a, y + 1), (x + 2, y + b), (x, y)]), None

    combs = [(_comb(x, x + 55, 2, 86.5, 5), None) for x in rng.uniform(1, 840, 60)]
    lines = [(np.array([(x, 1.5), (x + 3, 88.5)]), hair) for x in rng.uniform(1, 890, 6000)]
    specks = [(np.array([(x, y), (x + 4, y), (x + 4, y + 4), (x, y + 4), (x, y)]), None)
              for x, y in rng.uniform(0, (890, 80), (3000, 2))]  # rectangles: no rows or runs
    ells = [(np.array([(x, y), (x + 30, y), (x + 30, y + 9.3), (x + 11, y + 9.3), (x + 11, y + 20), (x, y + 20), (x, y)]), None)
            for x, y in rng.uniform(0, (860, 65), (300, 2))]
    P = _Paint
    yield "first", P(rng, [triangle(5, 5, 9, 9)], 60, 50)
    yield "edges", P(rng, [(_comb(2, 890, 2, 80, 60), None)], w, 90)
    yield "rows", P(rng, [triangle(5, 5, 200, 1900)], 300, 2000)
    yield "overflow rows", P(rng, [(_comb(2, 890, 2, 86, 300), None)], w, h)
    yield "runs", P(rng, ells, w, h)
    yield "pairs", P(rng, specks, w, h)
    yield "cells", P(rng, combs, w, h)
    yield "hairline runs", P(rng, lines, w, h)
    yield "hairline cells", P(rng, combs + lines, w, h)  # the combs' cells first, then hairlines until none are left


@pytest.mark.parametrize("form", ["gray", "clipped rgb"])
def test_a_batch_that_does_not_fit_is_rendered_again(rrb_lib, oracle, form):
    """Every count in turn: the first record renders twice (and says so in its launches and waits), the second is
    launched whole, and the page is the oracle's after both."""
    rng = np.random.default_rng(3)
    again = set()
    with rrb_lib.B200Backend(0) as be:
        for name, s in _growing(rng):
            rgb = clip = None
            n, w, h = len(s.strokes), int(s.page_width[0]), int(s.page_height[0])
            if form != "gray":
                rgb = rng.integers(0, 256, (n, 3), np.uint8)
                clip = np.tile([3.5, 2.25, w - 8.75, h - 1.5], (n, 1))
            bpp = 1 if rgb is None else 3
            exp = np.full(bpp * s.arena_bytes, 255, np.uint8)
            oracle.render_scene_paint(s, exp, s.strokes, rgb=rgb, clip=clip)
            with rrb_lib.B200Backend(0) as fresh:
                pages = fresh.alloc_device(bpp * s.arena_bytes)
                by_size = _paint(fresh, rrb_lib, s, pages, rgb, clip)
                fresh.free_device(pages)
            pages = be.alloc_device(bpp * s.arena_bytes)
            for k in range(2):
                st = _paint(be, rrb_lib, s, pages, rgb, clip)
                got = np.empty(bpp * s.arena_bytes, np.uint8)
                be.wait_download(be.download_async(pages, got))
                d = np.nonzero(got != exp)[0]
                assert d.size == 0, f"{name}, record {k}: {d.size} bytes differ, first at {d[:5]}"
                if k == 0 and st["kernel_launches"] >= by_size["kernel_launches"] + 10:
                    assert st["host_syncs"] > by_size["host_syncs"]
                    again.add(name)
            assert st["host_syncs"] < by_size["host_syncs"]
            be.free_device(pages)
    assert {"edges", "rows", "overflow rows", "runs", "pairs", "hairline runs", "hairline cells"} <= again
