"""A memory budget that a batch rendered by size just fits: launching it whole
first, on scratch sized by points, refuses nothing that would fit without."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _record(be, rrb_lib, s, pages):
    keep = []
    p = rrb_lib.batch_params(s.pts, s.flags, s.path_pt_off, s.fill_rule, s.gray, s.alpha, s.path_page, s.page_width,
                             s.page_height, s.page_offset, pages, keep=keep)
    be.begin_page()
    be.record_fill_buffer(pages, 255)
    try:
        be.record_path_batch(p)
    finally:
        be.wait_page(be.submit_page())
    got = np.empty(s.arena_bytes, np.uint8)
    be.wait_download(be.download_async(pages, got))
    return got


def _need(rrb_lib, s):
    """Device bytes of a context that has rendered s once, by size."""
    with rrb_lib.B200Backend(0) as be:
        _record(be, rrb_lib, s, be.alloc_device(s.arena_bytes))
        return be.detect_vram_budget().used_bytes


# Curves (three points a piece: bounds three times the sizes) and straight edges; one page and several.
@pytest.mark.parametrize("scene", [dict(kind=1, n_paths=1500, page_w=900, page_h=1100), dict(kind=0, n_paths=700, page_w=600, page_h=700),
                                   dict(kind=2, n_pages=4, page_scale=0.15, paths_scale=0.05)])
@pytest.mark.parametrize("slack", [0, 1 << 20, 8 << 20])
def test_what_fits_by_size_is_rendered(rrb_lib, oracle, scene, slack):
    s = rrb_lib.Scene(seed=17, **scene)
    small = rrb_lib.Scene(kind=1, seed=2, n_paths=20, page_w=200, page_h=150)
    exp = s.blank_arena()
    oracle.render_scene(s, exp, threads=4)
    budget = _need(rrb_lib, s) + small.arena_bytes + (64 << 10) + slack
    with rrb_lib.B200Backend(0, mem_budget=budget) as be:
        pages, pages2 = be.alloc_device(s.arena_bytes), be.alloc_device(small.arena_bytes)
        for _ in range(3):
            _record(be, rrb_lib, small, pages2)
            assert np.array_equal(_record(be, rrb_lib, s, pages), exp)


# Room for all of the bounds, and for all but the last and largest of them.
@pytest.mark.parametrize("rest,want,fits", [(24 << 20, 16 << 20, True), (6 << 20, 4 << 20, False)])
def test_bounds_are_given_back(rrb_lib, rest, want, fits):
    """Memory beside the sizes of a batch can be had although a whole launch has filled it with bounds."""
    s = rrb_lib.Scene(kind=1, seed=18, n_paths=1500, page_w=900, page_h=1100)
    need = _need(rrb_lib, s)
    with rrb_lib.B200Backend(0, mem_budget=need + rest) as be:
        pages = be.alloc_device(s.arena_bytes)
        first = _record(be, rrb_lib, s, pages)
        by_size = be.last_batch_stats()["host_syncs"]
        _record(be, rrb_lib, s, pages)
        assert (be.last_batch_stats()["host_syncs"] < by_size) == fits  # whole
        assert be.detect_vram_budget().used_bytes > need + rest - want
        buf = be.alloc_device(want)
        assert be.detect_vram_budget().used_bytes <= need + rest
        assert np.array_equal(_record(be, rrb_lib, s, pages), first)
        be.free_device(buf)
        assert np.array_equal(_record(be, rrb_lib, s, pages), first)


def test_the_second_overflow_list_is_not_needed_without_overflow_rows(rrb_lib, oracle):
    s = rrb_lib.Scene(kind=1, seed=19, n_paths=3000, page_w=1200, page_h=900)
    exp = s.blank_arena()
    oracle.render_scene(s, exp, threads=4)
    with rrb_lib.B200Backend(0) as be:
        _record(be, rrb_lib, s, be.alloc_device(s.arena_bytes))
        need, st = be.detect_vram_budget().used_bytes, be.last_batch_stats()
    assert st["row_overflows"] == 0
    with rrb_lib.B200Backend(0, mem_budget=need - 8 * st["row_groups"]) as be:  # 10 bytes a row with the headroom
        pages = be.alloc_device(s.arena_bytes)
        for _ in range(2):
            assert np.array_equal(_record(be, rrb_lib, s, pages), exp)
