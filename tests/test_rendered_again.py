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
