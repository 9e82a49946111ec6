"""Binning by blocks of 256 paths, or of 2,048 where a batch would have more
than 2^24 (supertile, block) items: what a batch is refused for, and pages at
both block sizes and at the edges of a block."""

import ctypes as C

import numpy as np
import pytest


def _triangles(n, w, h, seed):
    """n one-triangle paths of a few pixels over a w x h page."""
    rng = np.random.default_rng(seed)
    at = rng.random((n, 2)) * (w - 6, h - 6)
    pts = np.empty((n, 4, 2))
    pts[:, 0], pts[:, 1], pts[:, 2] = at, at + (5.2, 1.1), at + (1.7, 4.9)
    pts[:, 3] = pts[:, 0]
    return _batch(pts.reshape(-1, 2), np.tile(np.array([5, 0, 0, 6], np.uint8), n), np.arange(n + 1, dtype=np.uint64) * 4,
                  w, h, rng)


def _batch(pts, flags, off, w, h, rng):
    class S:
        pass

    s, n = S(), len(off) - 1
    s.pts, s.flags, s.path_pt_off = np.ascontiguousarray(pts, np.float64), flags, off
    s.fill_rule, s.path_page = np.zeros(n, np.uint8), np.zeros(n, np.uint32)
    s.gray, s.alpha = rng.integers(0, 256, n).astype(np.uint8), rng.integers(90, 201, n).astype(np.uint8)
    s.page_width, s.page_height = np.array([w], np.uint32), np.array([h], np.uint32)
    s.page_offset, s.arena_bytes = np.zeros(1, np.uint64), w * h
    return s


# 2^20 supertiles in a column. 262,144 paths: 2^30 items at blocks of 256, 2^27 of
# 2,048 (beyond 524,287 paths blocks of 256 alone would be refused); 2^22 paths: 2^31 of 2,048.
@pytest.mark.parametrize("paths,ok", [(1, True), (262144, True), (600000, True), (4194304 - 2048, True), (4194304, False)])
def test_as_many_paths_as_before_are_accepted(rrb_lib, paths, ok):
    s = _batch(np.zeros((0, 2)), np.zeros(0, np.uint8), np.zeros(paths + 1, np.uint64), 1, 1 << 28, np.random.default_rng(0))
    s.pts, s.flags = np.zeros((1, 2)), np.zeros(1, np.uint8)  # every path but the last is empty
    s.path_pt_off[-1] = 1
    keep = []
    p = rrb_lib.batch_params(s.pts, s.flags, s.path_pt_off, s.fill_rule, s.gray, s.alpha, s.path_page, s.page_width,
                             s.page_height, s.page_offset, None, keep=keep)
    msg = C.create_string_buffer(256)
    rc = rrb_lib.lib().rrb_validate_path_batch(C.byref(p), 1 << 28, msg, 256)
    assert (rc == 0) == ok and (ok or b"too many tiles" in msg.value)


# 16 x 2^22 pixels have 16,384 supertiles: 262,144 paths are the last count with
# blocks of 256 (2^24 items), 262,145 the first with 2,048.
@pytest.mark.gpu
@pytest.mark.parametrize("paths,w,h", [(255, 300, 200), (256, 300, 200), (257, 300, 200), (2049, 600, 300),
                                       (262144, 16, 1 << 22), (262145, 16, 1 << 22)])
def test_pages_at_block_edges(rrb_lib, oracle, paths, w, h):
    s = _triangles(paths, w, h, paths)
    exp = np.full(s.arena_bytes, 255, np.uint8)
    oracle.render_scene(s, exp, threads=4)
    with rrb_lib.B200Backend(0) as be:
        pages, keep = be.alloc_device(s.arena_bytes), []
        p = rrb_lib.batch_params(s.pts, s.flags, s.path_pt_off, s.fill_rule, s.gray, s.alpha, s.path_page, s.page_width,
                                 s.page_height, s.page_offset, pages, keep=keep)
        be.begin_page()
        be.record_fill_buffer(pages, 255)
        be.record_path_batch(p)
        be.wait_page(be.submit_page())
        got = np.empty(s.arena_bytes, np.uint8)
        be.wait_download(be.download_async(pages, got))
        be.free_device(pages)
    d = np.nonzero(got != exp)[0]
    assert d.size == 0, f"{d.size} bytes differ, first at {d[:5]}"
