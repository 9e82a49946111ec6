"""Curves with long chords are handed to a warp each without counting first:
also those that have few segments after all (controls near the middle of the
chord: one leaf whatever the length), those just below and above the chord, and
curves with a chord of zero and many segments. Below and above the piece count
from which only curves of more than 16 segments go to a warp."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(n, w, h, seed):
    """n closed paths of three cubics between corners of a triangle."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(2, (w - 30, h - 30), (n, 2))
    # Chords around 0.63 and 10.1 pixels (the two limits at flatness 0.1), longer ones, and none at all.
    size = rng.choice([0.0, 0.3, 0.6, 0.64, 1.0, 10.0, 10.2, 14.0, 28.0], n)[:, None]
    corners = np.stack([a, a + size * (1, 0), a + size * (0.6, 0.8), a], 1)
    pts, flags = np.empty((n, 10, 2)), np.tile(np.array([5, 8, 8, 0, 8, 8, 0, 8, 8, 6], np.uint8), n)
    pts[:, 0] = corners[:, 0]
    for k in range(3):
        p, q = corners[:, k], corners[:, k + 1]
        mid = (p + q) / 2
        off = rng.choice([0.0, 0.05, 0.3, 3.0, 9.0], (n, 2, 1)) * rng.uniform(-1, 1, (n, 2, 2))
        pts[:, 3 * k + 1], pts[:, 3 * k + 2], pts[:, 3 * k + 3] = mid + off[:, 0], mid + off[:, 1], q

    class S:
        pass

    s = S()
    s.pts, s.flags, s.path_pt_off = pts.reshape(-1, 2), flags, np.arange(n + 1, dtype=np.uint64) * 10
    s.fill_rule, s.path_page = rng.integers(0, 2, n).astype(np.uint8), np.zeros(n, np.uint32)
    s.gray, s.alpha = rng.integers(0, 256, n).astype(np.uint8), rng.integers(90, 201, n).astype(np.uint8)
    s.page_width, s.page_height = np.array([w], np.uint32), np.array([h], np.uint32)
    s.page_offset, s.arena_bytes = np.zeros(1, np.uint64), w * h
    return s


@pytest.mark.parametrize("n,w,h", [(1, 40, 40), (200, 300, 200), (45000, 1300, 900)])
def test_routed_curves_match_oracle(rrb_lib, oracle, n, w, h):
    s = _scene(n, w, h, n)
    exp = np.full(s.arena_bytes, 255, np.uint8)
    oracle.render_scene(s, exp, threads=4)
    with rrb_lib.B200Backend(0) as be:
        pages, keep = be.alloc_device(s.arena_bytes), []
        p = rrb_lib.batch_params(s.pts, s.flags, s.path_pt_off, s.fill_rule, s.gray, s.alpha, s.path_page, s.page_width,
                                 s.page_height, s.page_offset, pages, keep=keep)
        for _ in range(2):  # by size, then launched whole
            be.begin_page()
            be.record_fill_buffer(pages, 255)
            be.record_path_batch(p)
            be.wait_page(be.submit_page())
            got = np.empty(s.arena_bytes, np.uint8)
            be.wait_download(be.download_async(pages, got))
            d = np.nonzero(got != exp)[0]
            assert d.size == 0, f"{d.size} bytes differ, first at {d[:5]}"
            assert be.last_batch_stats()["pieces"] > (131072 if n > 40000 else 0)
        be.free_device(pages)
