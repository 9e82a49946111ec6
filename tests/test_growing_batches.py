"""Batches uploaded per call on one context, growing and changing in kind: each
is launched whole on the buffers that the ones before left, and rendered again
with the sizes read back where one of them does not fit (edges, row groups,
row runs, supertile pairs, cells, overflow rows). Translucent paint, so that a
page touched twice would show."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Comb:
    """One path of n teeth: rows of 2 n crossings (the overflow paths), on a w x h page."""

    def __init__(self, n, w, h):
        x = np.linspace(2, w - 2, 2 * n)
        y = np.where(np.arange(2 * n) % 2, h - 3.0, 2.0)
        self.pts = np.vstack([np.stack([x, y], 1), [(w - 2, h - 1.0), (2, h - 1.0), (x[0], y[0])]])
        m = len(self.pts)
        self.flags = np.array([5] + [0] * (m - 2) + [6], np.uint8)
        self.path_pt_off = np.array([0, m], np.uint64)
        self.fill_rule, self.gray = np.zeros(1, np.uint8), np.array([40], np.uint8)
        self.alpha, self.path_page = np.array([130], np.uint8), np.zeros(1, np.uint32)
        self.page_width, self.page_height = np.array([w], np.uint32), np.array([h], np.uint32)
        self.page_offset, self.arena_bytes = np.zeros(1, np.uint64), w * h


def test_growing_batches_match_oracle(rrb_lib, oracle):
    S = rrb_lib.Scene
    scenes = [S(kind=1, seed=1, n_paths=1, page_w=60, page_h=50), S(kind=1, seed=2, n_paths=3, page_w=70, page_h=900),
              S(kind=0, seed=3, n_paths=30, page_w=300, page_h=200), _Comb(30, 400, 60), _Comb(400, 900, 90),
              S(kind=2, seed=4, n_pages=3, page_scale=0.08, paths_scale=0.02),
              S(kind=2, seed=5, n_pages=6, page_scale=0.12, paths_scale=0.1), _Comb(40, 400, 60),
              S(kind=0, seed=6, n_paths=400, page_w=700, page_h=500), _Comb(1500, 3200, 70),
              S(kind=1, seed=7, n_paths=2500, page_w=900, page_h=700), S(kind=1, seed=8, n_paths=1, page_w=60, page_h=50)]
    with rrb_lib.B200Backend(0) as be:
        waits = []
        for i, s in enumerate(scenes):
            s.alpha = np.maximum(np.minimum(s.alpha, 200), 30).astype(np.uint8)
            exp = np.full(s.arena_bytes, 255, np.uint8)
            for _ in range(2):
                oracle.render_scene(s, exp, threads=4)
            pages, keep = be.alloc_device(s.arena_bytes), []
            p = rrb_lib.batch_params(s.pts, s.flags, s.path_pt_off, s.fill_rule, s.gray, s.alpha, s.path_page,
                                     s.page_width, s.page_height, s.page_offset, pages, keep=keep)
            be.begin_page()
            be.record_fill_buffer(pages, 255)
            for _ in range(2):  # the second finds the buffers that the first left
                be.record_path_batch(p)
                waits.append(be.last_batch_stats()["host_syncs"])
            be.wait_page(be.submit_page())
            got = np.empty(s.arena_bytes, np.uint8)
            be.wait_download(be.download_async(pages, got))
            be.free_device(pages)
            d = np.nonzero(got != exp)[0]
            assert d.size == 0, f"scene {i}: {d.size} bytes differ, first at {d[:5]}"
        assert min(waits) < max(waits)  # some were launched whole, some rendered again
