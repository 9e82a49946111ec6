"""Paths around the sizes where a path moves from a thread to a warp (64 points)
and to a block (1,024 points, 1,024 edges): the walk, the packing of its pieces
and the path boxes, with subpaths, curves and closing pieces across the steps
of 32 and 256 points, and paths that are not well formed among them."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _path(rng, n, w, h, broken):
    """n points of random subpaths: lines and curves, closed exactly or not, one malformed if broken."""
    pts, fl = [], []
    c = rng.uniform([0, 0], [w, h])
    while len(fl) < n:
        left = n - len(fl)
        k = int(min(left, rng.choice([1, 2, 5, 40, 300, 700])))
        start = len(fl)
        pts.append(c)
        fl.append(1)
        while len(fl) - start < k:
            c = np.clip(c + rng.normal(0, 9, 2), [-5, -5], [w + 5, h + 5])
            if k - (len(fl) - start) >= 3 and rng.random() < 0.4:
                pts += [c + rng.normal(0, 6, 2), c + rng.normal(0, 6, 2), c]
                fl += [8, 8, 0]
            else:
                pts.append(c)
                fl.append(0)
        if rng.random() < 0.5:
            pts[-1] = pts[start]
        fl[-1] |= 2
        c = rng.uniform([0, 0], [w, h])
    pts, fl = np.array(pts[:n]), np.array(fl[:n], np.uint8)
    if broken:
        fl[int(rng.integers(1, n))] ^= int(rng.choice([1, 2, 8]))
    return pts, fl


@pytest.mark.parametrize("sizes", [(63, 64, 65, 1023, 1024, 1025), (31, 255, 256, 257, 1280, 2049),
                                   (1500,) * 40, (3,) * 200 + (5000,) + (70,) * 60])
@pytest.mark.parametrize("broken", [False, True])
def test_long_paths_match_oracle(backend, oracle, rrb_lib, sizes, broken):
    rng = np.random.default_rng(len(sizes) + broken)
    w, h = 260, 190
    parts = [_path(rng, n, w, h, broken and rng.random() < 0.5) for n in sizes]
    n = len(parts)

    class S:
        pts = np.concatenate([p for p, _ in parts])
        flags = np.concatenate([f for _, f in parts])
        path_pt_off = np.concatenate([[0], np.cumsum([len(f) for _, f in parts])]).astype(np.uint64)
        fill_rule = rng.integers(0, 2, n).astype(np.uint8)
        gray = rng.integers(0, 256, n).astype(np.uint8)
        alpha = rng.integers(40, 256, n).astype(np.uint8)
        path_page = np.zeros(n, np.uint32)
        page_width, page_height = np.array([w], np.uint32), np.array([h], np.uint32)
        page_offset = np.zeros(1, np.uint64)

    exp = np.full(w * h, 255, np.uint8)
    oracle.render_scene(S, exp)
    pages, keep = backend.alloc_device(w * h), []
    try:
        p = rrb_lib.batch_params(S.pts, S.flags, S.path_pt_off, S.fill_rule, S.gray, S.alpha, S.path_page,
                                 S.page_width, S.page_height, S.page_offset, pages, keep=keep)
        backend.begin_page()
        backend.record_fill_buffer(pages, 255)
        backend.record_path_batch(p)
        backend.wait_page(backend.submit_page())
        got = np.empty(w * h, np.uint8)
        backend.wait_download(backend.download_async(pages, got))
        d = np.nonzero(got != exp)[0]
        assert d.size == 0, f"{d.size} bytes differ, first at {d[:5]}"
    finally:
        backend.free_device(pages)
