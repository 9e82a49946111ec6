"""Edge records at the ends of the number range: coordinates far off the page,
beyond int32 in AA units or in 16.16, steep and flat slopes (the fixed-point
step saturates), halves that round away from zero, and signed zeros. The
device converts with single instructions what the reference clamps step by step."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(rng, n, w, h, far):
    pts, flags, off = [], [], [0]
    for _ in range(n):
        k = int(rng.integers(3, 7))
        p = rng.uniform([-10, -10], [w + 10, h + 10], (k, 2))
        hit = rng.random((k, 2)) < 0.4
        p[hit] = rng.choice(far, hit.sum()) * rng.choice([-1.0, 1.0], hit.sum())
        if rng.random() < 0.3:
            p[1, 1] = p[0, 1] + rng.choice([1e-9, 1e-6, 0.125, 0.25])  # slopes that saturate, quarter rows
        if rng.random() < 0.3:
            p[2, 0] = p[1, 0] + (p[2, 1] - p[1, 1]) * (rng.integers(-9, 9) + 0.5) / 65536.0  # dxdy on a half
        pts += list(p) + [p[0]]
        flags += [5] + [0] * (k - 1) + [6]
        off.append(len(flags))

    class S:
        pass

    S.pts, S.flags, S.path_pt_off = np.array(pts), np.array(flags, np.uint8), np.array(off, np.uint64)
    S.fill_rule = rng.integers(0, 2, n).astype(np.uint8)
    S.gray, S.alpha = rng.integers(0, 256, n).astype(np.uint8), rng.integers(40, 256, n).astype(np.uint8)
    S.path_page = np.zeros(n, np.uint32)
    S.page_width, S.page_height = np.array([w], np.uint32), np.array([h], np.uint32)
    S.page_offset = np.zeros(1, np.uint64)
    return S


@pytest.mark.parametrize("far", [(0.0, 1e5, 32767.99, 8191.9999), (3e8, 536870911.75, 536870912.0, 1e9),
                                 (1e18, 1e100, 4.0e149), (0.0, 0.25, 0.5, 1e-300)])
def test_far_edges_match_oracle(backend, oracle, rrb_lib, far):
    rng = np.random.default_rng(int(far[-1] % 97) + len(far))
    w, h = 70, 50
    for rowmap in (0, 1):
        s = _scene(rng, 60, w, h, far)
        exp = np.full(w * h, 255, np.uint8)
        oracle.render_scene(s, exp, rowmap=rowmap)
        pages, keep = backend.alloc_device(w * h), []
        try:
            p = rrb_lib.batch_params(s.pts, s.flags, s.path_pt_off, s.fill_rule, s.gray, s.alpha, s.path_page,
                                     s.page_width, s.page_height, s.page_offset, pages, rowmap=rowmap, keep=keep)
            backend.begin_page()
            backend.record_fill_buffer(pages, 255)
            backend.record_path_batch(p)
            backend.wait_page(backend.submit_page())
            got = np.empty(w * h, np.uint8)
            backend.wait_download(backend.download_async(pages, got))
            d = np.nonzero(got != exp)[0]
            assert d.size == 0, f"row map {rowmap}: {d.size} bytes differ, first at {d[:5]}"
        finally:
            backend.free_device(pages)
