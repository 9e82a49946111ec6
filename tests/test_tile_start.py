"""Where the composite of a tile starts: stacks of translucent rectangles that
cover whole tiles, with shapes that do not between them, over pages of random
bytes. A run of full layers that takes 0 and 255 to one value hides what lies
below; anything shorter, or cut by a shape in the tile, does not. Depths,
alphas and narrow last tiles sit around both sides of that line, and every page
must be the oracle's byte for byte."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Stack:
    def __init__(self, rng, w, h, n, alphas, shapes):
        pts, flags, off = [], [], [0]
        for _ in range(n):
            u = rng.random()
            if u < shapes:  # a shape inside the page: triangle, or an L of edges along the axes
                x, y = rng.uniform(0, w), rng.uniform(0, h)
                a, b = rng.uniform(2, w / 2), rng.uniform(2, h / 2)
                p = ([(x, y), (x + a, y), (x, y + b)] if rng.random() < 0.6 else
                     [(x, y), (x + a, y), (x + a, y + b / 2), (x + a / 2, y + b / 2), (x + a / 2, y + b), (x, y + b)])
            elif u < shapes + 0.15:  # an L that holds most tiles
                p = [(-3, -3), (w + 3, -3), (w + 3, h - 9), (w - 20, h - 9), (w - 20, h + 3), (-3, h + 3)]
            else:  # the page, or all of it but a margin
                m = rng.choice([-2.0, 0.0, 0.3, 7.0])
                p = [(m, m), (w - m, m), (w - m, h - m), (m, h - m)]
            p.append(p[0])
            pts += p
            flags += [5] + [0] * (len(p) - 2) + [6]
            off.append(len(flags))
        self.pts, self.flags = np.array(pts, float), np.array(flags, np.uint8)
        self.path_pt_off = np.array(off, np.uint64)
        self.fill_rule = rng.integers(0, 2, n).astype(np.uint8)
        self.gray = rng.integers(0, 256, n).astype(np.uint8)
        self.alpha = rng.choice(alphas, n).astype(np.uint8)
        self.path_page = np.zeros(n, np.uint32)
        self.page_width, self.page_height = np.array([w], np.uint32), np.array([h], np.uint32)
        self.page_offset = np.zeros(1, np.uint64)


@pytest.mark.parametrize("tile", [(16, 16), (32, 32), (64, 16), (128, 16), (128, 32)])
@pytest.mark.parametrize("rgb", [False, True])
def test_stacks_of_full_layers(backend, oracle, rrb_lib, tile, rgb):
    rng = np.random.default_rng(5 * tile[0] + tile[1] + rgb)
    backend.set_tuning(*tile)
    try:
        for n, alphas, shapes in ((1, [255], 0.0), (3, [254, 255], 0.0), (9, [128], 0.0), (31, [60], 0.0),
                                  (40, [8], 0.1), (60, [1, 0], 0.0), (200, [32, 64, 128, 200, 255], 0.3),
                                  (300, list(range(32, 256)), 0.05), (900, list(range(32, 255)), 0.5)):
            w, h = int(rng.choice([300, 257, 128])), int(rng.choice([70, 33, 64]))
            s = _Stack(rng, w, h, n, alphas, shapes)
            bpp = 3 if rgb else 1
            page = rng.integers(0, 256, w * h * bpp, np.uint8)
            colours = rng.integers(0, 256, (n, 3), np.uint8) if rgb else None
            for rowmap in (0, 1):
                exp = page.copy()
                oracle.render_scene_ex(s, exp, rgb=colours, rowmap=rowmap)
                buf, keep = backend.alloc_device(page.size), []
                try:
                    backend.upload_async(buf, page)
                    p = rrb_lib.batch_params(s.pts, s.flags, s.path_pt_off, s.fill_rule, s.gray, s.alpha, s.path_page,
                                             s.page_width, s.page_height, s.page_offset, buf, rowmap=rowmap, keep=keep)
                    backend.begin_page()
                    backend.record_path_batch_ex(p, colours)
                    backend.wait_page(backend.submit_page())
                    got = np.empty_like(page)
                    backend.wait_download(backend.download_async(buf, got))
                    d = np.nonzero(got != exp)[0]
                    assert d.size == 0, f"{n} layers, {w}x{h}, row map {rowmap}: {d.size} bytes, first {d[:5]}"
                finally:
                    backend.free_device(buf)
    finally:
        backend.set_tuning(64, 16, auto_tile=True)
