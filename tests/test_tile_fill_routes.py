"""tile_fill from segments goes straight to coverage or by sorted records, by what the sizes say is faster: which of
them a call takes (the records show in the memory that it uses), and the same coverage on both sides of each line."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(be, a):
    a = np.ascontiguousarray(a)
    buf = be.alloc_device(max(16, a.nbytes))
    be.wait_transfer(be.upload_async(buf, a.view(np.uint8).reshape(-1)))
    return buf


def _run(be, segs, w, h, rule):
    sb, cb = _dev(be, segs), be.alloc_device(w * h)
    try:
        used = be.detect_vram_budget().used_bytes
        be.begin_page()
        n = be.record_tile_fill_segs(sb, len(segs), cb, w, h, rule)
        be.wait_page(be.submit_page())
        used = be.detect_vram_budget().used_bytes - used
        got = np.empty(w * h, np.uint8)
        be.wait_download(be.download_async(cb, got))
        return got, n, used
    finally:
        be.free_device(sb)
        be.free_device(cb)


def _short(n, w, h, seed):
    rng = np.random.default_rng(seed)
    a = rng.uniform((-3, -3), (w + 3, h + 3), (n, 2))
    return np.concatenate([a, a + rng.normal(0, 2, (n, 2))], 1).astype(np.float32)


@pytest.mark.parametrize("w,h,n,by_records", [
    (17, 16, 8192, False), (17, 16, 8193, True), (300, 200, 32768, False), (300, 200, 32769, True),
    (4096, 4096, 17088, False), (4096, 4096, 17089, True), (8192, 8192, 4096, False), (8192, 8192, 32768, True)])
def test_the_sizes_choose_the_route(rrb_lib, oracle, w, h, n, by_records):
    segs = _short(n, w, h, n)
    recs, starts, counts, gw = oracle.build_tile_records(segs, 0.0, 0.0, w, h)
    with rrb_lib.B200Backend(0) as be:
        got, n_recs, used = _run(be, segs, w, h, 0)
    assert n_recs == len(recs)
    assert (used >= 32 * n_recs) == by_records
    assert np.array_equal(got, oracle.tile_fill(recs, starts, counts, gw, w, h, eo=False).ravel())
