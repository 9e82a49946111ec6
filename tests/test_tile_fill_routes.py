"""tile_fill from segments goes straight to coverage or by sorted records, by what the sizes and the segments say is
faster: which of them a call takes (the records show in the memory that it uses), and the same coverage on both sides of each
line."""

import ctypes as C

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
    (33, 30, 24576, None), (33, 30, 24577, True), (300, 200, 32768, False), (300, 200, 32769, True),
    (4096, 4096, 17088, False), (4096, 4096, 17089, True), (8192, 8192, 4096, False), (8192, 8192, 32768, True)])
def test_the_sizes_choose_the_route(rrb_lib, oracle, w, h, n, by_records):
    segs = _short(n, w, h, n)
    recs, starts, counts, gw = oracle.build_tile_records(segs, 0.0, 0.0, w, h)
    with rrb_lib.B200Backend(0) as be:
        got, n_recs, used = _run(be, segs, w, h, 0)
    assert n_recs == len(recs)
    assert by_records is None or (used >= 32 * n_recs) == by_records  # None: what the segments say
    assert np.array_equal(got, oracle.tile_fill(recs, starts, counts, gw, w, h, eo=False).ravel())


def _contents(kind, n, w, h):
    rng = np.random.default_rng(n)
    if kind == "long":
        return rng.uniform((-3, -3, -3, -3), (w + 3, h + 3, w + 3, h + 3), (n, 4)).astype(np.float32)
    if kind == "short":
        return _short(n, w, h, n)
    if kind in ("line", "corner"):  # a line of text; a tenth of both sides
        a = rng.uniform((0, 0), (w, 14) if kind == "line" else (w / 10, h / 10), (n, 2))
        return np.concatenate([a, a + rng.normal(0, 1, (n, 2)) * ((60, 8) if kind == "line" else (8, 8))], 1).astype(np.float32)
    a = rng.uniform((0, 0), (w, 20), (n, 2))  # crowded: the first 28 pixel rows
    s = np.concatenate([a, a + rng.normal(0, 3, (n, 2))], 1).astype(np.float32)
    s[::97, 0], s[::89, 3] = np.nan, np.inf
    return s


@pytest.mark.parametrize("w,h,n,kind,by_records", [
    (1024, 1024, 4096, "long", True), (1024, 1024, 9000, "long", True), (1024, 1024, 9000, "crowded", True),
    (200, 200, 9000, "crowded", False), (3000, 1200, 30000, "long", True), (40, 17000, 20000, "crowded", True),
    # Crowded in columns too, and few: seen beside the scan from 512 segments on, before it from 4,097.
    (917, 1341, 4097, "line", True), (917, 1341, 4096, "line", True), (917, 1341, 2000, "line", True),
    (917, 1341, 511, "line", False), (3000, 100, 6000, "corner", True), (3000, 100, 3000, "corner", True),
    (3000, 100, 2000, "crowded", None), (16, 16, 513, "long", None), (1, 1, 600, "crowded", None),
    # Cells of eight tile rows, and of two groups of tiles.
    (1024, 1024, 3000, "short", False), (8192, 8192, 5000, "short", False), (1048560, 16, 5000, "short", None)])
def test_the_segments_choose_the_route(rrb_lib, oracle, w, h, n, kind, by_records):
    """by_records: where the times of the two routes are well apart (None: either)."""
    segs = _contents(kind, n, w, h)
    recs, starts, counts, gw = oracle.build_tile_records(segs, 0.0, 0.0, w, h)
    for rule in (0, 1):
        with rrb_lib.B200Backend(0) as be:
            got, n_recs, used = _run(be, segs, w, h, rule)
        assert n_recs == len(recs)
        assert by_records is None or (used >= 32 * n_recs) == by_records
        assert np.array_equal(got, oracle.tile_fill(recs, starts, counts, gw, w, h, eo=bool(rule)).ravel())


@pytest.mark.parametrize("n", [3000, 9000])
def test_without_a_count(rrb_lib, oracle, n):
    w = h = 1024
    segs = _contents("long", n, w, h)
    recs, starts, counts, gw = oracle.build_tile_records(segs, 0.0, 0.0, w, h)
    with rrb_lib.B200Backend(0) as be:
        sb, cb = _dev(be, segs), be.alloc_device(w * h)
        be.begin_page()
        p = rrb_lib._abi.AaFillParams(segs=sb.handle, n_segs=n, coverage=cb.handle, width=w, height=h, fill_rule=0)
        assert rrb_lib.lib().rrb_record_tile_fill_segs(be.handle, C.byref(p), None) == 0
        be.wait_page(be.submit_page())
        got = np.empty(w * h, np.uint8)
        be.wait_download(be.download_async(cb, got))
    assert np.array_equal(got, oracle.tile_fill(recs, starts, counts, gw, w, h, eo=False).ravel())
