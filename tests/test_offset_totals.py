"""Batches whose segments, pixel rows or supertile entries pass 2^32. The stages
address them by 32-bit offsets, which would wrap and leave a small total behind:
such a batch is refused with the pages untouched, and the context goes on."""

import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("counts,cap,fits", [
    ([5, 7], 12, True), ([5, 8], 12, False), ([], 0, True),
    ([0xFFFF0000], 0xFFFFFFFF, True), ([0xFFFF0000, 1], 0xFFFFFFFF, False),
    ([1 << 31, 1 << 31], 0xFFFFFFFF, False),          # wraps to 0
    ([0xFFFFFFFF, 0xFFFFFFFF, 10], 0xFFFFFFFF, False),  # wraps to 8
    ([1 << 22] * 1024, 0xFFFFFFFF, False), ([(1 << 22) - 64] * 1024, 0xFFFFFFFF, True)])
def test_a_total_that_wraps_does_not_fit(tmp_path_factory, counts, cap, fits):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not found")
    out = tmp_path_factory.getbasetemp() / "liboffset_totals.so"
    if not out.exists():
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-shared", "-Xcompiler",
                        "-fPIC", "-I", str(ROOT / "include"), "-o", str(out), str(ROOT / "tests" / "offset_totals_shim.cu")],
                       check=True, cwd=str(ROOT))
    a = np.array(counts, np.uint32)
    assert C.CDLL(str(out)).ot_fits(a.ctypes.data_as(C.c_void_p), C.c_uint64(len(a)), C.c_uint32(cap)) == fits


def _scene(pts, flags, n_paths, w, h):
    class S:
        pass

    s, per = S(), len(flags) // n_paths
    s.pts, s.flags = np.ascontiguousarray(pts, np.float64), np.ascontiguousarray(flags, np.uint8)
    s.path_pt_off = np.arange(n_paths + 1, dtype=np.uint64) * per
    s.fill_rule, s.path_page = np.zeros(n_paths, np.uint8), np.zeros(n_paths, np.uint32)
    s.gray, s.alpha = np.full(n_paths, 9, np.uint8), np.full(n_paths, 200, np.uint8)
    s.page_width, s.page_height = np.array([w], np.uint32), np.array([h], np.uint32)
    s.page_offset, s.arena_bytes = np.zeros(1, np.uint64), w * h
    return s


def _pairs():
    """2^18 rectangles and a few more over all 2^14 supertiles of a page 2^22 rows high: 2^32 supertile entries."""
    w, h, n = 16, 1 << 22, (1 << 18) + (1 << 12)
    one = np.array([[-1, -1], [w + 1, -1], [w + 1, h + 1], [-1, h + 1], [-1, -1]], np.float64)
    return _scene(np.tile(one, (n, 1)), np.tile(np.array([5, 0, 0, 0, 6], np.uint8), n), n, w, h)


def _rows():
    """1,100 paths of two specks at the ends of that page: 2^32 pixel rows, hardly any of them with a crossing."""
    w, h, n = 16, 1 << 22, 1100
    t = np.array([[2.0, 0.5], [9.0, 0.6], [4.0, 0.9], [2.0, 0.5]])
    one = np.concatenate([t, t + (0, h - 1)])
    return _scene(np.tile(one, (n, 1)), np.tile(np.array([5, 0, 0, 6, 5, 0, 0, 6], np.uint8), n), n, w, h)


def _segments():
    """5 x 2^20 curves of 1,024 segments each: 1.25 x 2^32 segments."""
    w, h, n, k = 16, 16, 5 << 10, 1 << 10
    one = np.zeros((3 * k + 1, 2))
    one[0] = (1, 1)
    one[1::3], one[2::3] = (4e6, 3e6), (-4e6, 5e6)
    one[3::3] = (9, 9)
    flags = np.full(3 * k + 1, 8, np.uint8)
    flags[0], flags[3::3], flags[-1] = 5, 0, 6
    return _scene(np.tile(one, (n, 1)), np.tile(flags, n), n, w, h)


@pytest.mark.gpu
@pytest.mark.parametrize("make", [_pairs, _rows, _segments])
def test_a_batch_past_32_bits_is_refused(rrb_lib, oracle, make):
    s = make()
    small = rrb_lib.Scene(kind=0, seed=5, n_paths=40, page_w=90, page_h=70)
    exp = small.blank_arena()
    oracle.render_scene(small, exp)
    with rrb_lib.B200Backend(0) as be:
        pages, keep = be.alloc_device(s.arena_bytes), []
        p = rrb_lib.batch_params(s.pts, s.flags, s.path_pt_off, s.fill_rule, s.gray, s.alpha, s.path_page, s.page_width,
                                 s.page_height, s.page_offset, pages, keep=keep)
        be.begin_page()
        be.record_fill_buffer(pages, 77)
        with pytest.raises(rrb_lib.BackendError) as e:
            be.record_path_batch(p)
        assert e.value.kind == "PoolExhausted" and "2^32" in str(e.value)
        be.wait_page(be.submit_page())
        got = np.empty(s.arena_bytes, np.uint8)
        be.wait_download(be.download_async(pages, got))
        assert (got == 77).all()
        got = small.blank_arena()
        be.render_scene(small, got)
        assert np.array_equal(got, exp)
        be.free_device(pages)
