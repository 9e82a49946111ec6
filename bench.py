"""Benchmark of the B200 anti-aliased fill (one JSON line on rank 0).

Workload (default): the mixed batch — 64 u8 pages whose sizes are drawn from
{A4, Letter, A3} x {150, 300, 600} dpi (1.17 Gpixel in all), 662,271 paths:
30% glyph outlines, 40% polygons, 30% axis-aligned rectangles covering 5-80%
of their page, alpha 32-255, seed 0 — rendered in ONE submission. A step
fills the pages with 255, flattens every path in FP64, builds the AA rows,
bins paths to tiles and composites them in order. `--workload glyphs` is the
glyph-dense text page (150,000 glyphs on one Letter @300 dpi page),
`--workload polygons` the 2,000-path polygon page.

  value  Mpixel/s with the path inputs already resident in device memory
         (rrb_batch_upload once, rrb_record_batch per step), timed with CUDA
         events on the backend's own stream, max over ranks.
  e2e    the same metric through rrb_render_pages_host_init with pinned HOST
         buffers: the path arrays go host->device, the pages start white on
         the device and come back to the host every step.
  bit_exact  every page of the batch against the CPU oracle: the mixed batch
         by the SHA-256 of each page that the oracle rendered
         (tests/golden/mixed_batch_digests.json), one-page workloads by the
         oracle's page itself.

Multi-GPU: pages are independent, so N ranks split a multi-page batch's pages
(strong scaling) or render replicas of a one-page workload (weak scaling),
with no collective on the data path; only the timing barrier and the
max-over-ranks reduction use torch.distributed.

`--impl reference` times the reference CPU scanline rasterizer's
restatement (oracle/; the reference itself is Rust and cannot be built here)
on the host cores, page-parallel as the reference's per-page workers: each
thread renders the leading paths of its own page of the batch.
"""

from __future__ import annotations

import argparse
import ctypes as C
import json
import os
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path[:0] = [str(ROOT / "pdf-raster_b200"), str(ROOT / "oracle")]

METRIC = "bit-exact Mpixel/s & edges/s, batched vs plain per-path GPU; p99 page latency"
WORKLOADS = {
    "glyphs": (dict(kind=1, seed=0),
               "glyph-dense text page: 150,000 quadratic glyph paths (2 contours avg, 12-60 quads each, "
               "8-12 pt em @300 dpi, 60 baselines) on one 2550x3300 u8 page (Letter @300 dpi), NZ, gray 0, alpha 255"),
    "mixed": (dict(kind=2, seed=0),
              "mixed pages in one batch: 64 u8 pages of {A4, Letter, A3} x {150, 300, 600} dpi (1.17 Gpixel), "
              "log-normal path count (median 5,000, sigma 1.2, cap 50,000; 662,271 paths) of 30% glyphs / 40% "
              "polygons / 30% axis-aligned rectangles covering 5-80% of the page, alpha 32-255, one submission"),
    "polygons": (dict(kind=0, seed=0),
                 "polygon page: 2,000 closed paths (1-3 contours x 4-32 line/cubic segments, jittered circles, "
                 "log-normal radius) on one 2550x3300 u8 page, NZ 70% / EO 30%, opaque"),
}
CLOCK_FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
                "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
                "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")


def dist_env():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    return int(os.environ.get("RANK", "0")), int(os.environ.get("LOCAL_RANK", "0")), ws


class Clocks:
    """nvidia-smi sampling during the timed region."""

    def __init__(self, device: int):
        self.device, self.proc, self.path = device, None, None

    def start(self):
        try:
            self.path = Path(os.environ.get("TMPDIR", "/tmp")) / f"rrb_clocks_{os.getpid()}.csv"
            self.f = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.device), f"--query-gpu={CLOCK_FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "100"], stdout=self.f,
                                         stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self) -> dict:
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        self.proc.wait()
        self.f.close()
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in self.path.read_text().splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx.append(float(f[2]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        self.path.unlink(missing_ok=True)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "samples": len(sm), "reasons": sorted(reasons)}


# DRAM bytes per flattened segment of the row stage on the glyph page:
# dram__bytes_read.sum + dram__bytes_write.sum of one ncu capture of k_rows on
# the glyph page reduced to 30,000 paths (10,979,156 segments, edge records
# larger than L2), scaled to a full launch by its segment count.
GLYPH_DRAM_BYTES_PER_SEGMENT = {
    "rows": (388_048_896 + 44_584_960) / 10_979_156,
}


# DRAM bytes per page pixel of the composite on the mixed batch:
# dram__bytes_read.sum + dram__bytes_write.sum of one ncu capture of
# k_composite<128, 16> on page 0 of the batch alone (3508x4961, 17,589 paths;
# the page's last layers stay in L2), scaled to a launch by its pixels.
MIXED_DRAM_BYTES_PER_PIXEL = {
    "composite": (16_695_808 + 1_127_680) / (3508 * 4961),
}


# Row-stage shapes (rrb_batch_stats.row_shape): list entries per AA row x
# warps per block x 32-edge groups staged per warp.
ROW_STAGES = ["12 entries x 8 warps, 512 edges staged per block", "16 entries x 4 warps, 256 edges per block",
              "12 entries x 8 warps, 256 edges per block", "8 entries x 16 warps, 1024 edges per block",
              "16 entries x 4 warps, 128 edges per block"]


L2_BYTES = 126 << 20
FLUSH_BYTES = 512 << 20


def needs_l2_flush(scene) -> bool:
    """Whether a step's inputs (path points and flags, and the pages) fit in
    twice the L2: then every timed step starts after an L2 flush."""
    return 17 * scene.n_pts + scene.pixels < 2 * L2_BYTES


def workload_config(desc, scene, rowmap):
    """The line's `config`: the workload alone, the same in the B200 line and
    the reference line of one workload (device choices go under `device`)."""
    inputs = 17 * scene.n_pts + scene.pixels
    l2 = (f"L2 flushed before every timed step ({FLUSH_BYTES >> 20} MB written; inputs {inputs / 1e6:.0f} MB)"
          if needs_l2_flush(scene) else f"inputs larger than L2 ({inputs / 1e6:.0f} MB of path points and pages)")
    return {"workload": desc, "paths": scene.n_paths, "pages": scene.n_pages,
            "rowmap": ["documented", "as_shipped"][rowmap], "l2": l2}


def measured_peak():
    """HBM copy bandwidth measured on this pool's B200s (MEASURED_PEAKS.json,
    `hbm_gbs`), else the recipe's fallback, 6,650 GB/s."""
    p = ROOT / "MEASURED_PEAKS.json"
    try:
        d = json.loads(p.read_text())
        v = d.get("hbm_gbs")
        if isinstance(v, dict):  # a burst / sustained pair
            v = v.get("burst", v.get("value"))
        if v:
            return float(v), "measured"
    except (OSError, ValueError, TypeError, AttributeError):
        pass
    return 6650.0, "fallback"


def oracle_page(scene, threads=1):
    import rr_oracle
    rr_oracle.build()
    a = scene.blank_arena()
    t = time.perf_counter()
    st = rr_oracle.render_scene(scene, a, threads=threads)
    return a, time.perf_counter() - t, st


class PathRange:
    """Paths [a, b) of a one-page scene, as a scene of their own (the oracle
    composites them onto the page exactly as it would inside the whole page)."""

    def __init__(self, page, a, b):
        p0, p1 = int(page.path_pt_off[a]), int(page.path_pt_off[b])
        self.pts, self.flags = page.pts[p0:p1], page.flags[p0:p1]
        self.path_pt_off = (page.path_pt_off[a:b + 1] - p0).astype(np.uint64)
        self.fill_rule, self.gray, self.alpha = page.fill_rule[a:b], page.gray[a:b], page.alpha[a:b]
        self.path_page = np.zeros(b - a, np.uint32)
        self.page_width, self.page_height = page.page_width, page.page_height
        self.page_offset = np.zeros(1, np.uint64)


def oracle_prefix(page, arena, budget_s):
    """The oracle, one thread, over the leading paths of a one-page scene
    until budget_s seconds: (paths done, seconds, unpinned tie rows)."""
    import rr_oracle
    rr_oracle.build()
    done, spent, ties, chunk = 0, 0.0, 0, 16
    while done < page.n_paths and spent < budget_s:
        e = min(page.n_paths, done + chunk)
        t = time.perf_counter()
        st = rr_oracle.render_scene(PathRange(page, done, e), arena)
        dt = time.perf_counter() - t
        spent += dt
        ties += st["unpinned_tie_rows"]
        done = e
        if dt < 0.25:
            chunk *= 2
    return done, spent, ties


class PageParallelSample:
    """A bounded sample of a multi-page batch for the CPU oracle, page-parallel
    as the reference renders pages (one page per rayon worker): thread t takes
    page t of the batch (pages reused when threads outnumber them) and renders
    its leading paths. calibrate() finds, on all threads at once, how many
    leading paths each renders in about budget_s; step() renders exactly those
    paths on every thread and returns the wall time; credited_px is each
    page's pixels times the share of its paths sampled, summed."""

    def __init__(self, scene, threads, budget_s):
        from rrb.shard import SceneShard
        self.threads = max(1, threads)
        self.subs = [SceneShard(scene, pages=(t % scene.n_pages, t % scene.n_pages + 1)) for t in range(self.threads)]
        ks = [0] * self.threads

        def cal(t):
            ks[t], _, _ = oracle_prefix(self.subs[t], self.subs[t].blank_arena(), budget_s)

        _run_threads(cal, self.threads)
        self.work = [PathRange(self.subs[t], 0, max(1, ks[t])) for t in range(self.threads)]
        self.paths = [w.fill_rule.size for w in self.work]
        self.credited_px = sum(sub.pixels * k / max(1, sub.n_paths) for sub, k in zip(self.subs, self.paths))
        self.arenas = [np.full(int(w.page_width[0]) * int(w.page_height[0]), 255, np.uint8) for w in self.work]

    def step(self) -> float:
        import rr_oracle
        for a in self.arenas:
            a.fill(255)
        t = time.perf_counter()
        _run_threads(lambda k: rr_oracle.render_scene(self.work[k], self.arenas[k]), self.threads)
        return time.perf_counter() - t

    def describe(self) -> str:
        return (f"{self.threads} host threads at once, thread t on page t of the batch (its first "
                f"{min(self.paths)}-{max(self.paths)} paths, the number each thread renders in about the budget), "
                "credited with each page's pixels times the share of its paths rendered")


def _run_threads(fn, n):
    ts = [threading.Thread(target=fn, args=(k,)) for k in range(n)]
    for x in ts:
        x.start()
    for x in ts:
        x.join()


def batch_digests_check(scene, pages_arena) -> dict | None:
    """Compare every page of the mixed batch with the oracle's pinned SHA-256
    digests (tests/golden/mixed_batch_digests.json, made by
    tests/golden/make_batch_digests.py); None when the scene is not that batch."""
    import hashlib
    path = ROOT / "tests" / "golden" / "mixed_batch_digests.json"
    if not path.exists() or scene.n_pages != 64:
        return None
    doc = json.loads(path.read_text())
    recs = doc["records"]
    ok, bad = 0, []
    for rec in recs:
        pg = rec["page"]
        o, w, h = int(scene.page_offset[pg]), int(scene.page_width[pg]), int(scene.page_height[pg])
        if (w, h) != (rec["width"], rec["height"]):
            return None
        d = hashlib.sha256(np.ascontiguousarray(pages_arena[o:o + w * h]).tobytes()).hexdigest()
        if d == rec["page_sha256"]:
            ok += 1
        else:
            bad.append(pg)
    return {"pages_checked": len(recs), "pages_bit_exact": ok, "pages_differing": bad,
            "reference": "SHA-256 of each page rendered by the CPU oracle (tests/golden/mixed_batch_digests.json)"}


def run_reference(args, rank, world):
    """The reference CPU path (its restatement) on the host cores."""
    if rank != 0:
        return
    import rr_oracle
    import rrb
    from rrb import scenes
    rr_oracle.build()
    # Inputs from the oracle's build of the workload generator (same source and
    # flags as the package's): this process maps oracle/ libraries only.
    scenes.use_library(rr_oracle.SCENES_LIB_PATH)
    if args.workload == "fill_ops":
        print(json.dumps({"impl": "reference", "unavailable": "the fill_ops line times aa_fill_cpu (the "
                                                             "reference's own CPU coverage) as its cpu_baseline"}))
        return
    render = rr_oracle.render_scene
    if args.workload == "strokes":
        from rrb.strokes import StrokePage
        scene = StrokePage(0, n_paths=args.paths or 20000)
        desc = scene.description

        def render(work, arena, threads=1):
            return rr_oracle.render_scene_paint(work, arena, work.strokes, threads=threads)
    else:
        kw, desc = WORKLOADS[args.workload]
        scene = rrb.Scene(**kw)
    cores = len(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else (os.cpu_count() or 1)
    threads = max(1, min(cores, args.ref_threads) if args.ref_threads > 0 else cores)
    if scene.n_pages > 1:
        # Page-parallel on the host cores: each thread renders the leading
        # paths of its own page (about 2 s of work each per step).
        sample = PageParallelSample(scene, threads, 2.0)
        step, px_per_step, sample_desc = sample.step, sample.credited_px, sample.describe()
        pages_per_step = threads
    else:
        arenas = [scene.blank_arena() for _ in range(threads)]

        def step():
            for a in arenas:
                a.fill(255)
            t = time.perf_counter()
            _run_threads(lambda k: render(scene, arenas[k], threads=1), threads)
            return time.perf_counter() - t

        px_per_step = scene.pixels * threads
        sample_desc = (f"{threads} copies of the page per step, one per host thread (the reference renders one "
                       "page per worker)")
        pages_per_step = threads
    for _ in range(args.warmup):
        step()
    times = [step() for _ in range(args.steps)]
    total = sum(times)
    mpx = px_per_step * args.steps / total / 1e6
    line = {"impl": "reference", "metric": METRIC, "value": mpx, "unit": "Mpixel/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * total / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u8",
            "data": "synthetic (seeded generator, seed 0; no public dataset for this path)",
            "config": (workload_config(desc, scene, args.rowmap) if args.workload != "strokes"
                       else {"workload": desc}),
            "pages_per_step": pages_per_step,
            "cpu_baseline": {"value": mpx, "unit": "Mpixel/s", "cores": threads, "kind": "port",
                             "sample": sample_desc,
                             "coverage_tier": ["scalar", "avx2", "avx512_bitalg"][rr_oracle.coverage_tier()]},
            "e2e": {"value": mpx, "unit": "Mpixel/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def pinned_copy(backend, arr, keep):
    arr = np.ascontiguousarray(arr)
    buf = backend.alloc_host_pinned(max(1, arr.nbytes))
    v = buf.array()[: arr.nbytes].view(arr.dtype)
    v[:] = arr.reshape(-1)
    keep.append(buf)
    return v


def run_rrb(args, rank, local, world):
    import rrb

    dist = None
    if world > 1:
        import torch
        import torch.distributed as tdist
        torch.cuda.set_device(local)
        tdist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=120))
        dist = tdist
    import torch

    kw, desc = WORKLOADS[args.workload]
    if args.paths:
        kw = dict(kw, n_paths=args.paths)
        desc += f" [reduced to {args.paths} paths]"
    full_scene = rrb.Scene(**kw)
    if args.pages:
        # A page range of a multi-page batch (profiling captures of a reduced case).
        from rrb.shard import SceneShard
        p0, p1 = (int(v) for v in args.pages.split(":"))
        full_scene = SceneShard(full_scene, pages=(p0, p1))
        desc += f" [pages {p0}:{p1} only]"
    # Several pages and several ranks: each rank renders its share of the
    # pages (strong scaling over the fixed batch); one page: replicas (weak).
    sharded = world > 1 and full_scene.n_pages > 1
    if sharded:
        from rrb.shard import SceneShard
        scene = SceneShard(full_scene, rank, world)
    else:
        scene = full_scene
    backend = rrb.B200Backend(local)
    if args.tile:
        # A fixed tile shape (profiling runs): no tile trials.
        tw, th = (int(v) for v in args.tile.split("x"))
        backend.set_tuning(tw, th)
    if args.wave_points:
        backend.set_tuning(wave_points=args.wave_points, auto_tile=not args.tile)
    tuning = backend.get_tuning()
    pages = backend.alloc_device(scene.arena_bytes)
    scene.view.pages = None
    batch = backend.batch_upload(scene.view)
    stream = torch.cuda.ExternalStream(backend.stream, device=torch.device("cuda", local))

    def step():
        backend.begin_page()
        backend.record_fill_buffer(pages, 255)
        batch.record(pages, args.rowmap)
        backend.wait_page(backend.submit_page())

    # Tuning renders (untimed, before the warm-up): the resident batch tries
    # each tile shape x row-stage shape and keeps the fastest.
    for _ in range(24):
        step()
        if backend.last_batch_stats()["trials_left"] == 0:
            break
    for _ in range(args.warmup):
        step()
    # ---- timed region: resident inputs, per-stage events inside the library
    backend.set_profiling(True)
    stage_acc, launches, step_ms = {}, 0, []
    # Start and end events per step: an L2 flush (small inputs) runs between
    # steps, outside the timed spans.
    ev0 = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    ev1 = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    flush = (torch.empty(FLUSH_BYTES, dtype=torch.uint8, device=f"cuda:{local}")
             if needs_l2_flush(full_scene) else None)
    clocks = Clocks(local)
    if dist:
        dist.barrier()
    torch.cuda.synchronize(local)
    clocks.start()
    for k in range(args.steps):
        if flush is not None:
            with torch.cuda.stream(stream):
                flush.fill_(k & 0xff)
        ev0[k].record(stream)
        step()
        ev1[k].record(stream)
        st = backend.last_batch_stats()
        launches += st["kernel_launches"]
        for name, (ms, nl) in backend.stage_times().items():
            a = stage_acc.setdefault(name, [0.0, 0])
            a[0] += ms
            a[1] += nl
    torch.cuda.synchronize(local)
    clk = clocks.stop()
    backend.set_profiling(False)
    step_ms = [ev0[k].elapsed_time(ev1[k]) for k in range(args.steps)]
    total_ms = sum(step_ms)
    if dist:
        t = torch.tensor([total_ms], device=f"cuda:{local}")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        total_ms = float(t.item())
    stats = backend.last_batch_stats()
    ms_per_step = total_ms / args.steps
    px = scene.pixels
    job_px = full_scene.pixels if sharded else px * world  # pixels all ranks render per step
    value = job_px * args.steps / (total_ms / 1e3) / 1e6
    edges_s = stats["segments"] * world * args.steps / (total_ms / 1e3)

    # ---- roofline of the dominant kernel (HBM-bound integer work)
    peak, peak_kind = measured_peak()
    stage_ms = {k: v[0] / args.steps for k, v in stage_acc.items()}
    dom = max(stage_ms, key=stage_ms.get)
    alg = {
        # page read + written once, each coverage cell (4 B) and pixel-row index entry (8 B) read once
        "composite": 2 * px + 4 * stats["spans"] + 8 * stats["row_groups"],
        # each edge record (32 B) read once, pixel-row index (8 B/entry) and cells (4 B) written once (an
        # upper bound where later layers hide rows: those are not built)
        "rows": 32 * stats["segments"] + 8 * stats["row_groups"] + 4 * stats["spans"],
        # path points (16 B) + flags read, edge records written
        "seg_write": 17 * scene.n_pts + 32 * stats["segments"],
        "seg_count": 17 * scene.n_pts + 4 * scene.n_pts,
    }
    alg_b = alg.get(dom)
    roofline = None
    if alg_b:
        # The stage runs its dominant kernel once per wave (k_rows beside the
        # short k_chunk_paths / k_recti launches): per launch = per step / waves.
        waves = max(1, int(stats.get("waves", 1)))
        dur = stage_ms[dom] / waves / 1e3
        ach = alg_b / waves / dur / 1e9
        per_seg = GLYPH_DRAM_BYTES_PER_SEGMENT.get(dom) if args.workload == "glyphs" else None
        per_px = MIXED_DRAM_BYTES_PER_PIXEL.get(dom) if args.workload == "mixed" else None
        traffic = (per_seg * stats["segments"] / waves if per_seg else
                   per_px * px / waves if per_px else None)
        roofline = {"kernel": dom, "bound": "hbm", "achieved": ach, "peak": peak, "unit": "GB/s",
                    "frac": ach / peak, "traffic": traffic, "peak_source": peak_kind,
                    "algorithmic_bytes_per_launch": alg_b / waves, "launch_ms": dur * 1e3,
                    "traffic_source": ("ncu capture of the glyph page at 30,000 paths, scaled by segments"
                                       if per_seg else
                                       "ncu capture of page 0 of the batch alone, scaled by pixels"
                                       if per_px else None)}

    # ---- plain per-path form on a sample of paths (one record_path_fill per path)
    plain = None
    if args.plain_sample > 0 and rank == 0:
        W, H = int(scene.page_width[0]), int(scene.page_height[0])
        n = min(args.plain_sample, scene.n_paths)
        t0 = torch.cuda.Event(enable_timing=True)
        t1 = torch.cuda.Event(enable_timing=True)
        backend.begin_page()
        backend.record_fill_buffer(pages, 255)
        t0.record(stream)
        for p in range(n):
            a, b = int(scene.path_pt_off[p]), int(scene.path_pt_off[p + 1])
            backend.record_path_fill(scene.pts[a:b], scene.flags[a:b], pages, W, H,
                                     fill_rule=int(scene.fill_rule[p]), gray=int(scene.gray[p]),
                                     alpha=int(scene.alpha[p]), rowmap=args.rowmap)
        t1.record(stream)
        backend.wait_page(backend.submit_page())
        torch.cuda.synchronize(local)
        per_path = t0.elapsed_time(t1) / n
        plain_mpx = px / (per_path * scene.n_paths / 1e3) / 1e6
        plain = {"mpixel_s": plain_mpx, "sample_paths": n, "ms_per_path": per_path,
                 "batched_speedup": value / world / plain_mpx}

    # ---- end to end through the public API with pinned host buffers
    keep = []
    h = {k: pinned_copy(backend, getattr(scene, k), keep) for k in (
        "pts", "flags", "path_pt_off", "fill_rule", "gray", "alpha", "path_page", "page_width", "page_height",
        "page_offset")}
    params = rrb.batch_params(h["pts"], h["flags"], h["path_pt_off"], h["fill_rule"], h["gray"], h["alpha"],
                              h["path_page"], h["page_width"], h["page_height"], h["page_offset"], pages,
                              rowmap=args.rowmap)
    host_page = pinned_copy(backend, scene.blank_arena(), keep)
    e2e_steps = max(1, min(args.steps, args.e2e_steps))
    # The pages start white (255), as the workload defines them: the device
    # fills them (rrb_render_pages_host_init), so only the path arrays go up
    # and the rendered pages come down.
    backend.render_pages_host(params, host_page, init=255)  # warm
    if dist:
        dist.barrier()
    t = time.perf_counter()
    for _ in range(e2e_steps):
        backend.render_pages_host(params, host_page, init=255)
    e2e_s = time.perf_counter() - t
    if dist:
        tt = torch.tensor([e2e_s], device=f"cuda:{local}")
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        e2e_s = float(tt.item())
    h2d = sum(int(h[k].nbytes) for k in h)
    # The host link alone: the same bytes as one pinned copy, for the bound e2e meets.
    scratch = backend.alloc_device(int(h["pts"].nbytes))
    backend.wait_transfer(backend.upload_async(scratch, h["pts"]))
    t = time.perf_counter()
    for _ in range(3):
        backend.wait_transfer(backend.upload_async(scratch, h["pts"]))
    link_gbs = 3 * h["pts"].nbytes / (time.perf_counter() - t) / 1e9
    backend.free_device(scratch)
    e2e = {"value": job_px * e2e_steps / e2e_s / 1e6, "unit": "Mpixel/s", "h2d_bytes_per_step": h2d,
           "d2h_bytes_per_step": int(host_page.nbytes), "steps": e2e_steps,
           "api": "rrb_render_pages_host_init (C ABI, pages filled with 255 on the device), pinned host buffers",
           "h2d_link_gbs": link_gbs, "h2d_bound_ms": h2d / link_gbs / 1e6}

    # ---- parity check and CPU baseline (rank 0, N = 1)
    gpu_page = np.empty(scene.arena_bytes, np.uint8)
    backend.wait_download(backend.download_async(pages, gpu_page))
    cpu = None
    bit_exact = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline and scene.n_pages == 1:
        ref, secs, ost = oracle_page(scene, threads=1)
        bit_exact = bool(np.array_equal(ref, np.asarray(host_page)) and np.array_equal(ref, gpu_page))
        cpu = {"value": px / secs / 1e6, "unit": "Mpixel/s", "cores": 1, "kind": "port",
               "sample": "the whole page (all paths), 1 host thread, C++ restatement of the reference CPU path",
               "seconds": secs, "unpinned_tie_rows": ost["unpinned_tie_rows"],
               "coverage_tier": ["scalar", "avx2", "avx512_bitalg"][__import__("rr_oracle").coverage_tier()]}
    parity = None
    if scene.n_pages > 1 and not sharded:
        # Every page of the batch, device and end-to-end arenas, against the
        # oracle's pinned page digests.
        parity = batch_digests_check(scene, gpu_page)
        e2e_parity = batch_digests_check(scene, np.asarray(host_page))
        if parity is not None:
            bit_exact = (parity["pages_bit_exact"] == parity["pages_checked"] and e2e_parity is not None and
                         e2e_parity["pages_bit_exact"] == e2e_parity["pages_checked"])
    if rank == 0 and world == 1 and not args.no_cpu_baseline and scene.n_pages > 1:
        import rr_oracle
        rr_oracle.build()
        cores = len(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else (os.cpu_count() or 1)
        threads = max(1, min(cores, args.ref_threads) if args.ref_threads > 0 else cores)
        sample = PageParallelSample(scene, threads, 2.0)
        secs = sample.step()
        cpu = {"value": sample.credited_px / secs / 1e6, "unit": "Mpixel/s", "cores": threads, "kind": "port",
               "sample": sample.describe() + "; C++ restatement of the reference CPU path, page-parallel",
               "seconds": secs,
               "coverage_tier": ["scalar", "avx2", "avx512_bitalg"][rr_oracle.coverage_tier()]}
    batch.free()
    if rank == 0:
        p50, p99 = (float(np.percentile(step_ms, q)) for q in (50, 99))
        line = {
            "metric": METRIC, "value": value, "unit": "Mpixel/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_per_step, "higher_is_better": True,
            "scaling": "strong" if sharded else "weak",
            "vs_baseline": None, "dtype": "u8",
            "data": "synthetic (seeded generator, seed 0; no public dataset for this path)",
            "config": workload_config(desc, full_scene, args.rowmap),
            "device": {"tile": f"{stats['tile_w']}x{stats['tile_h']} (chosen by trial among 64x16, 128x16 and 128x32)"
                               if tuning.auto_tile == 1 else f"{stats['tile_w']}x{stats['tile_h']}",
                       "row_stage": ROW_STAGES[int(stats["row_shape"])],
                       "parallelism": (f"pages sharded over {world} GPUs" if sharded
                                       else f"replicas x{world} (the page on every GPU)")},
            "edges_per_s": edges_s, "segments_per_step": stats["segments"],
            "input_segments_per_step": scene.n_lines + scene.n_cubics,
            "p50_page_ms": p50, "p99_page_ms": p99,
            "plain_per_path": plain, "bit_exact": bit_exact, "parity": parity,
            "roofline": roofline, "stages_ms": stage_ms,
            "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": launches, "clocks": clk,
        }
        print(json.dumps(line), flush=True)
    backend.free_device(pages)
    backend.close()
    if dist:
        dist.destroy_process_group()


def run_strokes(args, rank, local, world):
    """Stroke-heavy page through rrb_record_stroke_batch: host outlines (every
    cap, join and dash), hairline spans and fills, all composited on the
    device. A step is one whole call: the host stroker, the upload of the
    outlines and the device render."""
    import torch

    import rrb
    from rrb.strokes import StrokePage

    if world > 1:
        torch.cuda.set_device(local)
    page = StrokePage(0, n_paths=args.paths or 20000)
    backend = rrb.B200Backend(local)
    pages = backend.alloc_device(page.arena_bytes)
    keep = []
    params = rrb.batch_params(page.pts, page.flags, page.path_pt_off, page.fill_rule, page.gray, page.alpha,
                              page.path_page, page.page_width, page.page_height, page.page_offset, pages, keep=keep)
    stream = torch.cuda.ExternalStream(backend.stream, device=torch.device("cuda", local))
    # The per-path stroke parameters as the C array the call takes, made once
    # (as a caller keeps its paint records), like the batch arrays above.
    strokes = rrb.stroke_params(page.strokes, keep)

    def step():
        backend.begin_page()
        backend.record_fill_buffer(pages, 255)
        backend.record_stroke_batch(params, strokes)
        backend.wait_page(backend.submit_page())

    for _ in range(args.warmup):
        step()
    backend.set_profiling(True)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps + 1)]
    stage_acc, launches = {}, 0
    clocks = Clocks(local)
    torch.cuda.synchronize(local)
    clocks.start()
    ev[0].record(stream)
    for k in range(args.steps):
        step()
        ev[k + 1].record(stream)
        launches += backend.last_batch_stats()["kernel_launches"]
        for name, (ms, nl) in backend.stage_times().items():
            a = stage_acc.setdefault(name, [0.0, 0])
            a[0] += ms
            a[1] += nl
    torch.cuda.synchronize(local)
    clk = clocks.stop()
    backend.set_profiling(False)
    total_ms = ev[0].elapsed_time(ev[-1])
    step_ms = [ev[k].elapsed_time(ev[k + 1]) for k in range(args.steps)]
    stats = backend.last_batch_stats()
    stage_ms = {k: v[0] / args.steps for k, v in stage_acc.items()}
    device_ms = sum(stage_ms.values())
    value = page.pixels * world * args.steps / (total_ms / 1e3) / 1e6
    # End to end: the page arena from pinned host memory and back each step.
    host_page = pinned_copy(backend, page.blank_arena(), keep)
    e2e_steps = max(1, min(args.steps, args.e2e_steps))
    t = time.perf_counter()
    for _ in range(e2e_steps):
        host_page[:] = 255
        backend.begin_page()
        backend.upload_async(pages, host_page)
        backend.record_stroke_batch(params, strokes)
        backend.wait_page(backend.submit_page())
        backend.wait_download(backend.download_async(pages, host_page))
    e2e_s = time.perf_counter() - t
    e2e = {"value": page.pixels * world * e2e_steps / e2e_s / 1e6, "unit": "Mpixel/s",
           "h2d_bytes_per_step": int(page.pts.nbytes + page.flags.nbytes + page.path_pt_off.nbytes + 3 * page.n_paths
                                     + host_page.nbytes),
           "d2h_bytes_per_step": int(host_page.nbytes), "steps": e2e_steps,
           "api": "rrb_record_stroke_batch (C ABI) with the page uploaded from and read back to pinned host memory"}
    got = np.empty(page.arena_bytes, np.uint8)
    backend.wait_download(backend.download_async(pages, got))
    cpu = bit_exact = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        import rr_oracle
        rr_oracle.build()
        ref = page.blank_arena()
        t0 = time.perf_counter()
        ost = rr_oracle.render_scene_paint(page, ref, page.strokes)
        secs = time.perf_counter() - t0
        bit_exact = bool(np.array_equal(ref, got) and np.array_equal(ref, np.asarray(host_page)))
        cpu = {"value": page.pixels / secs / 1e6, "unit": "Mpixel/s", "cores": 1, "kind": "port",
               "sample": "the whole page (all paths), 1 host thread, C++ restatement of the reference's stroke() "
                         "and fill path", "seconds": secs, "unpinned_tie_rows": ost["unpinned_tie_rows"]}
    peak, peak_kind = measured_peak()
    dom = max(stage_ms, key=stage_ms.get) if stage_ms else None
    roofline = None
    alg = {"composite": 2 * page.pixels + 4 * stats["spans"] + 8 * stats["row_groups"],
           "rows": 32 * stats["segments"] + 8 * stats["row_groups"] + 4 * stats["spans"]}
    if dom in alg:
        waves = max(1, int(stats.get("waves", 1)))
        dur = stage_ms[dom] / waves / 1e3
        ach = alg[dom] / waves / dur / 1e9
        roofline = {"kernel": dom, "bound": "hbm", "achieved": ach, "peak": peak, "unit": "GB/s", "frac": ach / peak,
                    "traffic": None, "peak_source": peak_kind, "algorithmic_bytes_per_launch": alg[dom] / waves,
                    "launch_ms": dur * 1e3}
    backend.free_device(pages)
    backend.close()
    if rank == 0:
        p50, p99 = (float(np.percentile(step_ms, q)) for q in (50, 99))
        print(json.dumps({
            "metric": METRIC, "value": value, "unit": "Mpixel/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "u8",
            "data": "synthetic (seeded stroke page, seed 0; no public dataset for this path)",
            "config": {"workload": page.description, "paths": page.n_paths, "pages": 1, "rowmap": "documented",
                       "l2": "outlines and edge records larger than L2",
                       "parallelism": f"replicas x{world} (the page on every GPU)"},
            "device_ms_per_step": device_ms, "host_ms_per_step": stats["host_ns"] / 1e6,
            "outline_segments_per_step": stats["segments"],
            "p50_page_ms": p50, "p99_page_ms": p99, "bit_exact": bit_exact, "roofline": roofline,
            "stages_ms": stage_ms, "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": launches, "clocks": clk,
        }), flush=True)


def run_fill_ops(args, rank, world):
    """The reference's coverage operators (record_aa_fill / record_tile_fill)
    on the reference's own benchmark shapes (threshold_bench: a w x h square
    for 2^8 .. 2^22 pixels) and on glyph outlines (a 1024 x 1024 coverage
    window holding the flattened outlines of 48 glyphs). GPU time is the
    kernel with segments resident (CUDA events on the backend stream); e2e
    adds the segment upload and the coverage download; the CPU baseline is
    aa_fill_cpu (the oracle), 1 thread, on a bounded sample of rows."""
    if rank != 0:
        return
    import torch
    import rr_oracle
    import rrb
    rr_oracle.build()
    be = rrb.B200Backend(0)
    stream = torch.cuda.ExternalStream(be.stream, device=torch.device("cuda", 0))
    flush = torch.empty(FLUSH_BYTES, dtype=torch.uint8, device="cuda:0")

    def outline_segs(n_glyphs, size):
        sc = rrb.Scene(1, 7, n_paths=n_glyphs, page_w=size, page_h=size)
        out = []
        for i in range(sc.n_paths):
            a, b = int(sc.path_pt_off[i]), int(sc.path_pt_off[i + 1])
            for g in rr_oracle.xpath_new(sc.pts[a:b], sc.flags[a:b]):
                out.append((g.x1, g.y1, g.x0, g.y0) if g.flags & 0x04 else (g.x0, g.y0, g.x1, g.y1))
        return np.asarray(out, np.float32).reshape(-1, 4)

    def square(w, h):
        return np.array([[0, 0, w, 0], [w, 0, w, h], [w, h, 0, h], [0, h, 0, 0]], np.float32)

    def measure(segs, w, h, op, reps):
        sb = be.alloc_device(max(16, segs.nbytes))
        cb = be.alloc_device(w * h)
        be.upload_async(sb, segs.view(np.uint8).reshape(-1))

        def run():
            be.begin_page()
            if op == "aa_fill":
                be.record_aa_fill(sb, len(segs), cb, w, h, 0)
            else:
                be.record_tile_fill_segs(sb, len(segs), cb, w, h, 0)
            be.wait_page(be.submit_page())

        run()
        # These inputs fit in L2: every timed call starts after an L2 flush,
        # outside its events.
        evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(reps)]
        torch.cuda.synchronize()
        for k, (e0, e1) in enumerate(evs):
            with torch.cuda.stream(stream):
                flush.fill_(k & 0xff)
            e0.record(stream)
            run()
            e1.record(stream)
        torch.cuda.synchronize()
        ms = sum(e0.elapsed_time(e1) for e0, e1 in evs) / reps
        host = np.empty(w * h, np.uint8)
        t = time.perf_counter()
        for _ in range(reps):
            be.upload_async(sb, segs.view(np.uint8).reshape(-1))
            run()
            be.wait_download(be.download_async(cb, host))
        e2e_ms = (time.perf_counter() - t) * 1e3 / reps
        exp_rows = min(h, max(1, 2_000_000 // max(1, w * len(segs))))  # bounded CPU sample
        t = time.perf_counter()
        exp = rr_oracle.aa_fill_cpu(segs, 0.0, 0.0, w, exp_rows, False)
        cpu_s = time.perf_counter() - t
        same = bool(np.array_equal(exp.ravel(), host[: w * exp_rows])) if op == "aa_fill" else None
        be.free_device(sb)
        be.free_device(cb)
        return {"pixels": w * h, "segments": len(segs), "gpu_ms": ms, "gpu_mpixel_s": w * h / ms / 1e3,
                "e2e_ms": e2e_ms, "cpu_mpixel_s": w * exp_rows / cpu_s / 1e6, "cpu_sample_rows": exp_rows,
                "bit_exact_sample": same}

    out = {"aa_fill": {}, "tile_fill_segs": {}}
    for e in range(8, 23, 2):
        n = 1 << e
        w = int(np.ceil(np.sqrt(n)))
        h = (n + w - 1) // w
        for op in out:
            out[op][f"square_{n}px"] = measure(square(w, h), w, h, op, args.steps)
    segs = outline_segs(48, 1024)
    for op in out:
        out[op]["glyph_outlines_1024"] = measure(segs, 1024, 1024, op, args.steps)
    head = out["aa_fill"]["glyph_outlines_1024"]
    line = {"metric": "aa_fill coverage Mpixel/s (reference operator, 64 samples/pixel)", "unit": "Mpixel/s",
            "value": head["gpu_mpixel_s"], "higher_is_better": True, "n_gpus": 1, "steps": args.steps,
            "dtype": "f32", "data": "synthetic (seeded)",
            "config": {"workload": "48 glyph outlines flattened at 0.1 in a 1024x1024 coverage window; "
                                   "plus the reference threshold_bench squares 2^8..2^22 px",
                       "l2": f"L2 flushed before every timed call ({FLUSH_BYTES >> 20} MB written)"},
            "cpu_baseline": {"value": head["cpu_mpixel_s"], "unit": "Mpixel/s", "cores": 1, "kind": "port",
                             "sample": f"aa_fill_cpu on the first {head['cpu_sample_rows']} rows"},
            "ops": out}
    print(json.dumps(line), flush=True)
    be.close()


SERVING_POOL = 128  # requests 0..127 render the pages pinned in tests/golden/serving_request_digests.json


def request_pool(rrb, n):
    """The pages serving requests 0..n-1 ask for: request r is one page of the
    mixed-page generator seeded by its id (kind 2, seed r, one page). Returns
    [(params, scene kept alive, page bytes, pinned SHA-256 or None)]."""
    pinned = {}
    path = ROOT / "tests" / "golden" / "serving_request_digests.json"
    if path.exists():
        pinned = {r["request"]: r["page_sha256"] for r in json.loads(path.read_text())["records"]}
    out = []
    for r in range(n):
        sc = rrb.Scene(kind=2, seed=r, n_pages=1)
        sc.view.pages = None
        out.append((sc.view, sc, int(sc.page_width[0]) * int(sc.page_height[0]), pinned.get(r)))
    return out


def serve_rates(srv, reqs, rates, n_req, outs, seed=0):
    """Poisson arrivals at each rate, request i rendering pool page i mod len(pool)
    into outs[i mod len(pool)] (at most len(pool) requests per rate, so no two
    requests in flight share a buffer); latency percentiles of the completed
    requests and the number whose page equals the oracle's pinned digest."""
    assert n_req <= len(reqs)
    import hashlib
    rng = np.random.default_rng(seed)
    out = []
    for rate in rates:
        gaps = rng.exponential(1.0 / rate, n_req)
        tickets = []
        t0 = time.perf_counter()
        due = t0
        for i in range(n_req):
            due += gaps[i]
            dt = due - time.perf_counter()
            if dt > 0:
                time.sleep(dt)
            p, k, n, _ = reqs[i % len(reqs)]
            page = outs[i % len(reqs)]
            page.fill(0)
            tickets.append((srv.submit(p, page, keep=k), page, i % len(reqs)))
        res, exact, checked = [], 0, 0
        for t, page, r in tickets:
            res.append(srv.wait(t))
        wall = time.perf_counter() - t0
        for t, page, r in tickets:
            d = reqs[r][3]
            if d is not None:
                checked += 1
                exact += hashlib.sha256(page.tobytes()).hexdigest() == d
        lat = [x["latency_ns"] / 1e6 for x in res]
        px = sum(reqs[i % len(reqs)][2] for i in range(n_req))
        out.append({"rate_pages_s": rate, "requests": n_req, "completed_pages_s": n_req / wall,
                    "mpixel_s": px / wall / 1e6, "p50_ms": float(np.percentile(lat, 50)),
                    "p95_ms": float(np.percentile(lat, 95)), "p99_ms": float(np.percentile(lat, 99)),
                    "mean_ms": float(np.mean(lat)), "bit_exact_requests": f"{exact}/{checked}"})
    return out


def run_serving(args, rank, world):
    """Poisson page-render requests against the continuous-batching server
    under three scheduling policies: arrival order with the default 64x16
    tile; the autotuner's table (tile shape per batch from page size and edge
    density, arrival order); the learned cost model (tile shape per batch and
    shortest-predicted-first admission, falling back to the table). Every
    request's page is checked against the oracle's pinned digest."""
    if rank != 0:
        return
    import rrb
    from rrb.autotune import CostModel
    reqs = request_pool(rrb, min(args.requests, SERVING_POOL))
    rates = [float(r) for r in args.rates.split(",")]
    # Each pool page's result buffer, page-locked (as a serving client would
    # keep its result buffers) and reused by every request for that page.
    pin_ctx = rrb.B200Backend(0)
    pin_bufs = [pin_ctx.alloc_host_pinned(n) for _, _, n, _ in reqs]
    pin_outs = [b.array()[:n] for b, (_, _, n, _) in zip(pin_bufs, reqs)]
    model_path = Path(args.cost_model)
    model = CostModel.load(model_path) if model_path.exists() else None
    policies = ["arrival_order"] + (["autotuner_table", "cost_model"] if model is not None else [])
    report = {}
    for policy in policies:
        with rrb.Server(workers=args.workers, mem_budget=args.mem_budget_gb << 30, max_batch_pages=64) as srv:
            if policy == "cost_model":
                srv.set_cost_model(model)
            elif policy == "autotuner_table":
                srv.set_cost_model(table=model.table, shortest_first=False)
            # warm-up: every distinct page, queued at once (scratch reaches its working size)
            warm = [srv.submit(p, o, keep=k) for (p, k, n, _), o in zip(reqs, pin_outs)]
            for t in warm:
                srv.wait(t)
            # The same pages queued at once again, timed: the rate of full batches
            # with no arrival gaps, which the Poisson rates are measured against.
            outs = pin_outs
            for o in outs:
                o.fill(0)
            t0 = time.perf_counter()
            burst = [srv.submit(p, o, keep=k) for (p, k, n, _), o in zip(reqs, outs)]
            for t in burst:
                srv.wait(t)
            wall = time.perf_counter() - t0
            px = sum(n for _, _, n, _ in reqs)
            import hashlib
            exact = sum(d is not None and hashlib.sha256(o.tobytes()).hexdigest() == d
                        for (_, _, _, d), o in zip(reqs, outs))
            rep = {"burst": {"pages": len(reqs), "pages_s": len(reqs) / wall, "mpixel_s": px / wall / 1e6,
                             "bit_exact_requests": f"{exact}/{sum(d is not None for *_, d in reqs)}"},
                   "rates": serve_rates(srv, reqs, rates, min(args.requests, len(reqs)), pin_outs), "server_stats": srv.stats()}
            for r in rep["rates"]:
                r["vs_burst_pages_s"] = r["completed_pages_s"] / rep["burst"]["pages_s"]
            report[policy] = rep
    best = report.get("cost_model", report["arrival_order"])
    line = {"metric": "p99 page latency under Poisson load (continuous batching)", "unit": "ms",
            "value": best["rates"][-1]["p99_ms"], "higher_is_better": False, "n_gpus": 1,
            "config": {"workload": f"request r = one page of the mixed-page generator seeded by r (kind 2, seed r); "
                                   f"requests cycle through the {len(reqs)} pages pinned by the oracle",
                       "workers": args.workers, "mem_budget_gb": args.mem_budget_gb,
                       "cost_model": str(model_path) if model is not None else None},
            "serving": report}
    holdout = ROOT / "tests" / "golden" / "cost_model_holdout.npz"
    if model is not None and holdout.exists():
        # Device time of the held-out pages under each choice of tile shape
        # (the sweep's measured times): MAPE of the model's predictions and its
        # choices against the fixed default and the autotuner table.
        from rrb.autotune import evaluate
        d = np.load(holdout)
        line["cost_model_holdout"] = {k: (float(v) if isinstance(v, (float, np.floating)) else v)
                                      for k, v in evaluate(model, d["X"], d["ms"]).items()}
    if model is not None:
        line["model_vs_table"] = {r_m["rate_pages_s"]: {"mpixel_s": r_m["mpixel_s"] / max(1e-9, r_t["mpixel_s"]),
                                                       "p99": r_m["p99_ms"] / max(1e-9, r_t["p99_ms"])}
                                  for r_m, r_t in zip(report["cost_model"]["rates"], report["autotuner_table"]["rates"])}
    print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["rrb", "reference"], default="rrb")
    ap.add_argument("--workload", choices=list(WORKLOADS) + ["fill_ops", "strokes"], default="mixed")
    ap.add_argument("--rowmap", type=int, default=0)
    ap.add_argument("--plain-sample", type=int, default=2000)
    ap.add_argument("--e2e-steps", type=int, default=3)
    ap.add_argument("--ref-threads", type=int, default=0, help="host threads of the CPU reference (0: every core)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--paths", type=int, default=0, help="override the path count (profiling runs)")
    ap.add_argument("--tile", default="", help="WxH, a fixed tile shape instead of the trials (profiling runs)")
    ap.add_argument("--wave-points", type=int, default=0, help="path points per wave of pages (0: the library's)")
    ap.add_argument("--pages", default="", help="a:b, render only pages [a, b) of the batch (profiling runs)")
    ap.add_argument("--serving", action="store_true", help="Poisson request load against the server")
    ap.add_argument("--rates", default="50,200,1000,2000")
    ap.add_argument("--requests", type=int, default=128)
    ap.add_argument("--workers", type=int, default=2)
    ap.add_argument("--mem-budget-gb", type=int, default=60)
    ap.add_argument("--cost-model", default=str(ROOT / "pdf-raster_b200" / "rrb" / "cost_model.npz"))
    args = ap.parse_args()
    rank, local, world = dist_env()
    if args.serving:
        run_serving(args, rank, world)
    elif args.impl == "reference":
        run_reference(args, rank, world)
    elif args.workload == "fill_ops":
        run_fill_ops(args, rank, world)
    elif args.workload == "strokes":
        run_strokes(args, rank, local, world)
    else:
        run_rrb(args, rank, local, world)


if __name__ == "__main__":
    main()
