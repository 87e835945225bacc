"""Benchmark: volume-render Gsamples/s on the AMR perspective workload, with
the batched and served forms against the plain single-view kernel.

Workload (one "step" = one full render of one view): a 128^3 blob root grid
refined by factor 2 to 3 levels in 16^3 patches, decomposed by the kd-tree
into ~1100 bricks, rendered by VolumeRenderSampler through a perspective lens
at 1024x1024 with an 8-layer ColorTransferFunction, 1 sample per cell.
A sample is one trilinear sample + transfer-function evaluation + update
(= one cell visit at n_samples=1), counted exactly by the kernel.

Arms:
* default (``--impl ours``): ``value`` = samples / device time of the render
  launch with bricks, transfer function, kd order and pixel rectangles
  resident in HBM (L2 flushed between steps); ``e2e`` = the same render
  through the drop-in ``VolumeRenderSampler`` call surface from host numpy
  arrays to the host image, copies included.  The same line carries
  ``batched`` (64 views of mixed sizes and samplers: one CUDA-graph replay
  of the persistent launches against 64 plain launches), ``served`` (Poisson
  request streams through the render server against the same requests
  rendered one plain launch at a time), ``cpu_baseline`` (yt's compiled
  sampler on the host cores, the full frame) and ``accuracy`` (the GPU
  image against the float64 oracle's, the full frame).
* ``--impl reference``: yt's own compiled sampler on the host cores, the full
  frame per step, with the bricks and their order built by the reference's
  own compiled kd-tree and vertex centring (nothing of this package's native
  code is loaded).
"""
from __future__ import annotations

import argparse
import ctypes
import json
import os
import subprocess
import sys
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

BYTES_PER_SAMPLE = 32   # 8 float32 vertex values gathered per trilinear sample
BYTES_PER_RAY = 64      # float64 RGBA read + written per ray


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=100)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--res", type=int, default=1024)
    ap.add_argument("--root", type=int, default=128)
    ap.add_argument("--levels", type=int, default=3)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--workload", default="amr_vr",
                    choices=["amr_vr", "uniform", "multiview", "projection", "serve", "prep", "octree", "offaxis"],
                    help="amr_vr (default, the headline frame); the others print their own line")
    ap.add_argument("--tile-shape", type=int, default=-1, help="-1: from the autotuning table")
    ap.add_argument("--n-requests", type=int, default=2000, help="requests per rate (--workload serve)")
    ap.add_argument("--rates", default="50,100,200,500,1000,2000")
    ap.add_argument("--audit", type=int, default=20, help="requests re-rendered by the oracle (--workload serve)")
    ap.add_argument("--no-batched", action="store_true", help="default line without the batched record")
    ap.add_argument("--no-served", action="store_true", help="default line without the served record")
    ap.add_argument("--served-requests", type=int, default=200, help="requests per rate in the default line")
    ap.add_argument("--max-batch", type=int, default=64, help="requests per served batch (--workload serve)")
    ap.add_argument("--slots", type=int, default=4, help="streams of the render server (--workload serve)")
    ap.add_argument("--batch-pixels", type=int, default=512 * 512,
                    help="requests under this many pixels share a batch launch (--workload serve)")
    return ap.parse_args()


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), "measured"
    return 6800.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    def __init__(self, index=0):
        self.proc = None
        self.index = index
        self.path = Path("/tmp") / f"ytgb_clocks_{os.getpid()}.csv"

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.index}",
                 "--query-gpu=clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
                 "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
                 "clocks_event_reasons.sw_power_cap", "--format=csv,noheader,nounits", "-lms", "20"],
                stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except (FileNotFoundError, OSError):
            self.proc = None
        return self

    def __exit__(self, *a):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        if not self.path.exists():
            return None
        rows = []
        for line in self.path.read_text().splitlines():
            parts = [x.strip() for x in line.split(",")]
            if len(parts) < 7:
                continue
            try:
                rows.append((float(parts[0]), float(parts[1]), parts[3:7]))
            except ValueError:
                continue
        self.path.unlink(missing_ok=True)
        if not rows:
            return None
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for _, _, r in rows for i, v in enumerate(r) if v.lower() == "active"})
        return {"sm_mhz": float(np.median([r[0] for r in rows])), "sm_max_mhz": max(r[1] for r in rows),
                "reasons": reasons, "samples": len(rows)}


def reference_pkg():
    """yt's compiled package as timed (yt's own compiler flags) where built,
    else the -ffp-contract=off build."""
    from oracle import ref_workload as rw

    return rw.ref_pkg(True) or rw.ref_pkg(False) or (ROOT / "oracle" / "_ref" / "pkg")


def build_workload(args):
    from yt_gb300 import workloads

    t = time.time()
    w = workloads.amr_vr(root=args.root, levels=args.levels, res=args.res)
    return w, time.time() - t


def config_dict(args, n_bricks, n_grids):
    """The workload's description, identical in both arms."""
    return {"workload": "amr_vr: 128^3 blob root + 3 factor-2 levels (16^3 patches), kd bricks, "
                        "VolumeRenderSampler, perspective lens, 8-layer ColorTransferFunction, 1 sample/cell",
            "resolution": args.res, "bricks": n_bricks, "grids": n_grids, "root": args.root, "levels": args.levels,
            "l2": "flushed between steps (256 MiB write)"}


def reference_frame(args, res=None):
    """The benchmark frame built by the reference itself (its compiled kd-tree
    and vertex centring), or by the restatements where it is not built."""
    from oracle import ref_workload as rw

    return rw.amr_frame(root=args.root, levels=args.levels, res=res or args.res, timed=True, allow_port=True)


def single_thread_figure(frame, res):
    """yt's sampler on one host thread over a bounded sample of the frame:
    the same camera at ``res``^2, all bricks."""
    from oracle import ref_workload as rw

    small = frame.with_resolution(res)
    _, samples = rw.oracle_render(small, os.cpu_count() or 1)
    dt, _ = rw.render(small, 1)
    return {"value": samples / dt / 1e9, "unit": "Gsamples/s", "cores": 1, "seconds": dt,
            "sample": f"the same camera at {res}x{res} ({samples} samples), all {len(frame.bricks)} bricks"}


def run_reference(args):
    """yt's compiled sampler over the full frame on all host threads, with
    the bricks and order built by the reference (rank 0 only)."""
    rank, world, _ = dist_env()
    if rank != 0:
        return
    from oracle import ref_workload as rw

    threads = os.cpu_count() or 1
    frame = reference_frame(args)
    pgs = frame.partitioned_grids()
    _, samples = rw.oracle_render(frame, threads)   # the visit count (the sampler reports none)
    secs = []
    for i in range(args.warmup + args.steps):
        dt, _ = rw.render(frame, threads, pgs)
        if i >= args.warmup:
            secs.append(dt)
    sec = float(np.mean(secs))
    v = samples / sec / 1e9
    one = single_thread_figure(frame, max(64, args.res // 4))
    sample = (f"the full frame every step: {args.res}x{args.res}, all {len(frame.bricks)} bricks, {samples} samples; "
              "sampler calls only (bricks prepared beforehand, as render_source.py:594-596 times nothing else)")
    line = {"impl": "reference", "metric": "Gsamples/s", "value": v, "unit": "Gsamples/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * sec,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": config_dict(args, len(frame.bricks), frame.n_grids),
            "cpu_baseline": {"value": v, "unit": "Gsamples/s", "cores": threads, "kind": frame.kind,
                             "sample": sample, "single_thread": one},
            "e2e": {"value": v, "unit": "Gsamples/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "latency_ms": {"p50": 1e3 * float(np.percentile(secs, 50)), "p99": 1e3 * float(np.percentile(secs, 99))},
            "bricks_built_by": "reference amr_kdtools.Node + ghost_zone_interpolate" if frame.kind == "reference"
            else "oracle restatements (reference not built)",
            "native_libraries": rw.loaded_native_libraries(), "build_seconds": frame.build_seconds}
    print(json.dumps(line), flush=True)


def cpu_leg(args, r, cam, samples_gpu):
    """The CPU baseline and accuracy of the default line: yt's compiled
    sampler (all host threads) over the full frame built by the reference,
    its single-thread figure on a bounded sample, and the GPU image of the
    full frame against the float64 oracle's image of the reference-built
    frame."""
    from oracle import ref_workload as rw
    from yt_gb300 import _lib
    from yt_gb300.render import relative_error

    threads = os.cpu_count() or 1
    frame = reference_frame(args)
    dt, _ = rw.render(frame, threads)
    exact, samples = rw.oracle_render(frame, threads)
    img_g = r.render(cam, kind=_lib.VOLUME_RENDER).cpu().numpy()
    r.check()
    mx, rms = relative_error(img_g, exact, channels=(0, 1, 2))
    base = {"value": samples / dt / 1e9, "unit": "Gsamples/s", "cores": threads, "kind": frame.kind,
            "seconds": dt,
            "sample": f"the full frame ({args.res}x{args.res}, all {len(frame.bricks)} bricks, {samples} samples), "
                      "once; bricks and order built by the reference",
            "single_thread": single_thread_figure(frame, max(64, args.res // 4))}
    acc = {"max_rel_err": mx, "rms_rel_err": rms, "tau": 1e-6,
           "vs": f"float64 oracle (-ffp-contract=off, pinned bit for bit to yt's sampler) of the full "
                 f"{args.res}x{args.res} frame built by the reference",
           "samples_equal_oracle": int(samples) == int(samples_gpu)}
    return base, acc


def traffic_from_profile():
    p = ROOT / "profiles" / "traffic.json"
    if p.exists():
        try:
            return json.loads(p.read_text())
        except ValueError:
            return None
    return None


def run_ours(args):
    import torch

    from yt_gb300 import _lib
    from yt_gb300.render import Renderer, relative_error

    rank, world, local = dist_env()
    if world > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl")
    dev = torch.device("cuda", local if world > 1 else 0)
    torch.cuda.set_device(dev)
    w, t_build = build_workload(args)
    cam = w.views[0].camera
    r = Renderer(w.bricks, w.tf, device=dev, kdtree=w.kdtree)
    order = r.order(cam)
    view, ppos, pdir = r.view_args(cam)
    px_pos = torch.from_numpy(ppos).to(dev) if ppos is not None else None
    px_dir = torch.from_numpy(pdir).to(dev) if pdir is not None else None
    rects = r.bricks.rects(view, order)
    nx, ny = cam.resolution
    image = torch.zeros((nx, ny, 4), dtype=torch.float64, device=dev)
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device=dev)  # 256 MiB > L2
    stream = torch.cuda.current_stream(dev)
    from yt_gb300.autotune import tile_shape_for
    from yt_gb300.volume import render as vrender
    from yt_gb300.volume import render_tables

    # the rectangles and order stay resident, like the bricks and the TF
    tables = render_tables(r.bricks, view, order, rects)

    tile_shape = args.tile_shape if args.tile_shape >= 0 else tile_shape_for(
        _lib.VOLUME_RENDER, bool(r.packed.header.ctf_fast), view.lens)
    tflags = tile_shape << _lib.FLAG_TILE_SHIFT
    keep = []

    def step():
        image.zero_()
        vrender(r.bricks, view, order, _lib.VOLUME_RENDER, image, tf=r.packed, counters=r.counters, error=r.error,
                px_pos=px_pos, px_dir=px_dir, stream=stream, tables=tables, keep=keep, flags=tflags)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    r.check()
    keep.clear()
    r.counters.zero_()
    times = []
    launches = 0
    need = ctypes.c_int64()
    _lib.check(_lib.lib().ytgb_render_scratch(ctypes.byref(view), order.size, ctypes.byref(need)), "scratch")
    per_render = 3 if need.value else 1  # the render; the order of its tiles (their costs, the sort)
    if world > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    clocks = ClockSampler(dev.index)
    with clocks:
        t_wall0 = time.perf_counter()
        for _ in range(args.steps):
            flush.fill_(1.0)
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            image.zero_()
            e0.record(stream)
            vrender(r.bricks, view, order, _lib.VOLUME_RENDER, image, tf=r.packed, counters=r.counters,
                    error=r.error, px_pos=px_pos, px_dir=px_dir, stream=stream, tables=tables, keep=keep,
                    flags=tflags)
            e1.record(stream)
            launches += per_render
            times.append((e0, e1))
        torch.cuda.synchronize()
        t_wall = time.perf_counter() - t_wall0
    if world > 1:
        torch.distributed.barrier()
    r.check()
    keep.clear()
    ms = np.array([a.elapsed_time(b) for a, b in times])
    samples_total = int(r.counters[0].item())
    rays = int(r.counters[2].item()) // max(args.steps, 1)
    samples_step = samples_total // args.steps
    walks_step = int(r.counters[1].item()) // max(args.steps, 1)
    guarded_step = int(r.counters[3].item()) // max(args.steps, 1)
    t_total = float(ms.sum()) / 1e3
    if world > 1:
        import torch.distributed as dist

        tt = torch.tensor([t_total], device=dev)
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        t_total = float(tt.item())
    value = samples_total * world / t_total / 1e9
    hbm, peak_kind = peaks()
    alg_bytes = samples_step * BYTES_PER_SAMPLE + rays * BYTES_PER_RAY
    achieved = alg_bytes / (float(ms.mean()) / 1e3) / 1e9
    prof = traffic_from_profile() or {}
    traffic = prof.get("amr_vr_dram_bytes_per_launch")

    # e2e through the drop-in sampler API: host numpy bricks -> host image
    e2e = None
    if not args.no_e2e:
        from yt_gb300.image_samplers import VolumeRenderSampler
        from yt_gb300.partitioned_grid import PartitionedGrid

        p = cam.sampler_params()
        pgs = [PartitionedGrid(0, *w.bricks[k]) for k in order]
        ets = []
        h2d = d2h = 0
        for i in range(args.warmup + max(3, args.steps // 4)):
            img_h = np.zeros((nx, ny, 4))
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            s = VolumeRenderSampler(np.atleast_3d(p["vp_pos"]), np.atleast_3d(p["vp_dir"]), p["center"],
                                    p["bounds"], img_h, p["x_vec"], p["y_vec"], p["width"], "KDTree", w.tf, 1,
                                    lens_type=p["lens_type"], camera_data=p["camera_data"],
                                    zbuffer=np.ones((nx, ny)))
            for pg in pgs:
                s(pg, num_threads=0)
            out = s.aimage
            t1 = time.perf_counter()
            if i >= args.warmup:
                ets.append(t1 - t0)
        h2d = s.last_h2d_bytes
        d2h = s.last_d2h_bytes
        e2e_v = samples_step / float(np.median(ets)) / 1e9
        e2e = {"value": e2e_v, "unit": "Gsamples/s", "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": int(d2h),
               "ms_per_step": 1e3 * float(np.median(ets)), "path": "VolumeRenderSampler(...)(pg) per brick, aimage",
               "breakdown_ms": {k: round(v, 3) for k, v in s.last_timings.items()}}
        del out

    line = {"metric": "Gsamples/s", "value": value, "unit": "Gsamples/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": float(ms.mean()), "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32 sampling / f64 traversal", "data": "synthetic",
            "config": config_dict(args, len(w.bricks), w.info.get("grids")), "tile_shape": tile_shape,
            "latency_ms": {"p50": float(np.percentile(ms, 50)), "p99": float(np.percentile(ms, 99))},
            "samples_per_step": samples_step, "rays_per_step": rays, "brick_walks_per_step": walks_step,
            "out_of_brick_cells_per_step": guarded_step,
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": hbm, "unit": "GB/s",
                         "frac": achieved / hbm, "traffic": traffic,
                         "peak_source": peak_kind + " hbm_gbs (MEASURED_PEAKS.json)" if peak_kind == "measured"
                         else "fallback 6800 GB/s",
                         "algorithmic_bytes_per_launch": int(alg_bytes),
                         "model": f"{BYTES_PER_SAMPLE} B/sample + {BYTES_PER_RAY} B/ray"},
            "gpu_launches": launches, "e2e": e2e, "clocks": clocks.summary(), "build_seconds": t_build}

    solo = rank == 0 and world == 1
    if solo and not args.no_cpu_baseline:
        line["cpu_baseline"], line["accuracy"] = cpu_leg(args, r, cam, samples_step)
    if solo and not args.no_batched:
        line["batched"] = multiview_record(dev, steps=args.steps, warmup=args.warmup, tile_shape=args.tile_shape)
    if solo and not args.no_served:
        line["served"] = serve_record(dev, n_requests=args.served_requests,
                                      rates=[float(x) for x in args.rates.split(",")], audit=None,
                                      amr=(w.bricks, w.kdtree))
    if rank == 0:
        print(json.dumps(line), flush=True)
    if world > 1:
        import torch.distributed as dist

        dist.destroy_process_group()


def _timed_events(fn, steps, stream):
    import torch

    ts = []
    for _ in range(steps):
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        fn()
        e1.record(stream)
        ts.append((e0, e1))
    torch.cuda.synchronize()
    return np.array([a.elapsed_time(b) for a, b in ts])


def _audit_view(renderer, bricks, kd, camera, kind, image, tf=None, threads=None):
    """Max relative error of one rendered view against the float64 oracle."""
    from oracle import cpu as ocpu
    from yt_gb300 import _lib
    from yt_gb300.render import relative_error

    p = camera.sampler_params()
    name = {_lib.VOLUME_RENDER: "volume_render", _lib.PROJECTION: "projection", _lib.MIP: "mip",
            _lib.INTERPOLATED_PROJECTION: "interpolated_projection"}[kind]
    s = ocpu.OracleSampler(name, p["vp_pos"], p["vp_dir"], p["center"], p["bounds"], p["image"], p["x_vec"],
                           p["y_vec"], p["width"], lens_type=p["lens_type"], camera_data=p["camera_data"],
                           tf=tf if kind == _lib.VOLUME_RENDER else None)
    order = kd.viewpoint_order(camera.viewpoint) if kd is not None else None
    s.render(ocpu.OracleBricks(bricks), order, num_threads=threads or os.cpu_count() or 1)
    chans = (0, 1, 2) if kind in (_lib.VOLUME_RENDER, _lib.INTERPOLATED_PROJECTION) else (0,)
    return relative_error(image, p["image"], channels=chans)[0]


_MULTIVIEW = {}


def multiview_data():
    """The 64-view dataset (built once per process): a 4-level AMR volume,
    log10 for volume rendering and linear for interpolated projection."""
    if "w" not in _MULTIVIEW:
        from yt_gb300 import workloads
        from yt_gb300.amr_kdtree import AMRKDTree

        t0 = time.time()
        w = workloads.multiview()
        lin = AMRKDTree(w.kdtree.grids, log_field=False)
        _MULTIVIEW.update(w=w, lin=lin, lin_bricks=lin.bricks(), seconds=time.time() - t0)
    return _MULTIVIEW


def multiview_record(dev, steps, warmup, tile_shape=-1):
    """64 cameras on a Fibonacci sphere over a 4-level AMR volume (~3700
    bricks, 8^3-32^3), image sizes from {128,256,512,1024}^2, half volume
    rendering and half interpolated projection: 64 plain single-view
    launches (inputs prepared) against one CUDA-graph replay of the batched
    persistent launches, L2 flushed before each; both count their samples.
    Two views of the batch are audited against the float64 oracle."""
    import torch

    from yt_gb300 import _lib
    from yt_gb300.autotune import tile_shape_for
    from yt_gb300.batch import Batch, Job
    from yt_gb300.render import Renderer
    from yt_gb300.volume import render as vrender

    mv = multiview_data()
    w, lin = mv["w"], mv["lin"]
    r_vr = Renderer(w.bricks, w.tf, device=dev, kdtree=w.kdtree)
    r_pj = Renderer(mv["lin_bricks"], None, device=dev, kdtree=lin)
    ts = tile_shape if tile_shape >= 0 else None
    jobs = [Job(r_vr if v.kind == _lib.VOLUME_RENDER else r_pj, v.camera, v.kind) for v in w.views]
    stream = torch.cuda.current_stream(dev)
    prepared = []
    for j in jobs:
        rr = j.renderer
        view = j.camera.device_view()
        order = rr.order(j.camera)
        rects = rr.bricks.rects(view, order)
        img = torch.zeros((*j.camera.resolution, 4), dtype=torch.float64, device=dev)
        ctf = bool(j.kind == _lib.VOLUME_RENDER and rr.packed.header.ctf_fast)
        vts = ts if ts is not None else tile_shape_for(j.kind, ctf, view.lens)
        prepared.append((rr, view, order, rects, img, j.kind, vts))
    keep = []

    def plain():
        for rr, view, order, rects, img, kind, vts in prepared:
            img.zero_()
            vrender(rr.bricks, view, order, kind, img, tf=rr.packed if kind == _lib.VOLUME_RENDER else None,
                    counters=rr.counters, error=rr.error, stream=stream, rects=rects, keep=keep,
                    flags=vts << _lib.FLAG_TILE_SHIFT)

    b = Batch(jobs, device=dev, tile_shape=ts)
    graph = b.capture()
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device=dev)
    for _ in range(warmup):
        plain()
        graph.replay()
    torch.cuda.synchronize()
    keep.clear()
    r_vr.counters.zero_()
    r_pj.counters.zero_()
    b.counters.zero_()
    ms_plain, ms_batch = [], []
    clocks = ClockSampler(dev.index or 0)
    with clocks:
        for _ in range(steps):
            flush.fill_(1.0)
            ms_plain.append(_timed_events(plain, 1, stream)[0])
            keep.clear()
            flush.fill_(1.0)
            ms_batch.append(_timed_events(graph.replay, 1, stream)[0])
    r_vr.check()
    r_pj.check()
    b.check()
    samples_plain = int(r_vr.counters[0].item() + r_pj.counters[0].item()) // steps
    samples_batch = int(b.counters[0].item()) // steps
    walks_batch = int(b.counters[1].item()) // steps
    same_images = all(torch.equal(pimg.view(torch.int64), j.image.view(torch.int64))
                      for (_, _, _, _, pimg, _, _), j in zip(prepared, jobs))
    ms_plain, ms_batch = np.array(ms_plain), np.array(ms_batch)
    hbm, _ = peaks()
    rays = sum(int(np.prod(j.camera.resolution)) for j in jobs)
    alg = samples_batch * BYTES_PER_SAMPLE + rays * BYTES_PER_RAY

    def gbs(ms_arr):
        return alg / (float(ms_arr.mean()) / 1e3) / 1e9

    # audit: the smallest view of each sampler against the float64 oracle
    errs = []
    for kind in (_lib.VOLUME_RENDER, _lib.INTERPOLATED_PROJECTION):
        k = min((i for i, j in enumerate(jobs) if j.kind == kind), key=lambda i: np.prod(jobs[i].camera.resolution))
        j = jobs[k]
        bricks = w.bricks if kind == _lib.VOLUME_RENDER else mv["lin_bricks"]
        kd = w.kdtree if kind == _lib.VOLUME_RENDER else lin
        errs.append(_audit_view(j.renderer, bricks, kd, j.camera, kind, j.image.cpu().numpy(), tf=w.tf))
    return {"workload": "64 Fibonacci-sphere cameras, perspective, sizes {128..1024}^2, VR + interpolated "
                        "projection, 4-level AMR (64^3 root, patches 8^3-32^3)",
            "value": samples_batch / (ms_batch.mean() / 1e3) / 1e9, "unit": "Gsamples/s",
            "ms_per_step": float(ms_batch.mean()), "steps": steps,
            "latency_ms": {"p50": float(np.percentile(ms_batch, 50)), "p99": float(np.percentile(ms_batch, 99))},
            "plain": {"value": samples_plain / (ms_plain.mean() / 1e3) / 1e9, "ms_per_step": float(ms_plain.mean()),
                      "latency_ms": {"p50": float(np.percentile(ms_plain, 50)),
                                     "p99": float(np.percentile(ms_plain, 99))},
                      "launches": len(jobs), "roofline_frac": gbs(ms_plain) / hbm},
            "samples_per_step": samples_batch, "samples_match": samples_batch == samples_plain,
            "brick_walks_per_step": walks_batch,
            "images_identical_to_plain": bool(same_images),
            "launches_per_graph": len(b.groups), "work_items": b.total_tiles, "tile_shape": b.tile_shape,
            "roofline": {"bound": "hbm", "achieved": gbs(ms_batch), "peak": hbm, "unit": "GB/s",
                         "frac": gbs(ms_batch) / hbm, "model": f"{BYTES_PER_SAMPLE} B/sample + {BYTES_PER_RAY} B/ray"},
            "audit": {"views": 2, "max_rel_err": float(max(errs)), "vs": "float64 oracle, smallest view per sampler"},
            "bricks": len(w.bricks), "rays": rays, "l2": "flushed before each form's step",
            "clocks": clocks.summary(), "build_seconds": mv["seconds"]}


def run_multiview(args):
    import torch

    dev = torch.device("cuda", 0)
    rec = multiview_record(dev, args.steps, args.warmup, args.tile_shape)
    line = {"metric": "Gsamples/s", "workload": "multiview", "value": rec["value"], "unit": "Gsamples/s",
            "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "ms_per_step": rec["ms_per_step"],
            "higher_is_better": True, "batched": rec}
    print(json.dumps(line), flush=True)


def run_uniform(args):
    """The small plain case: one 64^3 blob grid as one brick, plane-parallel
    view down +z (width 1), 256^2, 4-layer ColorTransferFunction, 1 sample
    per cell.  Device time per frame (L2 flushed), the traversal trace and
    image against the float64 oracle of the frame the reference builds, and
    yt's compiled sampler on the host cores over the same frame."""
    import torch

    from oracle import ref_workload as rw
    from yt_gb300 import _lib, workloads
    from yt_gb300.render import Renderer, relative_error

    dev = torch.device("cuda", 0)
    n = args.root if args.root != 128 else 64
    res = args.res if args.res != 1024 else 256
    w = workloads.uniform_vr(n=n, res=res)
    cam = w.views[0].camera
    r = Renderer(w.bricks, w.tf, device=dev, kdtree=w.kdtree)
    img = torch.zeros((res, res, 4), dtype=torch.float64, device=dev)
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device=dev)
    stream = torch.cuda.current_stream(dev)

    def step():
        img.zero_()
        r.render(cam, kind=_lib.VOLUME_RENDER, image=img)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    r.counters.zero_()
    ms = []
    clocks = ClockSampler(0)
    with clocks:
        for _ in range(args.steps):
            flush.fill_(1.0)
            ms.append(_timed_events(step, 1, stream)[0])
    r.check()
    ms = np.array(ms)
    samples = int(r.counters[0].item()) // args.steps
    threads = os.cpu_count() or 1
    frame = rw.uniform_frame(n=n, res=res, timed=True, allow_port=True)
    dt, _ = rw.render(frame, threads)
    exact, samples_o = rw.oracle_render(frame, threads)
    mx, rms = relative_error(img.cpu().numpy(), exact, channels=(0, 1, 2))
    from oracle import cpu as ocpu

    p = frame.camera.sampler_params()
    so = ocpu.OracleSampler("volume_render", p["vp_pos"], p["vp_dir"], p["center"], p["bounds"], p["image"],
                            p["x_vec"], p["y_vec"], p["width"], lens_type=p["lens_type"],
                            camera_data=p["camera_data"], tf=frame.tf)
    h_ref, c_ref = so.trace(ocpu.OracleBricks(frame.bricks), None, num_threads=threads)
    h_gpu, c_gpu = r.trace(cam)
    hbm, _ = peaks()
    alg = samples * BYTES_PER_SAMPLE + res * res * BYTES_PER_RAY
    line = {"metric": "Gsamples/s", "workload": "uniform", "value": samples / (ms.mean() / 1e3) / 1e9,
            "unit": "Gsamples/s", "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": float(ms.mean()), "higher_is_better": True, "samples_per_step": samples,
            "latency_ms": {"p50": float(np.percentile(ms, 50)), "p99": float(np.percentile(ms, 99))},
            "roofline": {"bound": "hbm", "achieved": alg / (ms.mean() / 1e3) / 1e9, "peak": hbm, "unit": "GB/s",
                         "frac": alg / (ms.mean() / 1e3) / 1e9 / hbm},
            "cpu_baseline": {"value": samples_o / dt / 1e9, "unit": "Gsamples/s", "cores": threads,
                             "kind": frame.kind, "sample": f"the full frame ({samples_o} samples)"},
            "accuracy": {"max_rel_err": mx, "rms_rel_err": rms, "vs": "float64 oracle of the reference-built frame",
                         "trace_bit_exact": bool(np.array_equal(h_gpu, h_ref) and np.array_equal(c_gpu, c_ref)),
                         "samples_equal_oracle": samples == samples_o},
            "clocks": clocks.summary(),
            "config": {"workload": f"uniform: one {n}^3 blob brick, plane-parallel down +z, width 1, {res}^2, "
                                   "4-layer ColorTransferFunction, 1 sample/cell", "resolution": res,
                       "l2": "flushed between steps (256 MiB write)"}}
    print(json.dumps(line), flush=True)


def run_projection(args):
    """The precision study: a 512^3 float32 lognormal random field,
    ProjectionSampler and MIP at 2048^2 and three orientations, float32
    accumulation with and without compensation, each image's max and RMS
    relative error against the float64 oracle."""
    import torch

    from oracle import cpu as ocpu
    from yt_gb300 import _lib, workloads
    from yt_gb300.render import Renderer, relative_error

    dev = torch.device("cuda", 0)
    n = args.root if args.root != 128 else 512
    res = args.res if args.res != 1024 else 2048
    w = workloads.projection_study(n=n, res=res)
    field64 = [w.bricks[0][0][0].astype(np.float64)]
    r = Renderer(w.bricks, None, device=dev)
    stream = torch.cuda.current_stream(dev)
    views = []
    for v in w.views:
        for comp in (True, False):
            flags = 0 if comp else _lib.FLAG_NO_COMPENSATION
            r.counters.zero_()
            img = torch.zeros((res, res, 4), dtype=torch.float64, device=dev)

            def step():
                img.zero_()
                r.render(v.camera, kind=v.kind, image=img, flags=flags)

            for _ in range(args.warmup):
                step()
            torch.cuda.synchronize()
            r.counters.zero_()
            ms = _timed_events(step, args.steps, stream)
            samples = int(r.counters[0].item()) // args.steps
            out = img.cpu().numpy()
            entry = {"kind": "projection" if v.kind == _lib.PROJECTION else "mip",
                     "angle_deg": float(np.rad2deg(np.arctan2(v.camera.unit_vectors[2][1],
                                                              v.camera.unit_vectors[2][2]))),
                     "compensated": comp, "ms": float(ms.mean()), "Gsamples/s": samples / (ms.mean() / 1e3) / 1e9,
                     "cell_visits": samples}
            views.append((v, comp, entry, out))
    # float64 oracle per view (shared by both precisions)
    threads = os.cpu_count() or 1
    oracle_imgs = {}
    t_or = 0.0
    for v, comp, entry, out in ([] if args.no_cpu_baseline else views):
        key = id(v)
        if key not in oracle_imgs:
            p = v.camera.sampler_params()
            s = ocpu.OracleSampler("projection" if v.kind == _lib.PROJECTION else "mip", p["vp_pos"], p["vp_dir"],
                                   p["center"], p["bounds"], p["image"], p["x_vec"], p["y_vec"], p["width"],
                                   lens_type=p["lens_type"], camera_data=p["camera_data"])
            t = time.perf_counter()
            s.render(ocpu.OracleBricks([(field64, None, np.zeros(3), np.ones(3), [n, n, n])]), None,
                     num_threads=threads)
            t_or += time.perf_counter() - t
            oracle_imgs[key] = p["image"]
        mx, rms = relative_error(out, oracle_imgs[key], channels=(0,))
        entry["max_rel_err"], entry["rms_rel_err"] = mx, rms
    ents = [e for _, _, e, _ in views]
    comp_ents = [e for e in ents if e["compensated"]]
    tot_s = sum(e["cell_visits"] for e in comp_ents)
    tot_ms = sum(e["ms"] for e in comp_ents)
    hbm, _ = peaks()
    line = {"metric": "Gsamples/s", "workload": "projection", "value": tot_s / (tot_ms / 1e3) / 1e9,
            "unit": "Gsamples/s", "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": tot_ms, "higher_is_better": True, "views": ents,
            "roofline": {"bound": "hbm", "achieved": (tot_s * 4 + len(comp_ents) * res * res * 64) / (tot_ms / 1e3) / 1e9,
                         "peak": hbm, "unit": "GB/s", "model": "4 B/cell visit + 64 B/ray"},
            "cpu_oracle_seconds": t_or, "cpu_threads": threads,
            "config": {"workload": f"{n}^3 float32 lognormal GRF (P(k)~k^-3, seed 1), 2048^2 plane-parallel, "
                                   "angles 0/30/57 deg about x, ProjectionSampler + MIP", "resolution": res}}
    print(json.dumps(line), flush=True)


def serve_volumes(dev, amr=None):
    """The served form's resident data: the four volumes of the benchmark
    configurations (the 64^3 uniform blob, the 128^3-root AMR volume, the
    512^3 lognormal random field, the 4-level multi-view AMR volume) and 16
    seeded colour transfer functions."""
    from yt_gb300 import workloads

    t0 = time.time()
    w1 = workloads.uniform_vr()
    if amr is None:
        w2 = workloads.amr_vr()
        amr = (w2.bricks, w2.kdtree)
    w3 = workloads.projection_study(n=512, res=256, angles=(0.0,))
    mv = multiview_data()["w"]
    vols = {"uniform": (w1.bricks, w1.kdtree), "amr": amr, "grf": (w3.bricks, None),
            "multiview": (mv.bricks, mv.kdtree)}
    rng = np.random.default_rng(5)
    tfs = {}
    for k in range(16):
        lo, hi = sorted(rng.uniform(-0.3, 1.6, 2))
        tfs[f"tf{k}"] = workloads.color_tf((lo - 0.2, hi + 0.2), int(rng.integers(3, 9)))
    return vols, tfs, time.time() - t0


def serve_requests(vols, n, rate, seed):
    """A Poisson stream of ``n`` requests at ``rate`` per second: each names a
    volume, a transfer function, a camera on a jittered sphere and an image
    size from {256,512,1024,2048}^2 (projection or MIP for the random field,
    volume rendering otherwise)."""
    from yt_gb300 import _lib, testing
    from yt_gb300.camera import Camera
    from yt_gb300.serve import Request

    sizes = (256, 512, 1024, 2048)
    rr = np.random.default_rng(seed)
    t = 0.0
    out = []
    for i in range(n):
        t += rr.exponential(1.0 / rate)
        vol = str(rr.choice(list(vols)))
        p = testing.fibonacci_sphere(1, radius=1.0)[0] + rr.normal(0, 0.4, 3)
        res = int(rr.choice(sizes))
        if vol == "grf":
            cam = Camera(p, (0.5, 0.5, 0.5), 1.0, res, lens_type="plane-parallel")
            kind = _lib.PROJECTION if rr.random() < 0.5 else _lib.MIP
            out.append(Request(i, vol, None, cam, kind, arrival=t))
        else:
            cam = Camera(p, (0.5, 0.5, 0.5), 1.5, res, lens_type="perspective")
            out.append(Request(i, vol, f"tf{int(rr.integers(16))}", cam, _lib.VOLUME_RENDER, arrival=t))
    return out


def p99_flags(served, plain):
    """Whether the served form's p99 is at or below the plain form's, and
    whether the run tells the two apart at all (their bootstrap 95 %
    intervals overlap or not)."""
    sc, pc = served["p99_ci95_ms"], plain["p99_ci95_ms"]
    return {"served_beats_plain_p99": served["p99_ms"] <= plain["p99_ms"],
            "p99_intervals_overlap": sc[0] <= pc[1] and pc[0] <= sc[1]}


def serve_record(dev, n_requests, rates, audit=None, amr=None, max_batch=64, slots=4, batch_pixels=512 * 512):
    """Served rendering against plain: at each rate the same Poisson stream
    goes through the render server (HBM-budget admission, continuous
    batching on four streams) and through the plain form (one single-view
    launch per request on one stream); p50/p99 latency (arrival to
    completion) and Gsamples/s over the run's wall time.  Then every request
    offered at once (closed loop).  Audit: every 100th served request (1%),
    or ``audit`` of them spread evenly, re-rendered by the float64 oracle."""
    from yt_gb300 import _lib
    from yt_gb300.serve import RenderServer, latency_summary

    vols, tfs, t_build = serve_volumes(dev, amr)
    srv = RenderServer(vols, tfs, device=dev, hbm_budget=16 << 30, slots=slots, max_batch=max_batch,
                       batch_pixels=batch_pixels)
    plain_srv = RenderServer({}, {}, device=dev, hbm_budget=16 << 30, plain=True)
    plain_srv.volumes, plain_srv.tfs = srv.volumes, srv.tfs
    # warm-up: compile paths, stage tables
    srv.run(serve_requests(vols, 16, 1e6, 99), realtime=False)
    plain_srv.run(serve_requests(vols, 8, 1e6, 98), realtime=False)
    rows = []
    audit_set = []
    clocks = ClockSampler(dev.index or 0)
    with clocks:
        for k, rate in enumerate(rates):
            row = {"rate_req_s": rate}
            for label, server in (("served", srv), ("plain", plain_srv)):
                reqs = serve_requests(vols, n_requests, rate, 1000 + k)
                server.samples = 0
                server.keep_images = (lambda q: q.rid % 100 == 0) if label == "served" else False
                t = time.perf_counter()
                done = server.run(reqs, realtime=True)
                wall = time.perf_counter() - t
                row[label] = {**latency_summary(done), "Gsamples/s": server.samples / wall / 1e9, "wall_s": wall,
                              "samples": server.samples}
                if label == "served":
                    audit_set += [q for q in done if q.rid % 100 == 0]
            row.update(p99_flags(row["served"], row["plain"]))
            rows.append(row)
        closed = {}
        for label, server in (("served", srv), ("plain", plain_srv)):
            reqs = serve_requests(vols, n_requests, 1e9, 77)
            server.samples = 0
            server.keep_images = False
            t = time.perf_counter()
            done = server.run(reqs, realtime=False)
            wall = time.perf_counter() - t
            closed[label] = {**latency_summary(done), "Gsamples/s": server.samples / wall / 1e9, "wall_s": wall}
    if audit is not None and len(audit_set) > audit:
        pick = np.linspace(0, len(audit_set) - 1, audit).round().astype(int)
        audit_set = [audit_set[i] for i in pick]
    errs = []
    for q in audit_set:
        bricks, kd = vols[q.volume]
        if q.kind != _lib.VOLUME_RENDER:
            # the random field's float64 values (the device holds their float32 rounding)
            bricks = [([bricks[0][0][0].astype(np.float64)], None, bricks[0][2], bricks[0][3], bricks[0][4])]
        errs.append(_audit_view(None, bricks, kd, q.camera, q.kind, q.image.cpu().numpy(),
                                tf=tfs[q.tf] if q.tf else None))
        q.image = None
    return {"workload": "4 resident volumes (64^3 uniform, 128^3-root AMR, 512^3 GRF, 4-level AMR), 16 TFs, "
                        "Poisson arrivals, sizes {256,512,1024,2048}^2",
            "value": closed["served"]["Gsamples/s"], "unit": "Gsamples/s",
            "rates": rows, "closed_loop": closed,
            "served_beats_plain": {"p99_every_rate": all(r["served_beats_plain_p99"] for r in rows),
                                   "closed_loop_gsamples": closed["served"]["Gsamples/s"]
                                   > closed["plain"]["Gsamples/s"]},
            "audit": {"n": len(errs), "max_rel_err": float(max(errs)) if errs else None,
                      "vs": "float64 oracle", "sample": "every 100th served request"
                      + (f", {audit} of them spread evenly" if audit is not None else "")},
            "requests_per_rate": n_requests, "slots": slots, "max_batch": max_batch, "hbm_budget_gib": 16,
            "batch_pixels": batch_pixels,
            "plain": "the same requests, one render_kernel launch each, one stream, in arrival order",
            "clocks": clocks.summary(), "build_seconds": t_build}


def run_serve(args):
    import torch

    dev = torch.device("cuda", 0)
    rates = [float(x) for x in args.rates.split(",")]
    rec = serve_record(dev, args.n_requests, rates, audit=args.audit, max_batch=args.max_batch, slots=args.slots,
                       batch_pixels=args.batch_pixels)
    line = {"metric": "Gsamples/s & p50/p99 latency", "workload": "serve", "value": rec["value"],
            "unit": "Gsamples/s", "n_gpus": 1, "higher_is_better": True, "served": rec}
    print(json.dumps(line), flush=True)


def run_prep(args):
    """Time to first image's brick preparation for the AMR dataset: yt's
    host path (numpy vertex centring, log10, per-leaf slicing, then packing
    and upload) against the device path (cell data uploaded once, bricks
    computed by ytgb_vertex_bricks), each from the grids to a resident
    BrickSet; then one render from each, compared bit for bit."""
    import torch

    from yt_gb300 import testing, workloads
    from yt_gb300.amr_kdtree import AMRKDTree
    from yt_gb300.render import Renderer
    from yt_gb300.volume import BrickSet

    dev = torch.device("cuda", 0)
    grids = testing.amr_blob_grids(root=args.root, levels=args.levels, patch=16, seed=0)
    w = workloads.amr_vr(root=args.root, levels=args.levels, res=args.res)
    out = {"host_ms": [], "device_ms": [], "kd_ms": []}
    bs_h = bs_d = kd = None
    for i in range(args.warmup + max(1, min(args.steps, 5))):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        kd = AMRKDTree(grids, log_field=True)
        t1 = time.perf_counter()
        bs_h = BrickSet(kd.bricks(), device=dev)
        torch.cuda.synchronize()
        t2 = time.perf_counter()
        kd2 = AMRKDTree(grids, log_field=True)
        t3 = time.perf_counter()
        bs_d = kd2.device_brickset(dev)
        torch.cuda.synchronize()
        t4 = time.perf_counter()
        if i >= args.warmup:
            out["kd_ms"].append(1e3 * (t1 - t0))
            out["host_ms"].append(1e3 * (t2 - t1))
            out["device_ms"].append(1e3 * (t4 - t3))
    def valid(bs):
        arena = bs.data.cpu().numpy()
        off = bs.desc_host["data_offset"][: bs.n]
        return np.concatenate([arena[o: o + v] for o, v in zip(off, bs.verts[: bs.n])]).view(np.int32)

    vh, vd = valid(bs_h), valid(bs_d)
    same_data = bool(np.array_equal(vh, vd))
    n_diff = int((vh != vd).sum())
    cam = w.views[0].camera
    a = Renderer(bs_h, w.tf, device=dev, kdtree=kd).render(cam)
    b = Renderer(bs_d, w.tf, device=dev, kdtree=kd).render(cam)
    line = {"metric": "brick preparation ms", "workload": "prep", "value": float(np.median(out["device_ms"])),
            "unit": "ms", "higher_is_better": False, "host_ms": float(np.median(out["host_ms"])),
            "kd_build_ms": float(np.median(out["kd_ms"])), "bricks": bs_d.n, "grids": len(grids),
            "arena_identical": same_data, "arena_values_differing": n_diff, "arena_values": int(vh.size),
            "image_identical": bool(torch.equal(a.view(torch.int64), b.view(torch.int64))),
            "device_upload_bytes": getattr(kd2, "device_upload_bytes", None),
            "config": {"workload": f"{args.root}^3 root + {args.levels} levels, 16^3 patches, log10 field"}}
    print(json.dumps(line), flush=True)


def run_octree(args):
    """The octree path (cast_through_octree): a 217k-cell octree dataset
    (levels 5-9, cells refined where the blob field exceeds the 85th
    percentile of their level), perspective 1024^2, VolumeRenderSampler with
    an 8-layer ColorTransferFunction; device time per frame, yt's compiled
    octree sampler (on a 128^2 sample of the same camera, all host threads)
    and the oracle's float64 image of that sample for the error."""
    import torch

    from oracle import cpu as ocpu
    from yt_gb300 import _lib, testing, workloads
    from yt_gb300.camera import Camera
    from yt_gb300.octree import Octree, OctreeVolume, render_octree
    from yt_gb300.render import relative_error
    from yt_gb300.transfer_functions import pack

    dev = torch.device("cuda", 0)
    t0 = time.time()
    depth, ipos, lvl, cells = testing.octree_cells(base_level=5, max_level=9, seed=0, percentile=85.0)
    oc = Octree(np.zeros(3), np.ones(3), depth)
    oc.add_nodes(ipos, lvl, np.arange(ipos.shape[0], dtype=np.int32))
    vol = OctreeVolume(oc, cells, dev)
    vmin, vmax = float(cells[:, :8].min()), float(cells[:, :8].max())
    tf = workloads.color_tf((vmin, vmax), 8)
    packed = pack(tf)
    t_build = time.time() - t0
    res = args.res
    # slightly off the axis: a camera on the domain's mid-planes sends the
    # image diagonals' rays exactly through cell edges, where the reference's
    # traversal also hands the sampler cells the ray only grazes (exit < enter)
    cam = Camera((0.52, 0.47, -1.0), (0.5, 0.5, 0.5), (1.5, 1.5, 1.5), res, lens_type="perspective")
    view = cam.device_view()
    img = torch.zeros((res, res, 4), dtype=torch.float64, device=dev)
    counters = torch.zeros(4, dtype=torch.int64, device=dev)
    error = torch.zeros(1, dtype=torch.int32, device=dev)
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device=dev)
    stream = torch.cuda.current_stream(dev)

    def step():
        img.zero_()
        render_octree(vol, view, _lib.VOLUME_RENDER, img, tf=packed, counters=counters, error=error)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    counters.zero_()
    steps = max(1, min(args.steps, 20))
    evs = []
    clocks = ClockSampler(0)
    with clocks:
        for _ in range(steps):
            flush.fill_(1.0)
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            step()
            e1.record(stream)
            evs.append((e0, e1))
        torch.cuda.synchronize()
    assert int(error.item()) == 0
    ms = np.array([a.elapsed_time(b) for a, b in evs])
    samples = int(counters[0].item()) // steps
    # CPU: yt's compiled octree sampler on a bounded sample of the view
    cres = max(32, res // 8)
    ccam = Camera(cam.position, cam.focus, cam.width, cres, lens_type="perspective")
    p = ccam.sampler_params()
    cpu = {"value": None, "kind": None}
    threads = os.cpu_count() or 1
    try:
        ref_pkg = reference_pkg()
        if not any((ref_pkg / "yt" / "utilities" / "lib").glob("image_samplers*.so")):
            raise ImportError("reference sampler not built")
        sys.path.insert(0, str(ref_pkg))
        from yt.utilities.lib import image_samplers as RIS  # noqa: PLC0415
        from yt.utilities.lib._octree_raytracing import _OctreeRayTracing  # noqa: PLC0415
        from yt.utilities.lib.partitioned_grid import PartitionedGrid  # noqa: PLC0415

        roc = _OctreeRayTracing(np.zeros(3), np.ones(3), depth)
        roc.add_nodes(ipos, lvl, np.arange(ipos.shape[0], dtype=np.int32))
        dt = cells.reshape(1, -1, 14, 1)
        pg = PartitionedGrid(0, dt, np.ones(dt.shape[1:], dtype=np.uint8), np.zeros(3), np.ones(3),
                             np.array([1, 1, 1], dtype="int64"), n_fields=1)
        rimg = np.zeros((cres, cres, 4))
        s = RIS.VolumeRenderSampler(p["vp_pos"], p["vp_dir"], p["center"], p["bounds"], rimg, p["x_vec"],
                                    p["y_vec"], p["width"], "Octree", tf, 1, lens_type=p["lens_type"],
                                    camera_data=p["camera_data"], zbuffer=np.ones((cres, cres)))
        tc = time.perf_counter()
        s(pg, oct=roc, num_threads=threads)
        dtc = time.perf_counter() - tc
        cpu["kind"] = "reference"
    except ImportError:
        dtc = None
    so = ocpu.OracleSampler("volume_render", p["vp_pos"], p["vp_dir"], p["center"], p["bounds"], p["image"],
                            p["x_vec"], p["y_vec"], p["width"], lens_type=p["lens_type"],
                            camera_data=p["camera_data"], tf=tf)
    tc = time.perf_counter()
    cvis = ocpu.render_octree(so, cells, ocpu.OracleOctree(depth, np.zeros(3), np.ones(3), ipos, lvl))
    dto = time.perf_counter() - tc
    if dtc is None:
        dtc, cpu["kind"] = dto, "port"
    cpu["value"] = cvis / dtc / 1e9
    # GPU image of the same sample against the oracle
    gimg = torch.zeros((cres, cres, 4), dtype=torch.float64, device=dev)
    render_octree(vol, ccam.device_view(), _lib.VOLUME_RENDER, gimg, tf=packed)
    mx, rms = relative_error(gimg.cpu().numpy(), p["image"], channels=(0, 1, 2))
    hbm, _ = peaks()
    alg = samples * BYTES_PER_SAMPLE + res * res * BYTES_PER_RAY
    line = {"metric": "Gsamples/s", "workload": "octree", "value": samples / (ms.mean() / 1e3) / 1e9,
            "unit": "Gsamples/s", "n_gpus": 1, "steps": steps, "warmup": args.warmup,
            "ms_per_step": float(ms.mean()), "higher_is_better": True, "samples_per_step": samples,
            "roofline": {"bound": "hbm", "achieved": alg / (float(ms.mean()) / 1e3) / 1e9, "peak": hbm,
                         "unit": "GB/s", "frac": alg / (float(ms.mean()) / 1e3) / 1e9 / hbm,
                         "model": f"{BYTES_PER_SAMPLE} B/sample + {BYTES_PER_RAY} B/ray (the kd path's model)"},
            "cpu_baseline": {**cpu, "unit": "Gsamples/s", "cores": threads,
                             "sample": f"the same camera at {cres}x{cres} ({cvis} samples)"},
            "accuracy": {"max_rel_err": mx, "rms_rel_err": rms, "vs": f"float64 oracle at {cres}x{cres}"},
            "clocks": clocks.summary(),
            "config": {"workload": "octree: 217k cells, levels 5-9, perspective, 8-layer CTF, 1 sample/cell",
                       "cells": int(cells.shape[0]), "nodes": int(vol.n_nodes), "depth": depth,
                       "resolution": res, "l2": "flushed between steps (256 MiB write)"},
            "build_seconds": t_build}
    print(json.dumps(line), flush=True)


def run_offaxis(args):
    """Octree off-axis projection by cell splatting (add_cells_to_image_offaxis,
    the octree branch of off_axis_projection): the 217k cells of the octree
    workload (levels 5-9) projected along an oblique normal onto a
    plane-parallel 1024^2 image.  A sample is one stamp subcell of one cell
    (the reference's inner loop).  ``value``: device time with the cells and
    the view's stamps resident; ``e2e``: the drop-in call with host arrays
    (stamps, uploads, download).  CPU: yt's compiled splatting, all host
    threads, on every 8th cell."""
    import torch

    from oracle import cpu as ocpu
    from yt_gb300 import testing
    from yt_gb300.camera import Camera
    from yt_gb300.offaxis import CellSplat, add_cells_to_image_offaxis

    dev = torch.device("cuda", 0)
    _, _, _, cells = testing.octree_cells(base_level=5, max_level=9, seed=0, percentile=85.0)
    le, re = cells[:, 8:11], cells[:, 11:14]
    X = np.ascontiguousarray((le + re) / 2 - 0.5)
    dx = np.ascontiguousarray((re - le)[:, 0])
    q = np.ascontiguousarray(cells[:, :8].mean(axis=1))
    w = np.ones_like(dx)
    res = args.res
    cam = Camera((0.5 - 0.45, 0.5 + 0.6, 0.5 - 0.66), (0.5, 0.5, 0.5), (1, 1, 1), res, lens_type="plane-parallel")
    rot = np.ascontiguousarray(cam.inv_mat.T)
    splat = CellSplat(X, dx, q, w, device=dev)
    subcells = splat.subcells(res, res)
    bufs = (torch.zeros(res * res, dtype=torch.float64, device=dev),
            torch.zeros(res * res, dtype=torch.float64, device=dev))
    error = torch.zeros(1, dtype=torch.int32, device=dev)
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device=dev)
    stream = torch.cuda.current_stream(dev)

    def step():
        bufs[0].zero_()
        bufs[1].zero_()
        splat.project(rot, res, res, out=bufs, error=error)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    steps = max(1, min(args.steps, 20))
    evs = []
    clocks = ClockSampler(0)
    with clocks:
        for _ in range(steps):
            flush.fill_(1.0)
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            step()
            e1.record(stream)
            evs.append((e0, e1))
        torch.cuda.synchronize()
    assert int(error.item()) == 0
    ms = np.array([a.elapsed_time(b) for a, b in evs])
    # end to end through the drop-in: host arrays in, host images out
    e2e = []
    for _ in range(max(2, min(steps, 5))):
        b, bw = np.zeros((res, res)), np.zeros((res, res))
        torch.cuda.synchronize()
        tc = time.perf_counter()
        add_cells_to_image_offaxis(Xp=X, dXp=dx, qty=q, weight=w, rotation=rot, buffer=b, buffer_weight=bw,
                                   Nx=res, Ny=res, device=dev)
        e2e.append(time.perf_counter() - tc)
    e2e_s = float(np.median(e2e))
    # CPU: every 8th cell, yt's compiled splatting on all host threads (the
    # stamps use the full set's largest cell, as the full call would)
    sub = slice(0, None, 8)
    Xs, dxs, qs, ws = (np.ascontiguousarray(a[sub]) for a in (X, dx, q, w))
    dxs_stamp = dxs.copy()
    dxs_stamp[np.argmax(dxs)] = dx.max()
    ssub = CellSplat(Xs, dxs_stamp, qs, ws, device=dev)
    sub_subcells = ssub.subcells(res, res)
    threads = os.cpu_count() or 1
    cpu = {"value": None, "kind": None}
    rb, rbw = np.zeros((res, res)), np.zeros((res, res))
    try:
        ref_pkg = reference_pkg()
        if not any((ref_pkg / "yt" / "utilities" / "lib").glob("image_utilities*.so")):
            raise ImportError("reference splatting not built")
        sys.path.insert(0, str(ref_pkg))
        from yt.utilities.lib import image_utilities as RIU  # noqa: PLC0415

        tc = time.perf_counter()
        RIU.add_cells_to_image_offaxis(Xp=Xs, dXp=dxs_stamp, qty=qs, weight=ws, rotation=rot, buffer=rb,
                                       buffer_weight=rbw, Nx=res, Ny=res)
        dtc = time.perf_counter() - tc
        cpu["kind"] = "reference"
    except ImportError:
        tc = time.perf_counter()
        ocpu.add_cells_to_image_offaxis(Xp=Xs, dXp=dxs_stamp, qty=qs, weight=ws, rotation=rot, buffer=rb,
                                        buffer_weight=rbw, Nx=res, Ny=res)
        dtc = time.perf_counter() - tc
        cpu["kind"], threads = "port", 1
    cpu["value"] = sub_subcells / dtc / 1e9
    # accuracy: the device on the same subset against the oracle
    ob, obw = np.zeros((res, res)), np.zeros((res, res))
    ocpu.add_cells_to_image_offaxis(Xp=Xs, dXp=dxs_stamp, qty=qs, weight=ws, rotation=rot, buffer=ob,
                                    buffer_weight=obw, Nx=res, Ny=res)
    g = ssub.project(rot, res, res)
    gb = g[0].cpu().numpy().reshape(res, res)
    err = float(np.max(np.abs(gb - ob)) / np.max(np.abs(ob)))
    sec = ms.mean() / 1e3
    line = {"metric": "Gsamples/s", "workload": "offaxis", "value": subcells / sec / 1e9, "unit": "Gsamples/s",
            "n_gpus": 1, "steps": steps, "warmup": args.warmup, "ms_per_step": float(ms.mean()),
            "higher_is_better": True, "samples_per_step": subcells, "cells_per_s": dx.size / sec,
            "e2e": {"value": subcells / e2e_s / 1e9, "unit": "Gsamples/s", "ms": e2e_s * 1e3,
                    "h2d_bytes_per_step": int(splat.upload_bytes), "d2h_bytes_per_step": 2 * 8 * res * res},
            "cpu_baseline": {**cpu, "unit": "Gsamples/s", "cores": threads,
                             "sample": f"every 8th cell ({dxs.size} cells, {sub_subcells} subcells) at {res}^2"},
            "accuracy": {"max_rel_err": err, "vs": "float64 oracle on the CPU sample"},
            "clocks": clocks.summary(),
            "config": {"workload": "octree off-axis projection: 217k cells, levels 5-9, plane-parallel, "
                                   "oblique normal", "cells": int(dx.size), "resolution": res,
                       "l2": "flushed between steps (256 MiB write)"}}
    print(json.dumps(line), flush=True)


if __name__ == "__main__":
    a = parse()
    if a.impl == "reference":
        run_reference(a)
    elif a.workload == "uniform":
        run_uniform(a)
    elif a.workload == "multiview":
        run_multiview(a)
    elif a.workload == "projection":
        run_projection(a)
    elif a.workload == "serve":
        run_serve(a)
    elif a.workload == "prep":
        run_prep(a)
    elif a.workload == "octree":
        run_octree(a)
    elif a.workload == "offaxis":
        run_offaxis(a)
    else:
        run_ours(a)
