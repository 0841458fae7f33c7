"""Benchmark of the GB300 densifier on the 1920x960, 6-source workload.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

A step is one keyframe through the whole path, as the reference's
densification and fusion threads run it per keyframe in steady state:
Philox initialisation, init scoring, 8 red-black sweeps (propagation + 6
refinements per pixel visit, top-3 view selection), the post-filter, the
geometric-consistency filter of the keyframe's depth against four resident
neighbour depth maps (1 px round trip, 0.01 relative depth, 3 consistent
views of 5) and point fusion of the cleaned map against the four neighbour
maps (0.08 relative depth, the reference's example configuration).  The
metric is Mpix*views/s = (W*H/1e6) * sources / seconds per keyframe (whole
job: summed over GPUs; N > 1 runs independent replicas).

  value : device-resident inputs, CUDA-event time of the step on the
          request's stream; L2 is flushed (256 MB write) between steps.
  e2e   : the same step through the public C ABI from pinned host buffers:
          host->device copy of the 7 images, then pm_request_run,
          pm_filter_consistency_device and pm_fuse_device, then the
          device->host copy of the cleaned depth, the score map and the fused
          points, all inside the timed region.

served: the same densifier behind the served request loop (pm_server) on a
          keyframe stream along a trajectory through a hall of boxes, mixed
          1920x960 / 3840x1920 keyframes, 4-8 neighbours from a 40-keyframe
          device cache, prior results reused as initialisation (keyframes
          without one start coarse to fine); capacity
          (stream submitted at once) against the plain form on the same
          stream (one keyframe at a time, no prior, 8 sweeps), and p50/p99
          latency of 1920x960 keyframes with 6 neighbours arriving as a
          10 Hz Poisson stream in real time.

--impl reference times the reference's per-pixel CPU algorithm (the oracle's
restatement of the reference kernel arithmetic, OpenMP on all host cores) on
a bounded band of rows of the same workload.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

W, H, S, SWEEPS = 1920, 960, 6, 8
METRIC = "Mpix·views/s and p50/p99 keyframe latency, served vs plain at ≤1% depth error"
UNIT = "Mpix·views/s"
WORKLOAD = ("plain PatchMatch, one 1920x960 u8 equirect keyframe + 6 sources per step, 8 red-black sweeps, "
            "11x11 window at stride 2, top-3 view selection, post-filter, geometric-consistency filter "
            "(1 px round trip, 0.01 relative depth, 3 of 5 views) and point fusion (0.08) against 4 resident "
            "neighbour depth maps, room + 5 boxes + cylinder scene")
TOP_K = 3
CHAIN_FINE_SWEEPS = 2  # full-size sweeps of a coarse-to-fine chain (seeded from its half-size pass)
CLEAN_THR, CLEAN_PX, CLEAN_MIN = 0.01, 1.0, 3
FUSE_THR = 0.08
FLOP_PER_SAMPLE = 40  # algorithmic FP32 work of one (pixel, hypothesis, source, tap) sample
SFU_PER_SAMPLE = 4    # special-function operations of one sample (rcp, rsqrt and the two angles)


def _optional(fn, *a):
    """One optional form's block, or {"error": ...} when it raises: the
    headline line, measured before the optional forms, is printed either way."""
    try:
        return fn(*a)
    except Exception as e:  # noqa: BLE001 - reported in the line, with its traceback on stderr
        import traceback
        traceback.print_exc()
        return {"error": f"{type(e).__name__}: {e}"}


def _mpix_views(ms: float) -> float:
    return (W * H / 1e6) * S / (ms / 1e3)


def _samples_per_half_sweep() -> float:
    """Nominal samples of one half-sweep: every pixel's 14 candidates, as the
    reference scores them.  The kernel skips those that cannot be accepted."""
    ph = 5
    interior = (W - 2 * (ph + 1) + 1) * (H - 2 * (ph + 1) + 1)
    return interior / 2 * 14 * S * 36


def _samples_per_step() -> float:
    """Nominal samples of one keyframe's densification: init scoring (one
    hypothesis per interior pixel) and 2 x SWEEPS half-sweeps of 14."""
    return _samples_per_half_sweep() * (2 * SWEEPS + 1 / 7)


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu: int):
        self.gpu = gpu
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except (FileNotFoundError, OSError):
            self.proc = None
        return self

    def __exit__(self, *a):
        if self.proc is None:
            return
        self.proc.terminate()
        try:
            out, _ = self.proc.communicate(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
            out, _ = self.proc.communicate()
        self.lines = [ln for ln in out.splitlines() if ln.strip()]

    def summary(self):
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx.append(float(f[2]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower() in ("active", "1"):
                    reasons.add(n)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "reasons": sorted(reasons),
                "samples": len(sm)}


def _dist():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    if ws <= 1:
        return 0, 1, 0, None
    import torch.distributed as dist
    rank = int(os.environ["RANK"])
    local = int(os.environ.get("LOCAL_RANK", rank))
    dist.init_process_group("gloo")  # barriers and the max-reduction only; replicas share nothing
    return rank, ws, local, dist


def _barrier(dist):
    if dist is not None:
        dist.barrier()


def _allmax(dist, x: float) -> float:
    if dist is None:
        return x
    import torch
    t = torch.tensor([x], dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def _hbm_view(traffic, launch_ms):
    """The same launch against the measured HBM copy bandwidth: DRAM bytes
    (ncu) per launch over its CUDA-event time, to show it is not HBM-bound."""
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if traffic is None or not os.path.exists(path):
        return None
    peak = json.load(open(path)).get("hbm_gbs")
    if not peak:
        return None
    gbs = traffic / (launch_ms * 1e-3) / 1e9
    return {"bound": "hbm", "achieved": gbs, "peak": peak, "unit": "GB/s", "frac": gbs / peak,
            "peak_source": "MEASURED_PEAKS.json hbm_gbs (measured)"}


# Counters of this workload's launches from ncu captures (--profile-sweep),
# valid only for the kernel sources they were taken on: a different build
# reports null rather than a stale figure.  DRAM bytes of the 8th half-sweep
# (dram__bytes_read.sum + dram__bytes_write.sum); samples that were scored:
# texture instructions x active lanes (smsp__inst_executed_op_texture.sum x
# smsp__thread_inst_executed_per_inst_executed.ratio), summed over the 16
# half-sweeps, and over those and the two launches of the init scoring.
NCU = {"bytes_per_launch": 60010496, "sweep_samples": 25129033853, "step_samples": 25517314546,
       "sources_sha256": "91e84aaed48dd0584f5fe820d6caf3a90ec3caa6dee748b41b72585ebd83eb6c"}
KERNEL_SOURCES = ("patchmatch_gb300/csrc/pm_sweep.cuh", "patchmatch_gb300/csrc/pm_device.cuh",
                  "patchmatch_gb300/csrc/pm_inst.cu", "patchmatch_gb300/csrc/pm_types.h")


def kernel_sources_sha256() -> str:
    import hashlib
    h = hashlib.sha256()
    for f in KERNEL_SOURCES:
        with open(os.path.join(ROOT, f), "rb") as fh:
            h.update(fh.read())
    return h.hexdigest()


def _counted(key):
    return NCU[key] if NCU["sources_sha256"] == kernel_sources_sha256() else None


def cpu_sample(target_s: float = 12.0, threads: int = 0):
    """The reference's per-keyframe host work on the workload: the per-pixel
    densification (oracle, reference float arithmetic, top-3 views, OpenMP)
    on a band of rows, 8 sweeps, scaled to the full keyframe, plus the
    consistency filter and fusion of full-size maps (the reference runs both
    single-threaded, depthmap.cc:1320-1377,1535-1696).  Returns Mpix*views/s,
    the band rows, seconds per keyframe, threads and the seconds the sample took."""
    from oracle import oracle as O
    from patchmatch_gb300 import scene
    req = scene.config_request(2, seed=0)
    V = O.Views.from_request(req)
    cp = O.cost_params(arith=O.ARITH_F32_REF, combine=O.COMBINE_TOPK, top_k=TOP_K)
    threads = threads or os.cpu_count() or 1
    # calibrate on 4 rows x 1 sweep
    r0 = H // 2
    t = O.patchmatch(V, cp, iterations=1, row_lo=r0, row_hi=r0 + 4, threads=threads)["seconds"]
    per_row_sweep = max(t / 4.0, 1e-4)
    rows = int(max(2, min(H - 20, target_s / (per_row_sweep * SWEEPS))))
    lo = max(6, r0 - rows // 2)
    res = O.patchmatch(V, cp, iterations=SWEEPS, row_lo=lo, row_hi=lo + rows, threads=threads)
    dens = res["seconds"] * H / rows
    maps = [np.ascontiguousarray(v.depth, np.float32) for v in req.views[:5]]
    t0 = time.perf_counter()
    cleaned = O.clean([maps[1], maps[2], maps[0], maps[3], maps[4]], req.R[[1, 2, 0, 3, 4]], req.t[[1, 2, 0, 3, 4]],
                      center=2, thr=CLEAN_THR, min_consistent=CLEAN_MIN, reproj_px=CLEAN_PX)
    O.prune([cleaned] + maps[1:5], req.R[:5], req.t[:5], None, FUSE_THR)
    post = time.perf_counter() - t0
    secs = dens + post
    value = (W * H / 1e6) * S / secs
    return value, rows, secs, threads, res["seconds"] + post

def reference_gpu_sweep_ms():
    """The reference's own CUDA path (PatchMatchCuda.cu compiled unmodified,
    launched with its launch shape and per-pass synchronisation) timed per
    red+black sweep at 1920x960 with its two sources; None when the reference
    kernels were not built or no GPU is present."""
    try:
        import torch
        if not torch.cuda.is_available():
            return None
        from oracle import refkernels
        if not refkernels.available():
            return None
        from patchmatch_gb300 import scene
        req = scene.make_request(scene.ROOM_OBJECTS, W, H, 2, seed=33, bmin=0.1, bmax=0.8)
        rk = refkernels.RefKernels()
        rk.setup([v.gray_u8.astype(np.float32) for v in req.views], req.R, req.t)
        rk.run(1, 0.3, 20.0)
        return min(rk.time_passes(4) for _ in range(3))
    except Exception:
        return None


def run_reference(args):
    rank, ws, _, dist = _dist()
    if rank != 0:
        return
    steps = []
    info = None
    for k in range(args.warmup + args.steps):
        v, rows, _, threads, wall_s = cpu_sample(target_s=args.cpu_seconds)
        if k >= args.warmup:
            steps.append((v, wall_s))
        info = (rows, threads)
    value = statistics.median(v for v, _ in steps)
    rows, threads = info
    sample = (f"densification of rows {H // 2 - rows // 2}..+{rows} of the 1920x960x6 workload (all {SWEEPS} "
              "sweeps, top-3) scaled to the keyframe, plus the full-size consistency filter and fusion")
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": 1e3 * statistics.median(s for _, s in steps),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": WORKLOAD, "W": W, "H": H, "sources": S, "sweeps": SWEEPS,
                       "sample": sample},
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port", "sample": sample},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    ref_gpu = None if args.no_reference_gpu else reference_gpu_sweep_ms()
    if ref_gpu is not None:
        # the reference's CUDA path supports exactly two sources: 8 sweeps of
        # 1920x960 with 2 sources, as Mpix*views/s (sweeps only)
        line["reference_cuda"] = {"ms_per_sweep": ref_gpu, "sources": 2, "W": W, "H": H,
                                  "sweeps_value": (W * H / 1e6) * 2 / (SWEEPS * ref_gpu / 1e3), "unit": UNIT,
                                  "note": "PatchMatchCuda.cu compiled unmodified for sm_103a, its launch shape and "
                                          "per-pass device synchronisation; 2 sources (its only configuration)"}
    print(json.dumps(line))


def _stream_quality(res, stream):
    accs, valid = [], []
    for (rc, d, _, info), kf in zip(res, stream):
        if rc != 0:
            continue
        m = d > 0
        gt = kf.depth
        accs.append(float((np.abs(d[m] - gt[m]) / gt[m] < 0.01).mean()) if m.any() else 0.0)
        valid.append(float(m.mean()))
    return accs, valid


def _drive(native, ctx, stream, cfg, realtime: bool):
    """Submit a keyframe stream to a fresh server (at the arrival times when
    realtime, else all at once) and collect every result; with dense output,
    end the stream and collect the fused outputs too (statuses, point counts)."""
    srv = native.Server(ctx, cfg)
    t0 = time.perf_counter()
    tks = []
    for kf in stream:
        if realtime:
            dt = t0 + kf.t_s - time.perf_counter()
            if dt > 0:
                time.sleep(dt)
        tks.append(srv.submit(kf.gray_u8, kf.R, kf.t))
    res = [srv.wait(tk) for tk in tks]
    wall = time.perf_counter() - t0
    dense = None
    if cfg.dense_output:
        srv.finish()
        dense = []
        for tk in tks:
            st, _, xyz, _ = srv.wait_dense(tk)
            dense.append((st, 0 if xyz is None else len(xyz)))
    srv.close()
    return res, wall, dense


def run_served(native, scene, ctx, local: int, args) -> dict:
    """Served form against the plain form on the same keyframe stream."""
    stream = scene.served_stream(seed=0, duration_s=60.0, rate_hz=args.served_rate, t_end=args.served_seconds,
                                 device=local)
    base = dict(cache_capacity=40, min_sources=4, max_sources=8, min_baseline=0.05, max_baseline=3.0)
    p8 = native.default_params(iterations=SWEEPS)
    plain_cfg = native.server_config(params=p8, max_inflight=1, seed_from_prior=0, coarse_to_fine=0, **base)
    overlap_cfg = native.server_config(params=p8, max_inflight=4, seed_from_prior=0, coarse_to_fine=0, **base)
    served_cfg = native.server_config(params=p8, max_inflight=4, seed_from_prior=1, seeded_iterations=2,
                                      prior_lag=4, **base)
    out = {}
    for name, cfg in (("plain", plain_cfg), ("served_8_sweeps", overlap_cfg), ("served", served_cfg)):
        l0 = ctx.launches
        with ClockSampler(local) as clk:
            res, wall, _ = _drive(native, ctx, stream, cfg, realtime=False)
        work = sum(kf.shape[0] * kf.shape[1] * info["n_sources"] for (rc, _, _, info), kf in zip(res, stream)
                   if rc == 0) / 1e6
        accs, valid = _stream_quality(res, stream)
        out[name] = {"value": work / wall, "wall_s": wall, "keyframes": len(stream),
                     "densified": sum(r[0] == 0 for r in res),
                     "not_densified_too_few_neighbours": sum(r[0] == native.PM_ENOTREADY for r in res),
                     "seeded": sum(r[3]["seeded"] == 1 for r in res if r[0] == 0),
                     "coarse_to_fine": sum(r[3]["seeded"] == 2 for r in res if r[0] == 0),
                     "within_1pct_of_truth": float(np.mean(accs)) if accs else 0.0,
                     "valid_fraction": float(np.mean(valid)) if valid else 0.0,
                     "gpu_launches": int(ctx.launches - l0), "clocks": clk.summary()}
    out["ratio_served_over_plain"] = out["served"]["value"] / out["plain"]["value"]
    out["ratio_overlap_only_at_8_sweeps"] = out["served_8_sweeps"]["value"] / out["plain"]["value"]
    out["gain_note"] = ("served_8_sweeps: continuous batching alone, every keyframe 8 full sweeps from a random "
                        "start; served: the same plus prior results reused as initialisation (2 sweeps when seeded, "
                        "coarse to fine when no prior exists) - its gain over plain comes mainly from that "
                        "work reduction, at higher accuracy against the truth (within_1pct_of_truth); all forms "
                        "count every densified keyframe as (W*H/1e6)*sources")
    sizes = sorted({kf.shape for kf in stream})
    out["stream"] = (f"hall of boxes, 60 s trajectory through 20 waypoints, Poisson {args.served_rate:g} Hz "
                     f"arrivals over the first {args.served_seconds:g} s, sizes {[f'{w}x{h}' for h, w in sizes]} "
                     f"(3:1), 4-8 neighbours within 0.05-3 m from a 40-keyframe device cache; submitted at once")
    out["forms"] = {"plain": "max_inflight 1, no prior, 8 sweeps",
                    "served_8_sweeps": "max_inflight 4, no prior, no coarse-to-fine, 8 sweeps",
                    "served": "max_inflight 4, prior result "
                    "reused as initialisation (lag 4), 2 sweeps when seeded; a keyframe without a prior runs "
                    "8 sweeps at half resolution, then 2 at full resolution seeded from them"}

    # latency: 1920x960 keyframes with 6 neighbours at 10 Hz, real time
    lstream = scene.served_stream(seed=1, duration_s=60.0, rate_hz=10.0, sizes=((1920, 960),), p_sizes=(1.0,),
                                  t_end=args.latency_seconds, device=local)
    lat_cfg = native.server_config(params=p8, max_inflight=4, seed_from_prior=1, seeded_iterations=2, prior_lag=1,
                                   cache_capacity=40, min_sources=6, max_sources=6, min_baseline=0.05,
                                   max_baseline=3.0, dense_output=1)
    with ClockSampler(local) as clk:
        res, wall, dense = _drive(native, ctx, lstream, lat_cfg, realtime=True)
    lat_all = [r[3]["latency_ms"] for r in res if r[0] == 0]
    lat_seeded = [r[3]["latency_ms"] for r in res if r[0] == 0 and r[3]["seeded"] == 1]
    accs, valid = _stream_quality(res, lstream)
    pct = lambda a, q: float(np.percentile(a, q)) if a else None
    out["latency"] = {"p50_ms": pct(lat_all, 50), "p99_ms": pct(lat_all, 99), "max_ms": max(lat_all, default=None),
                      "steady_p50_ms": pct(lat_seeded, 50), "steady_p99_ms": pct(lat_seeded, 99),
                      "keyframes": len(lstream), "densified": len(lat_all), "seeded": len(lat_seeded),
                      "within_1pct_of_truth": float(np.mean(accs)) if accs else 0.0,
                      "dense_output": {"fused": sum(st == 0 for st, _ in dense),
                                       "points_per_fused_keyframe": float(np.mean([n for st, n in dense if st == 0]))
                                       if any(st == 0 for st, _ in dense) else 0.0,
                                       "not_fused_window_never_filled": sum(st == native.PM_ENOTREADY
                                                                            for st, _ in dense)},
                      "workload": f"1920x960, 6 neighbours, Poisson 10 Hz for {args.latency_seconds:g} s in real "
                                  "time, each keyframe seeded from the one before it (lag 1), the first coarse to "
                                  "fine; consistency filter (centre of 5, 1 px / 0.01) and fusion (head of 5, "
                                  "0.08) run on the stream alongside; steady = keyframes seeded from an earlier "
                                  "result",
                      "clocks": clk.summary()}
    return out


def run_pipeline(native, scene, ctx, local: int, steps: int) -> dict:
    """The stages after densification at 1920x960 over a 5-keyframe window
    (the reference's cleaner and pruner queues): geometric-consistency filter
    (pm_filter_consistency) and point fusion (pm_fuse), each timed through the
    C ABI with host buffers in and out (copies included)."""
    import torch
    sc = scene.Scene(scene.ROOM_OBJECTS, 14)
    R, t = sc.poses(5, 14, 0.1, 0.4, 15.0)
    d = torch.empty((H, W), dtype=torch.float32, device=f"cuda:{local}")
    rgb = torch.empty((H, W, 3), dtype=torch.uint8, device=f"cuda:{local}")
    rng = np.random.default_rng(0)
    depths = []
    for v in range(5):
        sc.render_device(R[v], t[v], W, H, depth=d, bgr=rgb if v == 0 else None)
        torch.cuda.synchronize()
        dv = d.cpu().numpy() * (1 + rng.normal(0, 0.004, (H, W))).astype(np.float32)
        dv[rng.random((H, W)) < 0.1] = 0
        depths.append(dv.astype(np.float32))
    bgr = np.ascontiguousarray(rgb.cpu().numpy())
    import ctypes as C
    L = native.lib()
    Rd = np.ascontiguousarray(R, np.float64)
    td = np.ascontiguousarray(t, np.float64)
    work = [d.copy() for d in depths]          # pm_fuse edits the later maps in place
    ptrs = (C.c_void_p * 5)(*[w.ctypes.data for w in work])
    cleaned = np.zeros((H, W), np.float32)
    pruned = np.zeros((H, W), np.float32)
    xyz = np.zeros((H * W, 3), np.float64)
    cols = np.zeros((H * W, 3), np.uint8)
    ij = np.zeros((H * W, 2), np.int32)
    pts = native.Points(H * W, 0, xyz.ctypes.data, cols.ctypes.data, ij.ctypes.data)

    def clean():
        ctx.check(L.pm_filter_consistency(ctx.h, W, H, 5, C.cast(ptrs, C.c_void_p), Rd.ctypes.data, td.ctypes.data,
                                          2, CLEAN_THR, CLEAN_MIN, CLEAN_PX, cleaned.ctypes.data))

    def fuse():
        ctx.check(L.pm_fuse(ctx.h, W, H, 5, C.cast(ptrs, C.c_void_p), Rd.ctypes.data, td.ctypes.data,
                            bgr.ctypes.data, FUSE_THR, pruned.ctypes.data, C.byref(pts)))

    out = {}
    for name, fn in (("filter", clean), ("fuse", fuse)):
        ts = []
        for k in range(max(3, steps) + 1):
            for w, d0 in zip(work, depths):
                np.copyto(w, d0)               # fresh maps, outside the timed call
            t0 = time.perf_counter()
            fn()
            if k:
                ts.append(time.perf_counter() - t0)
        out[f"{name}_ms"] = 1e3 * statistics.median(ts)
    out["fused_points"] = int(pts.count)
    # the same calls on device buffers (pm_filter_consistency_device,
    # pm_fuse_device), CUDA events on the context's stream
    dev = torch.device("cuda", local)
    dd = [torch.from_numpy(x).to(dev) for x in depths]
    dw = [torch.empty_like(x) for x in dd]
    dclean = torch.empty((H, W), dtype=torch.float32, device=dev)
    dpr = torch.empty((H, W), dtype=torch.float32, device=dev)
    dxyz = torch.empty((H * W, 3), dtype=torch.float32, device=dev)
    dcnt = torch.zeros(1, dtype=torch.int32, device=dev)
    wsb = native.fuse_workspace_bytes(W, H)
    wsbuf = torch.empty(wsb + 256, dtype=torch.uint8, device=dev)
    wsp = (wsbuf.data_ptr() + 255) & ~255
    cst = torch.cuda.ExternalStream(ctx.stream_handle)
    for name, fn in (("filter_device", lambda: ctx.filter_consistency_device(
            [x.data_ptr() for x in dd], W, H, R, t, 2, CLEAN_THR, dclean.data_ptr(), CLEAN_MIN, CLEAN_PX)),
                     ("fuse_device", lambda: ctx.fuse_device([x.data_ptr() for x in dw], W, H, R, t, FUSE_THR,
                                                             dpr.data_ptr(), dxyz.data_ptr(), dcnt.data_ptr(), wsp,
                                                             wsb))):
        ts = []
        for k in range(max(3, steps) + 1):
            with torch.cuda.stream(cst):
                for a, b in zip(dw, dd):
                    a.copy_(b)
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record(cst)
            fn()
            with torch.cuda.stream(cst):
                e1.record(cst)
            e1.synchronize()
            if k:
                ts.append(e0.elapsed_time(e1))
        out[f"{name}_ms"] = statistics.median(ts)
    out["workload"] = ("1920x960, 5 depth maps (0.4 % noise, 10 % holes); filter: centre map 2, 1 % depth "
                       "threshold, 1 px round trip, 3 consistent views; fuse: head map 0 against 1-4, 8 % "
                       "threshold; one C ABI call each, host buffers in and out (copies included, buffers "
                       "preallocated), and the device-buffer calls (CUDA events)")
    return out


BATCH_SIZES = ((960, 480), (1920, 960), (2880, 1440), (3840, 1920))


def run_batched(native, scene, ctx, local: int, args) -> dict:
    """Batched form: requests of sizes drawn from BATCH_SIZES with 3-10
    sources (room scenes, per-request seeds), densified one at a time
    (pm_request_run, 8 sweeps), as one batch (pm_batch, executor chosen by
    pm_batch_tune on the first 16 requests) and as one batch of coarse-to-fine
    chains: a request 1920 wide becomes a half-size request (8 sweeps, images
    resized on the device) plus the full-size request seeded from it (2
    sweeps); wider ones a quarter-size (8), half-size (2) and full-size (2)
    chain; 960 wide ones stay at 8 sweeps.  Measured per request at 6 sources:
    these chains keep the post-filtered coverage and reach at least plain's
    accuracy, while a single full-size sweep loses a fifth of the coverage.
    Every form is credited (W*H/1e6)*sources per request; accuracy is the
    fraction of post-filtered pixels within 1 % of the rendered truth."""
    import torch
    rng = np.random.default_rng(12345)
    reqs, work, truth, views_dev = [], 0.0, [], []
    dev = torch.device("cuda", local)
    for k in range(args.batched_requests):
        W, H = BATCH_SIZES[rng.integers(len(BATCH_SIZES))]
        S = int(rng.integers(3, 11))
        sc = scene.Scene(scene.ROOM, 1000 + k)
        R, t = sc.poses(S + 1, 1000 + k, 0.2, 0.5, 15.0)
        r = ctx.request(W, H, S, native.default_params(iterations=SWEEPS, seed=k, keyframe_id=k))
        imgs = []
        for v in range(S + 1):
            img = torch.empty((H, W), dtype=torch.uint8, device=dev)
            dmap = torch.empty((H, W), dtype=torch.float32, device=dev) if v == 0 else None
            sc.render_device(R[v], t[v], W, H, gray=img, depth=dmap,
                             stream=torch.cuda.current_stream(dev).cuda_stream)
            torch.cuda.current_stream(dev).synchronize()
            r.set_view(v, img.data_ptr(), R[v], t[v])
            r.synchronize()
            if v == 0:
                truth.append(dmap.cpu().numpy())
            imgs.append(img)
        views_dev.append((imgs, R, t))
        reqs.append(r)
        work += W * H / 1e6 * S
    torch.cuda.synchronize()

    def accuracy(rs):
        acc = []
        for r, gt in zip(rs, truth):
            d = r.read(want=("depth",))["depth"]
            m = d > 0
            acc.append(float((np.abs(d[m] - gt[m]) / gt[m] < 0.01).mean()) if m.any() else 0.0)
        return float(np.mean(acc))

    # plain: one keyframe at a time (each request's graph captured by an untimed run)
    for r in reqs:
        r.run()
        r.synchronize()
    t0 = time.perf_counter()
    for r in reqs:
        r.run()
        r.synchronize()
    plain_s = time.perf_counter() - t0
    plain_acc = accuracy(reqs)
    # batched: executor tuned on a subset, then the whole set in one graph
    sub = native.Batch(ctx, reqs[:16])
    tuning = sub.tune()
    sub.close()
    b = native.Batch(ctx, reqs)
    b.set_executor(tuning["executor"], tuning["grid_mult"])
    l0 = ctx.launches
    b.run()
    b.synchronize()
    l1 = ctx.launches

    def timed(batch):
        stream = torch.cuda.ExternalStream(batch.stream_handle)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        with ClockSampler(local) as clk:
            t1 = time.perf_counter()
            with torch.cuda.stream(stream):
                e0.record(stream)
            batch.run()
            with torch.cuda.stream(stream):
                e1.record(stream)
            batch.synchronize()
            wall = time.perf_counter() - t1
        return e0.elapsed_time(e1) / 1e3, wall, clk.summary()

    batch_s, batch_wall, batch_clk = timed(b)
    b.close()
    # coarse-to-fine chains in one batch: 1920 wide: half size (8 sweeps) then
    # full size (2); wider: quarter size (8), half (2), full (2)
    coarse = []
    for r, (imgs, R, t) in zip(reqs, views_dev):
        if r.W < 1920:
            continue
        levels = [4, 2] if r.W >= 2880 else [2]
        prev = None
        for lv, f in enumerate(levels):
            c = ctx.request(r.W // f, r.H // f, r.S,
                            native.default_params(iterations=SWEEPS if lv == 0 else CHAIN_FINE_SWEEPS,
                                                  seed=r.params.seed, keyframe_id=r.params.keyframe_id))
            for v, img in enumerate(imgs):
                small = ctx.resize(img, r.W // f, r.H // f)
                torch.cuda.synchronize()
                c.set_view(v, small.data_ptr(), R[v], t[v])
                c.synchronize()
            if prev is not None:
                c.set_prior(prev)
            coarse.append(c)
            prev = c
        r.set_params(native.default_params(iterations=CHAIN_FINE_SWEEPS, seed=r.params.seed,
                                           keyframe_id=r.params.keyframe_id))
        r.set_prior(prev)
    chain = native.Batch(ctx, coarse + reqs)
    chain.set_executor(tuning["executor"], tuning["grid_mult"])
    l2 = ctx.launches
    chain.run()
    chain.synchronize()
    l3 = ctx.launches
    chain_s, chain_wall, chain_clk = timed(chain)
    chain_acc = accuracy(reqs)
    chain.close()
    names = {native.BATCH_PERSISTENT: "persistent tile queue", native.BATCH_LAUNCHES: "per-request launches",
             native.BATCH_STREAMS: "parallel graph branches",
             native.BATCH_MIXED: "one persistent tile queue over all source counts"}
    for r in reqs:
        r.set_prior(None)
        r.close()
    for c in coarse:
        c.set_prior(None)
    for c in coarse:
        c.close()
    return {"requests": len(reqs), "work_mpix_views": work,
            "plain": {"value": work / plain_s, "seconds": plain_s, "form": "pm_request_run one at a time, 8 sweeps",
                      "within_1pct_of_truth": plain_acc},
            "batched": {"value": work / batch_s, "seconds": batch_s, "wall_s": batch_wall,
                        "executor": names[tuning["executor"]], "grid_mult": tuning["grid_mult"],
                        "gpu_launches": int(l1 - l0), "clocks": batch_clk,
                        "form": "one graph, 8 sweeps, maps bit-identical to plain"},
            "batched_coarse_to_fine": {"value": work / chain_s, "seconds": chain_s, "wall_s": chain_wall,
                                       "gpu_launches": int(l3 - l2), "clocks": chain_clk,
                                       "within_1pct_of_truth": chain_acc, "coarse_requests": len(coarse),
                                       "form": f"one graph; 1920 wide: half size {SWEEPS} sweeps, then full size "
                                               f"{CHAIN_FINE_SWEEPS} seeded from it; 2880 and 3840 wide: quarter "
                                               f"size {SWEEPS}, half {CHAIN_FINE_SWEEPS}, full {CHAIN_FINE_SWEEPS}, "
                                               f"each seeded from the one before; 960 wide: {SWEEPS} sweeps"},
            "ratio_batched_over_plain": plain_s / batch_s,
            "ratio_coarse_to_fine_batch_over_plain": plain_s / chain_s,
            "tuning_ms_first16": dict(zip(["persistent x1", "persistent x2", "per-request launches",
                                           "parallel graph branches", "mixed persistent"], tuning["candidate_ms"])),
            "workload": f"{len(reqs)} requests, sizes uniform over {[f'{w}x{h}' for w, h in BATCH_SIZES]}, 3-10 "
                        f"sources, room scenes with per-request seeds; the 8-sweep batch is bit-identical to "
                        "plain, the coarse-to-fine batch does less work at the accuracy shown"}


class KeyframeStep:
    """One keyframe through the path on the device: pm_request_run
    (densification + post-filter), pm_filter_consistency_device against four
    resident neighbour depth maps (window order n0 n1 keyframe n2 n3, centre
    2) and pm_fuse_device of the cleaned map against the four neighbours (head
    0), all on the request's stream.  The neighbours are sources 1-4 of the
    request, each densified once beforehand with the other six views as its
    sources; fusion edits later maps in place, so each step fuses fresh device
    copies of them (copied on the stream inside the step)."""

    def __init__(self, native, ctx, req, params, local):
        import torch
        self.torch, self.native, self.ctx = torch, native, ctx
        dev = torch.device("cuda", local)
        imgs = [np.ascontiguousarray(v.gray_u8) for v in req.views]
        self.imgs = imgs
        self.R, self.t = req.R, req.t
        self.r = ctx.request(W, H, S, params)
        self.r.set_views(imgs, req.R, req.t)
        self.nbr = []
        for q in (1, 2, 3, 4):
            order = [q] + [k for k in range(S + 1) if k != q]
            rq = ctx.request(W, H, S, native.default_params(iterations=params.iterations, combine=params.combine,
                                                            top_k=params.top_k, seed=params.seed, keyframe_id=q))
            rq.set_views([imgs[k] for k in order], req.R[order], req.t[order])
            rq.run()
            rq.synchronize()
            self.nbr.append(torch.from_numpy(rq.read()["depth"]).to(dev))
            rq.close()
        self.work = [torch.empty_like(n) for n in self.nbr]
        self.cleaned = torch.zeros((H, W), dtype=torch.float32, device=dev)
        self.pruned = torch.zeros((H, W), dtype=torch.float32, device=dev)
        self.xyz = torch.zeros((H * W, 3), dtype=torch.float32, device=dev)
        self.ij = torch.zeros((H * W, 2), dtype=torch.int32, device=dev)
        self.count = torch.zeros(1, dtype=torch.int32, device=dev)
        self.ws_bytes = native.fuse_workspace_bytes(W, H)
        self.ws = torch.empty(self.ws_bytes + 256, dtype=torch.uint8, device=dev)
        self.ws_ptr = (self.ws.data_ptr() + 255) & ~255
        win = [1, 2, 0, 3, 4]
        self.R_win, self.t_win = req.R[win], req.t[win]
        self.R_fuse, self.t_fuse = req.R[:5], req.t[:5]
        self.st = self.r.stream_handle
        self.es = torch.cuda.ExternalStream(self.st)

    def enqueue(self):
        """The step, enqueued on the request's stream."""
        torch = self.torch
        self.r.run()
        ptrs = [n.data_ptr() for n in self.nbr]
        self.ctx.filter_consistency_device([ptrs[0], ptrs[1], self.r.depth_device_ptr, ptrs[2], ptrs[3]], W, H,
                                           self.R_win, self.t_win, 2, CLEAN_THR, self.cleaned.data_ptr(),
                                           min_consistent=CLEAN_MIN, reproj_px=CLEAN_PX, stream=self.st)
        with torch.cuda.stream(self.es):
            for w, n in zip(self.work, self.nbr):
                w.copy_(n, non_blocking=True)
        self.ctx.fuse_device([self.cleaned.data_ptr()] + [w.data_ptr() for w in self.work], W, H, self.R_fuse,
                             self.t_fuse, FUSE_THR, self.pruned.data_ptr(), self.xyz.data_ptr(),
                             self.count.data_ptr(), self.ws_ptr, self.ws_bytes, ij_ptr=self.ij.data_ptr(),
                             stream=self.st)

    def close(self):
        self.r.close()
        self.es = None
        self.nbr = self.work = self.cleaned = self.pruned = self.xyz = self.ij = self.count = self.ws = None


def run_precision(native, scene, ctx, local: int) -> dict:
    """Precision form: one 3840x1920 keyframe with 8 sources as FP16 images
    (sigma-2 noise on unrounded intensities, FP32 NCC moments), densified at
    full resolution (8 sweeps) and coarse to fine over its 3-level FP16
    pyramid (960x480 8 sweeps, 1920x960 and 3840x1920 2 seeded sweeps each),
    timed with CUDA events on the requests' stream; accuracy against the
    scene's analytic depth.  The cost error against the FP64 oracle is
    measured by tests/test_gpu_precision.py."""
    import torch
    Wp, Hp, Sp = 3840, 1920, 8
    dev = torch.device("cuda", local)
    sc = scene.Scene(scene.ROOM, 77)
    R, t = sc.poses(Sp + 1, 77, 0.2, 0.5, 15.0)
    imgs = []
    for v in range(Sp + 1):
        g = torch.empty((Hp, Wp), dtype=torch.float32, device=dev)
        sc.render_device_f32(R[v], t[v], Wp, Hp, g, noise_sigma=2.0, noise_seed=100 + v)
        imgs.append(g.clamp(0, 255).half())
    truth = torch.empty((Hp, Wp), dtype=torch.float32, device=dev)
    sc.render_device(R[0], t[0], Wp, Hp, depth=truth)
    torch.cuda.synchronize()
    gt = truth.cpu().numpy()
    del truth

    def request(views, Wl, Hl, iterations):
        r = ctx.request(Wl, Hl, Sp, native.default_params(image_format=native.IMAGE_F16, iterations=iterations))
        for k, im in enumerate(views):
            r.set_view(k, im.data_ptr(), R[k], t[k])
        r.synchronize()
        return r

    def accuracy(r):
        d = r.read(want=("depth",))["depth"]
        m = d > 0
        e = np.abs(d[m] - gt[m]) / gt[m]
        return {"within_1pct_of_truth": float((e < 0.01).mean()), "median_rel_error": float(np.median(e)),
                "valid_fraction": float(m.mean())}

    def timed(first, run, reps=3):
        """ms per run on the last request's stream (all levels run on one stream
        per request; the chain's levels are ordered by their prior events)."""
        stream = torch.cuda.ExternalStream(first.stream_handle)
        run()
        torch.cuda.synchronize()
        ms = []
        for _ in range(reps):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                e0.record(stream)
            last = run()
            last_stream = torch.cuda.ExternalStream(last.stream_handle)
            with torch.cuda.stream(last_stream):
                e1.record(last_stream)
            torch.cuda.synchronize()
            ms.append(e0.elapsed_time(e1))
        return float(np.mean(ms))

    full = request(imgs, Wp, Hp, SWEEPS)
    with ClockSampler(local) as clk:
        ms_full = timed(full, lambda: (full.run(), full)[1])
    a_full = accuracy(full)
    full.close()
    pyr = [ctx.pyramid_f16(im, 3) for im in imgs]
    lv2 = request([p[2] for p in pyr], Wp // 4, Hp // 4, SWEEPS)
    lv1 = request([p[1] for p in pyr], Wp // 2, Hp // 2, CHAIN_FINE_SWEEPS)
    lv0 = request(imgs, Wp, Hp, CHAIN_FINE_SWEEPS)
    lv1.set_prior(lv2)
    lv0.set_prior(lv1)

    def chain():
        lv2.run()
        lv1.run()
        lv0.run()
        return lv0

    ms_c2f = timed(lv2, chain)
    a_c2f = accuracy(lv0)
    for r in (lv0, lv1, lv2):
        r.close()
    del pyr, imgs
    torch.cuda.synchronize()
    work = Wp * Hp / 1e6 * Sp
    return {"workload": f"{Wp}x{Hp} FP16 keyframe, {Sp} sources, sigma-2 noise, fold combination, texture "
                        f"sampler, {SWEEPS} sweeps, post-filter",
            "full": {"ms": ms_full, "value": work / (ms_full / 1e3), "unit": UNIT, **a_full},
            "coarse_to_fine": {"ms": ms_c2f, "value": work / (ms_c2f / 1e3), "unit": UNIT,
                               "levels": f"{Wp // 4}x{Hp // 4} {SWEEPS} sweeps, then {Wp // 2}x{Hp // 2} and "
                                         f"{Wp}x{Hp} {CHAIN_FINE_SWEEPS} seeded sweeps each", **a_c2f},
            "clocks": clk.summary(),
            "cost_error_vs_fp64": "tests/test_gpu_precision.py (1e6 hypotheses x 8 sources)"}


def run_ours(args):
    import torch
    rank, ws, local, dist = _dist()
    torch.cuda.set_device(local)
    from patchmatch_gb300 import native, scene

    req = scene.config_request(2, seed=rank)
    ctx = native.Context(local)
    p = native.default_params(iterations=SWEEPS, seed=rank, combine=native.COMBINE_TOPK, top_k=TOP_K)
    ks = KeyframeStep(native, ctx, req, p, local)
    r = ks.r
    stream = ks.es
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=f"cuda:{local}")

    # --- device-resident steps ---
    for _ in range(args.warmup):
        ks.enqueue()
    r.synchronize()
    torch.cuda.synchronize()
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    launches0 = ctx.launches
    _barrier(dist)
    torch.cuda.synchronize()
    t_wall = time.perf_counter()
    with ClockSampler(local) as clk:
        for k in range(args.steps):
            with torch.cuda.stream(stream):
                flush.fill_(k & 0xFF)  # L2 flush between steps, outside the events
                ev[k][0].record(stream)
            ks.enqueue()
            with torch.cuda.stream(stream):
                ev[k][1].record(stream)
        r.synchronize()
        torch.cuda.synchronize()
    wall = time.perf_counter() - t_wall
    _barrier(dist)
    gpu_launches = ctx.launches - launches0
    ms = [a.elapsed_time(b) for a, b in ev]
    ms_step = _allmax(dist, sum(ms) / len(ms))
    value = ws * _mpix_views(ms_step)
    lat = np.array(ms)
    fused_points = int(ks.count.item())
    cleaned_valid = float((ks.cleaned > 0).float().mean().item())

    # --- dominant kernel: one red-black half-sweep, the mean of a keyframe's 16 on the request's stream ---
    r.run()
    r.init()
    nhalf = 2 * SWEEPS
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with torch.cuda.stream(stream):
        e0.record(stream)
    r.sweep(0, nhalf)
    with torch.cuda.stream(stream):
        e1.record(stream)
    r.synchronize()
    sweep_ms = e0.elapsed_time(e1) / nhalf
    peak = ctx.probe_fp32_peak()

    # --- end to end through the C ABI from pinned host buffers ---
    pin = [torch.from_numpy(im).pin_memory() for im in ks.imgs]
    d_out = torch.empty((H, W), dtype=torch.float32).pin_memory()
    s_out = torch.empty((H, W), dtype=torch.float32).pin_memory()
    n_pin = torch.empty(1, dtype=torch.int32).pin_memory()
    xyz_pin = torch.empty((H * W, 3), dtype=torch.float32).pin_memory()
    ij_pin = torch.empty((H * W, 2), dtype=torch.int32).pin_memory()
    import ctypes as C
    L = native.lib()
    maps = native.Maps()
    maps.score = s_out.data_ptr()

    def e2e_step():
        for k in range(S + 1):
            ctx.check(L.pm_request_set_view(r.h, k, C.byref(native.make_view(pin[k].data_ptr(), req.R[k],
                                                                              req.t[k]))))
        ks.enqueue()
        ctx.check(L.pm_request_read_async(r.h, C.byref(maps), 0))
        with torch.cuda.stream(stream):
            d_out.copy_(ks.cleaned, non_blocking=True)
            n_pin.copy_(ks.count, non_blocking=True)
        r.synchronize()
        n = int(n_pin.item())
        with torch.cuda.stream(stream):
            xyz_pin[:n].copy_(ks.xyz[:n], non_blocking=True)
            ij_pin[:n].copy_(ks.ij[:n], non_blocking=True)
        r.synchronize()
        return n

    for _ in range(max(1, args.warmup)):
        e2e_step()
    _barrier(dist)
    e2e_t = []
    n_pts = 0
    for _ in range(args.steps):
        flush.fill_(1)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        n_pts = e2e_step()
        e2e_t.append(time.perf_counter() - t0)
    e2e_ms = _allmax(dist, 1e3 * sum(e2e_t) / len(e2e_t))
    e2e_value = ws * _mpix_views(e2e_ms)
    e2e_d2h = int(2 * 4 * W * H + 4 + n_pts * (12 + 8))
    gt = req.views[0].depth
    dn = d_out.numpy().copy()  # no view may keep the pinned buffer alive past the request's stream
    m = dn > 0
    valid = float(m.mean())
    acc = float((np.abs(dn[m] - gt[m]) / gt[m] < 0.01).mean()) if m.any() else 0.0
    filt = r.read()["depth"]
    mf = filt > 0
    acc_filt = float((np.abs(filt[mf] - gt[mf]) / gt[mf] < 0.01).mean()) if mf.any() else 0.0

    # two sources (the reference CUDA path's only configuration), per red+black sweep
    req2 = scene.make_request(scene.ROOM_OBJECTS, W, H, 2, seed=33, bmin=0.1, bmax=0.8)
    r2 = ctx.request(W, H, 2, native.default_params(iterations=SWEEPS))
    r2.set_views([v.gray_u8 for v in req2.views], req2.R, req2.t)
    r2.run()
    r2.synchronize()
    st2 = torch.cuda.ExternalStream(r2.stream_handle)
    two = []
    for _ in range(3):
        r2.init()
        a2, b2 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        with torch.cuda.stream(st2):
            a2.record(st2)
        r2.sweep(0, 2 * SWEEPS)
        with torch.cuda.stream(st2):
            b2.record(st2)
        r2.synchronize()
        two.append(a2.elapsed_time(b2) / SWEEPS)
    r2.close()
    two_source = {"ms_per_sweep": min(two), "sources": 2, "W": W, "H": H,
                  "sweeps_value": (W * H / 1e6) * 2 / (SWEEPS * min(two) / 1e3), "unit": UNIT,
                  "note": "compare with reference_cuda in the --impl reference line (same scene and sizes)"}
    served = None if args.no_served else _optional(run_served, native, scene, ctx, local, args)
    batched = None if args.no_batched else _optional(run_batched, native, scene, ctx, local, args)
    precision = None if args.no_precision else _optional(run_precision, native, scene, ctx, local)
    pipeline = _optional(run_pipeline, native, scene, ctx, local, args.steps)
    traffic = _counted("bytes_per_launch")
    # the roofline terms of the cost kernel (samples/s): 40 FP32 flop, 4
    # special-function operations and 1 bilinear fetch per sample
    sfu = ctx.probe_sfu_peak()
    tex = ctx.probe_tex_peak()
    terms = {"fp32": peak * 1e12 / FLOP_PER_SAMPLE, "sfu": sfu * 1e9 / SFU_PER_SAMPLE, "tex": tex * 1e9}
    binding = min(terms, key=terms.get)
    scored, scored_step = _counted("sweep_samples"), _counted("step_samples")
    samples_s = scored / nhalf / (sweep_ms * 1e-3) if scored else None
    achieved = FLOP_PER_SAMPLE * samples_s / 1e12 if scored else None
    nominal_s = _samples_per_half_sweep() / (sweep_ms * 1e-3)
    line = None
    if rank == 0:
        cpu = None
        if not args.no_cpu and ws == 1:  # the CPU leg runs at N = 1 only
            def cpu_leg():
                v, rows, secs, threads, _ = cpu_sample(target_s=args.cpu_seconds)
                return {"value": v, "unit": UNIT, "cores": threads, "kind": "port",
                        "sample": f"densification of {rows} rows x 1920 of the same workload (all {SWEEPS} "
                                  f"sweeps, top-3, reference float arithmetic, OpenMP) scaled to the keyframe, "
                                  f"plus the full-size consistency filter and fusion: {secs:.1f} s per keyframe"}
            cpu = _optional(cpu_leg)
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded ray-cast scene, analytic ground truth)",
            "config": {"workload": WORKLOAD, "W": W, "H": H, "sources": S, "sweeps": SWEEPS, "image": "u8",
                       "parallelism": "replicas" if ws > 1 else "single GPU",
                       "l2": "flushed between steps (256 MB write outside the timed events)"},
            "latency_ms": {"p50": float(np.percentile(lat, 50)), "p99": float(np.percentile(lat, 99)),
                           "form": "plain (one keyframe at a time)"},
            "quality": {"cleaned_valid_fraction": valid, "cleaned_within_1pct_of_truth": acc,
                        "postfiltered_valid_fraction": float(mf.mean()), "postfiltered_within_1pct_of_truth": acc_filt,
                        "fused_points": fused_points},
            "e2e": {"value": e2e_value, "unit": UNIT, "ms_per_step": e2e_ms,
                    "h2d_bytes_per_step": int((S + 1) * W * H), "d2h_bytes_per_step": e2e_d2h,
                    "form": "images from pinned host memory -> pm_request_set_view, pm_request_run, "
                            "pm_filter_consistency_device, pm_fuse_device -> cleaned depth, score and fused "
                            "points (xyz, pixel) to pinned host memory"},
            "roofline": {"bound": "fp32", "kernel": "tile_kernel (red-black half-sweep)",
                         "achieved": achieved, "peak": peak, "unit": "TFLOP/s",
                         "frac": achieved / peak if scored else None,
                         "peak_source": "in-run FFMA probe (pm_probe_fp32_peak); MEASURED_PEAKS.json has no FP32 figure",
                         "flop_per_sample": FLOP_PER_SAMPLE, "samples_per_launch": scored / nhalf if scored else None,
                         "samples_source": "samples that were scored (ncu, current sources, mean of the keyframe's "
                                           "half-sweeps), null when the kernel sources differ from the profiled",
                         "launch_ms": sweep_ms, "traffic": traffic,
                         "traffic_source": "ncu dram__bytes_read.sum + dram__bytes_write.sum of the current sources' "
                                           "sweep kernel, null when the kernel sources differ from the profiled",
                         "terms_samples_per_s": terms, "binding_term": binding,
                         "achieved_samples_per_s": samples_s,
                         "frac_of_binding": samples_s / terms[binding] if scored else None,
                         "nominal_equivalent": {
                             "samples_per_launch": _samples_per_half_sweep(), "samples_per_s": nominal_s,
                             "tflops": FLOP_PER_SAMPLE * nominal_s / 1e12,
                             "note": "as if all 14 candidates of every pixel were scored; not a rate of the hardware"},
                         "probes": {"fp32_tflops": peak, "sfu_gops": sfu, "tex_gfetches": tex},
                         "hbm_view": _hbm_view(traffic, sweep_ms)},
            "value_vs_roofline": {
                "samples_per_step": scored_step,
                "frac": {k: scored_step / v / (ms_step / 1e3) for k, v in terms.items()} if scored_step else None,
                "nominal_samples_per_step": _samples_per_step(),
                "note": "the whole step (densification, post-filter, consistency filter, fusion) against the "
                        "time that the samples it scores take at each roofline term"},
            "served": served,
            "batched": batched,
            "precision": precision,
            "pipeline": pipeline,
            "two_source_sweeps": two_source,
            "cpu_baseline": cpu,
            "clocks": clk.summary(),
            "gpu_launches": int(gpu_launches),
            "wall_s_timed_region": wall,
        }
        print(json.dumps(line), flush=True)
    # the pinned e2e buffers were copied on the request's stream: free them
    # while that stream still exists (their allocator records events on it)
    del pin, d_out, s_out, n_pin, xyz_pin, ij_pin
    torch.cuda.synchronize()
    del ev, e0, e1, stream
    ks.close()
    del ks
    torch.cuda.synchronize()
    ctx.close()
    if dist is not None:
        dist.destroy_process_group()


def run_profile_sweep():
    """One densification of the 1920x960x6 keyframe (init scoring, 16
    half-sweeps, post-filter) and nothing else: the case the sweep kernel's
    ncu captures select launches from (tile_kernel launches 0 and 1 are the
    init scoring, launch k + 1 the k-th half-sweep)."""
    from patchmatch_gb300 import native, scene
    req = scene.config_request(2, seed=0)
    with native.Context(0) as ctx:
        r = ctx.request(W, H, S, native.default_params(iterations=SWEEPS, combine=native.COMBINE_TOPK, top_k=TOP_K))
        r.set_views([v.gray_u8 for v in req.views], req.R, req.t)
        r.run()
        r.synchronize()
        r.close()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--cpu-seconds", type=float, default=12.0)
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline leg")
    ap.add_argument("--no-served", action="store_true", help="skip the served-form measurement")
    ap.add_argument("--no-batched", action="store_true", help="skip the batched-form measurement")
    ap.add_argument("--no-precision", action="store_true", help="skip the precision-form measurement")
    ap.add_argument("--no-reference-gpu", action="store_true",
                    help="reference arm: skip timing the reference's CUDA path")
    ap.add_argument("--batched-requests", type=int, default=64, help="requests in the batched-form measurement")
    ap.add_argument("--served-rate", type=float, default=4.0, help="arrival rate of the capacity stream (Hz)")
    ap.add_argument("--served-seconds", type=float, default=30.0, help="length of the capacity stream (s)")
    ap.add_argument("--latency-seconds", type=float, default=20.0, help="length of the 10 Hz latency stream (s)")
    ap.add_argument("--profile-sweep", action="store_true",
                    help="densify one keyframe and exit (the case for ncu captures of the sweep kernel)")
    args = ap.parse_args()
    if args.profile_sweep:
        run_profile_sweep()
    elif args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    import faulthandler
    faulthandler.enable()
    main()
