#!/usr/bin/env python3
"""Throughput benchmark of the B200 path tracer (one JSON line on stdout).

Workload: the instancing + environment-light scene — 1024 instances of a
subdivision-4 icosphere (5120 triangles, fBm-displaced), random rotations and
per-axis scale U[0.5,2]^3, Lambert / GGX metal / plastic materials, a
1024x512 float sky with a 0.5 degree sun sampled by its 2D CDF; 1920x1080,
64 spp, max depth 8, RR from depth 4, seed 1, clamp 0. A step is one full
render of that frame (132.7 M camera paths).

Metric: Mrays/s = (radiance + shadow traces) / render time, the reference
renderer's definition (src/capi_render.cpp:266-292). `value` is the scene
resident on the device, timed with CUDA events on the launching stream, L2
flushed (256 MiB write) between steps; `e2e` is the same metric through
sundog_render_ex with host buffers (asset load, CDF + BVH build, uploads,
render, film download all inside the timed call).

Multi-GPU (torchrun): one process per GPU; with N ranks the frame takes
64 N spp and rank r renders its 64x64 film tiles t with t % N == r (every
rank about the one-GPU frame's paths: scaling "weak"); no data-path
collective, time = max over ranks; one all-gather of the disjoint films
after the timed steps assembles the frame (film_gather_ms).

--impl reference: the CPU oracle (oracle/, a restatement of the reference's
render path; the reference itself needs OptiX and cannot run here) on the
host cores, each step a bounded row sample of the same frame.
"""

import argparse
import ctypes
import hashlib
import json
import os
import re
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "Mrays/s"
UNIT = "Mrays/s"
WORKLOADS = {
    0: ("cornell: 5 Lambert rects, emissive rect (17,12,4), GGX metal sphere r 0.3, glass "
        "sphere ior 1.5; 256x256, 16 spp, depth 8, seed 1, clamp 0", (256, 256, 16)),
    1: ("instancing+env: 1024 fBm icosphere-4 instances (5.24M tris), 1024x512 HDR sky "
        "+ sun, 1920x1080, 64 spp, depth 8, seed 1, clamp 0", (1920, 1080, 64)),
    2: ("volumes: 64-step flame with its point lights, water ior 1.33 with fBm normals and "
        "Beer absorption, nested glass sphere, 5 rough glass panels, 2048-tri emissive mesh "
        "light; 2560x1440, 256 spp, depth 8, seed 1, clamp 0", (2560, 1440, 256)),
}
# sundog's own gallery scenes that load no asset files, replayed from the call
# streams its unchanged scenelib sends (tests/golden/abi_<scene>.json), with
# the reference's published throughput at its benchmark settings (1920x1080,
# 64 spp, the scene's own depth / clamp / seed; GB200, OptiX with software
# traversal; reference docs/BENCHMARKS.md).
GALLERY = {
    "01-marble-run": (1209.0, "docs/BENCHMARKS.md:9"),
    "02-cornell-lume": (819.0, "docs/BENCHMARKS.md:10"),
}


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--config", type=int, default=1, choices=[0, 1, 2],
                    help="workload: 0 Cornell box, 1 instancing + env map (default), 2 volumes")
    ap.add_argument("--scene", default=None, choices=sorted(GALLERY),
                    help="instead of a config: one of sundog's gallery scenes at its "
                         "published benchmark settings (1920x1080, 64 spp)")
    ap.add_argument("--width", type=int, default=0, help="override the workload's width")
    ap.add_argument("--height", type=int, default=0, help="override the workload's height")
    ap.add_argument("--spp", type=int, default=0, help="override the workload's spp")
    ap.add_argument("--cpu-seconds", type=float, default=15.0,
                    help="target CPU time of the cpu_baseline sample")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--chunk-spp", type=int, default=0,
                    help="samples per path-kernel pass (0: the library's choice, per-sample "
                         "buffers near 1 GiB)")
    ap.add_argument("--engine", type=int, default=0, choices=[0, 1, 2],
                    help="path-tracing kernels: 0 automatic, 1 megakernel, 2 wavefront")
    ap.add_argument("--guiding", action="store_true",
                    help="learned-guiding equal-time relMSE line instead of Mrays/s")
    ap.add_argument("--guide-spp", type=int, default=0,
                    help="0: the guided scene's config (instancing 64, volumes 256)")
    ap.add_argument("--guide-width", type=int, default=0,
                    help="0: the guided scene's config (instancing 1920, volumes 2560)")
    ap.add_argument("--guide-height", type=int, default=0,
                    help="0: the guided scene's config (instancing 1080, volumes 1440)")
    ap.add_argument("--guide-ref-spp", type=int, default=16384)
    ap.add_argument("--guide-seeds", type=int, default=4)
    ap.add_argument("--guide-scene", default="instancing", choices=["instancing", "volumes"],
                    help="scene of the guiding line: the instancing config's 1024 instances "
                         "under the sun-and-sky env map (the guiding config's scene), or the "
                         "volumes config's flame / water / glass")
    ap.add_argument("--serving", action="store_true",
                    help="render-server line (Poisson jobs, p50/p99 latency) instead of Mrays/s")
    ap.add_argument("--serve-jobs", type=int, default=60)
    ap.add_argument("--serve-rate", type=float, default=20.0)
    ap.add_argument("--serve-batch", type=int, default=0,
                    help="camera paths per server batch (0 = the server's default)")
    ap.add_argument("--serve-engine", type=int, default=0, choices=[0, 1, 2],
                    help="server kernels: 0 wavefront, 1 megakernel")
    return ap.parse_args()


def asset_dir():
    d = os.path.join(tempfile.gettempdir(), "sundog_b200_assets")
    os.makedirs(d, exist_ok=True)
    return d


def resolve_workload(args):
    """Fills args.width / height / spp from the workload and returns its
    description and the reference's published Mrays/s for it (or None)."""
    if args.scene:
        w, h, spp = 1920, 1080, 64
        desc = ("sundog gallery scene %s (its scenelib call stream replayed unchanged), "
                "1920x1080, 64 spp, the scene's own depth, clamp and seed" % args.scene)
        published = GALLERY[args.scene]
    else:
        desc, (w, h, spp) = WORKLOADS[args.config]
        published = None
    args.width = args.width or w
    args.height = args.height or h
    args.spp = args.spp or spp
    if (args.width, args.height, args.spp) != (w, h, spp):
        desc += " [overridden: %dx%d, %d spp]" % (args.width, args.height, args.spp)
    return desc, published


def make_scene(args):
    if args.scene:
        from sundog_b200 import callstream
        return callstream.CallStreamScene(
            os.path.join(ROOT, "tests", "golden", "abi_%s.json" % args.scene))
    from sundog_b200 import workloads
    make = {0: lambda: workloads.cornell(width=args.width, height=args.height, spp=args.spp),
            1: lambda: workloads.instancing(asset_dir(), width=args.width, height=args.height,
                                            spp=args.spp),
            2: lambda: workloads.volumes(asset_dir(), width=args.width, height=args.height,
                                         spp=args.spp)}
    return make[args.config]()


# ---- clocks ---------------------------------------------------------------------------

class ClockSampler(object):
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.idx = gpu_index
        self.proc = None
        self.out = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.idx), "--query-gpu=" + self.FIELDS,
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=self.out, stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.out.flush()
        self.out.seek(0)
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in self.out.read().splitlines():
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax.append(float(parts[2]))
            except ValueError:
                continue
            for n, v in zip(names, parts[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        os.unlink(self.out.name)
        return {"sm_mhz": float(np.median(sm)) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "samples": len(sm), "reasons": sorted(reasons)}


# ---- roofline ---------------------------------------------------------------------------

def measured_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.isfile(p):
        with open(p) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


KERNEL_SOURCES = ("pt_kernel.cu", "wavefront.cu", "bvh_device.cu")


def code_digest(csrc=os.path.join(ROOT, "sundog_b200", "csrc")):
    """Digest of the path-tracing kernels' code: their sources and every
    header, comments and spacing aside. A committed ncu summary names the
    digest it was captured at."""
    names = sorted(n for n in os.listdir(csrc) if n in KERNEL_SOURCES or n.endswith((".cuh", ".h")))
    h = hashlib.sha256()
    for n in names:
        with open(os.path.join(csrc, n)) as f:
            text = re.sub(r"//[^\n]*|/\*.*?\*/", " ", f.read(), flags=re.S)
        h.update((n + " " + " ".join(text.split()) + "\n").encode())
    return h.hexdigest()[:12]


def profile_figures(name, folder=os.path.join(ROOT, "profiles"), code=None):
    """`key: value` figures of a committed ncu summary (measured on a small
    case), or {} when it is missing or its `code:` is not the present
    kernels': counters of another kernel say nothing about this one's time."""
    p = os.path.join(folder, name)
    if not os.path.isfile(p):
        return {}
    with open(p) as f:
        text = f.read()
    m = re.search(r"^code:\s*(\w+)\s*$", text, re.M)
    if not m or m.group(1) != (code or code_digest()):
        return {}
    return {m.group(1): float(m.group(2))
            for m in re.finditer(r"^([a-z0-9_]+):\s*([0-9][0-9.eE+-]*)\s*$", text, re.M)
            if m.group(1) != "code"}


def ncu_traffic_per_path(engine=0):
    """DRAM bytes (read + write) per camera path of the path-tracing kernels,
    from the committed ncu summary of a smaller render of the same workload
    (traffic is per-path work: path state between stages, per-sample
    radiance writes, stack lines), so a chunk's traffic is this times its
    paths; None without a summary of the present kernels. engine 1 = the
    persistent megakernel, else the wavefront engine."""
    name = "pt_persistent_instancing.md" if engine == 1 else "wf_render_dram_instancing_small.md"
    return profile_figures(name).get("dram_bytes_per_path")


# Algorithmic bytes of the traversal on the BVH it walks (the library's 4-wide
# nodes by default): 32 B per child box tested (AABB 24 + link 8), 36 B per
# triangle, 48 B per quadric (its affine), 64 B per instance transform entered.
def bytes_per_ray(c):
    total = 32.0 * c.box_tests + 36.0 * c.tri_tests + 48.0 * c.quadric_tests + 64.0 * c.blas_entries
    return total / max(c.rays, 1)


def sum_counts(a, b):
    """Both ray kinds' traversal counts together (the path loop's are a's)."""
    from sundog_b200 import abi
    c = abi.TraceCounts()
    for f, _ in abi.TraceCounts._fields_:
        setattr(c, f, getattr(a, f) + (0 if f.startswith("loop") else getattr(b, f)))
    return c


def l2_copy_gbps(stream):
    """L2-resident copy bandwidth measured here (read + write bytes over
    CUDA-event time): a 24 MiB float buffer copied into another,
    both held in the 126 MB L2 after the first pass -- the L2 denominator of
    the trace stage's roofline, measured like the HBM copy peak (best of 30
    after 200 warm-up copies)."""
    import torch
    n = 24 << 18  # 24 MiB of float32
    a = torch.ones(n, dtype=torch.float32, device="cuda")
    b = torch.empty_like(a)
    best = 0.0
    with torch.cuda.stream(stream):
        for _ in range(200):  # clocks up, both buffers resident in L2
            b.copy_(a)
        for _ in range(30):
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            for _ in range(10):
                b.copy_(a)
            e1.record(stream)
            e1.synchronize()
            ms = e0.elapsed_time(e1) / 10
            best = max(best, 2 * n * 4 / (ms / 1e3) / 1e9)
    return best


def stage_roofline(lib, ses, stream, flush, rad, shd, peak, workload):
    """One more render of the frame (after the timed steps, not part of
    `value`) with per-stage CUDA events: each stage kernel's own time, and for
    the two traversal stages their algorithmic bytes (radiance and shadow
    rays counted apart) over that time. L2 bytes and issue-slot utilisation
    come from the committed small-case ncu summary of the trace stage, if it is
    of the present kernels."""
    import torch
    from sundog_b200 import abi
    abi.check(lib.sundog_session_set_stage_timing(ses.handle, 1), "stage timing", lib)
    flush.fill_(1)
    torch.cuda.synchronize()
    ses.render(stream=stream.cuda_stream)
    t = abi.StageTimes()
    abi.check(lib.sundog_session_stage_times(ses.handle, ctypes.byref(t)), "stage times", lib)
    abi.check(lib.sundog_session_set_stage_timing(ses.handle, 0), "stage timing", lib)
    total = t.start_ms + t.trace_ms + t.shade_a_ms + t.shadow_ms + t.shade_b_ms
    b_rad, b_shd = bytes_per_ray(rad), bytes_per_ray(shd)
    out = {}
    for name, ms, rays, bpr in (("wfTraceFetch", t.trace_ms, t.radiance_rays, b_rad),
                                ("wfShadow", t.shadow_ms, t.shadow_rays, b_shd)):
        ach = bpr * rays / (ms / 1e3) / 1e9 if ms > 0 else None
        out[name] = {"ms_per_step": ms, "launches": t.iterations, "rays": rays,
                     "mrays_per_s": rays / (ms / 1e3) / 1e6 if ms > 0 else None,
                     "bytes_per_ray": bpr, "achieved_gbps": ach,
                     "frac_of_hbm": ach / peak if ach else None,
                     "share_of_stage_time": ms / total if total else None}
    # The second is one interval: scenes with flames run all three in it.
    for name, ms in (("wfStart", t.start_ms), ("wfFlameScan + wfFlame + wfShade", t.shade_a_ms),
                     ("wfLate", t.shade_b_ms)):
        out[name] = {"ms_per_step": ms, "share_of_stage_time": ms / total if total else None}
    prof = profile_figures("wf_trace_l2_issue_%s.md" % workload) if workload else {}
    if prof:
        tr = out["wfTraceFetch"]
        if "l2_bytes_per_ray" in prof and tr["ms_per_step"]:
            tr["l2_gbps"] = prof["l2_bytes_per_ray"] * tr["rays"] / (tr["ms_per_step"] / 1e3) / 1e9
        for k in ("l2_bytes_per_ray", "l2_hit_rate_pct", "issue_slot_util_pct",
                  "lanes_per_instruction", "warps_active_pct"):
            if k in prof:
                tr[k] = prof[k]
        tr["ncu_summary"] = "profiles/wf_trace_l2_issue_%s.md" % workload
    l2 = l2_copy_gbps(stream)
    out["l2_copy_peak_gbps"] = l2
    tr = out["wfTraceFetch"]
    if tr.get("achieved_gbps"):
        tr["algorithmic_frac_of_l2"] = tr["achieved_gbps"] / l2
    if tr.get("l2_gbps"):
        tr["frac_of_l2"] = tr["l2_gbps"] / l2
    out["iterations"] = t.iterations
    out["note"] = ("per-stage CUDA events in one extra render after the timed steps; "
                   "bytes per ray on the walked BVH (32 B per child box tested), radiance and "
                   "shadow rays counted apart")
    return out


# ---- CPU baseline (oracle on the host cores) ------------------------------------------

def oracle_missing():
    """Why the oracle cannot derive a scene here, or None: its scene code is
    built from the reference's sources, which have to be mounted once."""
    from oracle import oracle
    try:
        oracle.ref_scene_lib()
    except oracle.SceneCodeMissing as e:
        return str(e)
    return None


def oracle_sample(scene, base_dir, args, seconds, threads):
    """Render a band of rows of the same frame with the CPU oracle."""
    from oracle import oracle
    # The scene as sundog's own scene code derives it (oracle/_ref), so the
    # CPU arm loads nothing of this library.
    text, r = oracle.reference_scene_text(scene, base_dir, width=args.width, height=args.height,
                                          spp=args.spp)
    osc = oracle.OracleScene(text)
    W, H, spp = r["width"], r["height"], r["spp"]
    # calibrate on one row
    t0 = time.perf_counter()
    _, rays0, _, _ = osc.render(0, H // 2, W, 1, 0, spp, threads=threads)
    dt = max(time.perf_counter() - t0, 1e-3)
    rows = int(max(1, min(H, seconds / dt)))
    y0 = max(0, H // 2 - rows // 2)
    t0 = time.perf_counter()
    _, rays, _, _ = osc.render(0, y0, W, rows, 0, spp, threads=threads)
    dt = time.perf_counter() - t0
    osc.close()
    return {"value": rays / dt / 1e6, "unit": UNIT, "cores": threads, "kind": "port",
            "sample": "rows %d..%d of the %dx%d frame at %d spp (%d paths, %d rays, %.1f s)"
                      % (y0, y0 + rows - 1, W, H, spp, rows * W * spp, rays, dt)}, rays, dt


def run_reference(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return 0
    why = oracle_missing()
    if why:
        print(json.dumps({"impl": "reference", "unavailable": why}), flush=True)
        return 0
    desc, published = resolve_workload(args)
    scene = make_scene(args)
    threads = os.cpu_count() or 1
    per_step = max(2.0, min(args.cpu_seconds, 240.0 / max(args.steps + args.warmup, 1)))
    for _ in range(args.warmup):
        oracle_sample(scene, asset_dir(), args, per_step / 4, threads)
    vals, rays_all, t_all, last = [], 0, 0.0, None
    for _ in range(args.steps):
        cb, rays, dt = oracle_sample(scene, asset_dir(), args, per_step, threads)
        rays_all += rays
        t_all += dt
        last = cb
    value = rays_all / t_all / 1e6
    last["value"] = value
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1000.0 * t_all / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic" if not args.scene else "sundog gallery scene (recorded call stream)",
            "impl": "reference",
            "config": {"workload": desc, "width": args.width, "height": args.height,
                       "spp": args.spp},
            "cpu_baseline": last,
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


# ---- ranks ---------------------------------------------------------------------------------

def shard_plan(rank, world, spp):
    """Rank's part of the job: the 64x64 film tiles t with t % world == rank
    of one frame of spp x world samples (sundog_render_ext shard_count /
    shard_index). Weak scaling: every rank traces about the one-GPU frame's
    paths. No data-path collective; the disjoint films are gathered once after
    the timed steps, into the frame a single GPU would render bit for bit."""
    return {"shard_count": world if world > 1 else 0, "shard_index": rank, "spp": spp * world}


def reduce_max_sum(dist, device, t_max, *sums):
    """Whole-job figures over ranks: the slowest rank's time, summed counts."""
    if dist is None:
        return (t_max,) + tuple(float(x) for x in sums)
    import torch
    t = torch.tensor([float(t_max)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    c = torch.tensor([float(x) for x in sums], dtype=torch.float64, device=device)
    dist.all_reduce(c, op=dist.ReduceOp.SUM)
    return (float(t.item()),) + tuple(float(x) for x in c.tolist())


# ---- our arm ------------------------------------------------------------------------------

def run_ours(args):
    import torch
    from sundog_b200 import abi, build
    from sundog_b200 import scene as sc

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                device_id=torch.device("cuda", local))
    if not os.path.isfile(abi.LIB_PATH):
        build.build()
    lib = abi.load()

    desc, published = resolve_workload(args)
    scene = make_scene(args)
    base = asset_dir()
    plan = shard_plan(rank, world, args.spp)
    fspp = plan["spp"]
    ses = sc.Session(scene, base_dir=base, engine=args.engine, shard_count=plan["shard_count"],
                     shard_index=rank, spp=fspp, width=args.width, height=args.height,
                     chunk_spp=args.chunk_spp)
    stream = torch.cuda.current_stream()
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")

    for _ in range(args.warmup):
        ses.render(stream=stream.cuda_stream)

    clocks = ClockSampler(local)
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    clocks.start()
    step_ms, rays, paths, launches, kernel_ms = [], 0, 0, 0, 0.0
    t_wall = time.perf_counter()
    for _ in range(args.steps):
        flush.fill_(1)  # evict L2 between timed steps
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        res = ses.render(stream=stream.cuda_stream)
        e1.record(stream)
        e1.synchronize()
        step_ms.append(e0.elapsed_time(e1))
        rays += res.rays_traced
        paths += res.paths
        launches += res.kernel_launches
        kernel_ms += res.kernel_ms
    torch.cuda.synchronize()
    wall = time.perf_counter() - t_wall
    clk = clocks.stop()
    total_ms, rays_all, paths_all = reduce_max_sum(dist, "cuda", float(sum(step_ms)), rays, paths)
    value = rays_all / (total_ms / 1000.0) / 1e6

    # The frame on every rank: one all-gather of the disjoint tile films
    # (after the timed steps; not part of `value`).
    gather_ms = None
    if dist:
        from sundog_b200 import shard
        film = shard.session_film(ses)
        torch.cuda.synchronize()
        dist.barrier()
        g0 = torch.cuda.Event(enable_timing=True)
        g1 = torch.cuda.Event(enable_timing=True)
        g0.record(stream)
        shard.gather(film, world)
        g1.record(stream)
        g1.synchronize()
        gather_ms, = reduce_max_sum(dist, "cuda", g0.elapsed_time(g1))

    line = None
    roofline, st = None, ses.stats
    if rank == 0:
        rad, shd = abi.TraceCounts(), abi.TraceCounts()
        abi.check(lib.sundog_session_trace_counts_split(ses.handle, ctypes.byref(rad),
                                                        ctypes.byref(shd)), "counts", lib)
        counts = sum_counts(rad, shd)
        bpr = bytes_per_ray(counts)
        # Roofline unit: one chunk of samples (one persistent launch, or one
        # wavefront pass over the chunk's paths), timed by the session's events.
        kernel_launches = max(1, -(-fspp // max(st.chunk_spp, 1)))  # chunks per step
        mean_launch_ms = kernel_ms / (args.steps * kernel_launches)
        rays_per_launch = rays / (args.steps * kernel_launches)
        achieved = bpr * rays_per_launch / (mean_launch_ms / 1000.0) / 1e9
        peak, peak_kind = measured_peaks()
        per_path = ncu_traffic_per_path(args.engine)
        paths_per_launch = paths / args.steps / kernel_launches
        traffic = per_path * paths_per_launch if per_path is not None else None
        roofline = {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                    "frac": achieved / peak, "traffic": traffic,
                    "peak_source": peak_kind,
                    "bytes_per_ray": bpr,
                    "counts_per_ray": {"box_tests": counts.box_tests / counts.rays,
                                       "tri_tests": counts.tri_tests / counts.rays,
                                       "quadric_tests": counts.quadric_tests / counts.rays,
                                       "blas_entries": counts.blas_entries / counts.rays},
                    "simt": {"traversal_lanes_per_iter": counts.trav_lanes / max(counts.trav_iters, 1),
                             "path_loop_lanes_per_iter": counts.loop_lanes / max(counts.loop_iters, 1),
                             "traversal_iters_per_ray": 32.0 * counts.trav_iters / max(counts.rays, 1)},
                    "note": "algorithmic bytes on the walked BVH (4-wide nodes; 32 B per child "
                            "box tested, 36 B/tri, 48 B/quadric, 64 B/instance) per chunk of "
                            "samples (one persistent launch "
                            "or one wavefront pass) over its CUDA-event duration; the BVH (<4 MB) "
                            "and env tables are cache-resident, so HBM is a loose bound"}
        if args.engine != 1:
            # ncu summaries exist for the configs' own workloads at their sizes
            # (the L2 bytes per ray are per ray, independent of the frame size).
            prof = None if args.scene else "config%d" % args.config
            roofline["per_kernel"] = stage_roofline(lib, ses, stream, flush, rad, shd, peak, prof)
    # The timed session's device memory goes back before the end-to-end calls,
    # which then run as a one-shot caller's would.
    ses.close()

    # End to end through the public API with host buffers, every rank its
    # own tile shard (asset load, CDF + BVH build, upload, render, film
    # download inside the timed call); whole job = slowest rank, summed rays.
    e2e = None
    if not args.no_e2e:
        def e2e_run(keep):
            """Calls of sundog_render_ex from the scene handle; keep = the
            device-memory cache (off: every call allocates and frees all its
            device buffers, the library's default)."""
            abi.check(lib.sundog_set_device_memory_cache(1 if keep else 0), "cache", lib)
            h = scene.build(base, lib)
            try:
                film = np.zeros((args.height, args.width, 4), np.float32)
                o = abi.options(quiet=True, spp=fspp, width=args.width, height=args.height)
                ext = abi.RenderExt(film.ctypes.data, None, None, 0, 1, 0, 0, 0, args.engine,
                                    plan["shard_count"], rank)
                rr = abi.RenderResult()
                abi.check(lib.sundog_render_ex(h, ctypes.byref(o), ctypes.byref(ext),
                                               ctypes.byref(rr)), "render_ex", lib)  # warm
                h0, d0 = ctypes.c_uint64(), ctypes.c_uint64()
                lib.sundog_transfer_bytes(ctypes.byref(h0), ctypes.byref(d0))
                # Up to 5 calls: a single slow driver call (tens to hundreds of
                # ms, at random on this hardware) then moves the mean less.
                e_steps = max(1, min(args.steps, 5))
                if dist:
                    dist.barrier()
                t0 = time.perf_counter()
                erays = 0
                calls = []
                for _ in range(e_steps):
                    tc = time.perf_counter()
                    abi.check(lib.sundog_render_ex(h, ctypes.byref(o), ctypes.byref(ext),
                                                   ctypes.byref(rr)), "render_ex", lib)
                    calls.append(1000.0 * (time.perf_counter() - tc))
                    erays += rr.rays_traced
                et = time.perf_counter() - t0
                h1, d1 = ctypes.c_uint64(), ctypes.c_uint64()
                lib.sundog_transfer_bytes(ctypes.byref(h1), ctypes.byref(d1))
            finally:
                lib.sundog_scene_destroy(h)
                abi.check(lib.sundog_set_device_memory_cache(0), "cache", lib)
            et, erays, hb, db = reduce_max_sum(dist, "cuda", et, erays, h1.value - h0.value,
                                               d1.value - d0.value)
            return {"value": erays / et / 1e6, "unit": UNIT,
                    "h2d_bytes_per_step": int(hb / e_steps),
                    "d2h_bytes_per_step": int(db / e_steps),
                    "ms_per_step": 1000.0 * et / e_steps,
                    "last_call_ms": {"load": rr.load_ms, "build": rr.build_ms,
                                     "render": rr.render_ms, "total": rr.total_ms},
                    "call_ms": {"min": min(calls), "median": float(np.median(calls)),
                                "max": max(calls)}}
        plain = e2e_run(False)
        e2e = e2e_run(True)
        e2e["path"] = ("sundog_set_device_memory_cache(1) once, then sundog_render_ex per step "
                       "and rank: OBJ/HDR load, CDF + BVH build on the device, upload, render, "
                       "film download (the per-sample buffer and path pool kept between calls); "
                       "slowest rank")
        e2e["default_memory_settings"] = {
            "value": plain["value"], "ms_per_step": plain["ms_per_step"],
            "last_call_ms": plain["last_call_ms"], "call_ms": plain["call_ms"],
            "note": "the library's default: every device buffer allocated and freed inside "
                    "each call, as the reference's render does"}

    if rank == 0:
        cpu = None
        if not args.no_cpu_baseline:
            why = oracle_missing()
            if why:
                cpu = {"unavailable": why}
            else:
                cpu, _, _ = oracle_sample(scene, base, args, args.cpu_seconds,
                                          os.cpu_count() or 1)
        line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
                "steps": args.steps, "warmup": args.warmup,
                "ms_per_step": total_ms / args.steps, "higher_is_better": True,
                "scaling": "weak",
                "vs_baseline": value / published[0] if published and world == 1 else None,
                "published_reference": {"mrays_per_s": published[0], "source": published[1],
                                        "hardware": "GB200 (no RT cores: OptiX software "
                                                    "traversal), sundog's own build"}
                if published else None,
                "dtype": "f32", "data": "synthetic" if not args.scene else
                "sundog gallery scene (recorded call stream)",
                "config": {"workload": desc, "width": args.width, "height": args.height,
                           "spp": args.spp, "paths_per_step": int(paths_all / args.steps),
                           "l2": "flushed between steps (256 MiB write); BVH + env tables "
                                 "re-fetched each step",
                           "parallelism": ("dp%d: rank r renders the 64x64 tiles t with t %% %d == r "
                                           "of one %d-spp frame" % (world, world, fspp))
                                          if world > 1 else "dp1 (whole frame)",
                           "grid": st.grid, "block": st.block, "chunk_spp": st.chunk_spp,
                           "engine": ["automatic (wavefront)", "megakernel",
                                      "wavefront"][args.engine]},
                "samples_per_sec": paths_all / (total_ms / 1000.0) if total_ms else None,
                "film_gather_ms": gather_ms,
                "wall_s": wall,
                "gpu_launches": launches,
                "roofline": roofline,
                "cpu_baseline": cpu,
                "e2e": e2e,
                "clocks": clk}
    if dist:
        dist.barrier()
        dist.destroy_process_group()
    if line is not None:
        print(json.dumps(line), flush=True)
    return 0


# ---- learned guiding: equal-time relMSE ------------------------------------------------

def _relmse(img, ref):
    img = img[..., :3].astype(np.float64)
    ref = ref[..., :3].astype(np.float64)
    e = (img - ref) ** 2 / (ref ** 2 + 1e-2)
    return float(e.mean()), e.mean(axis=-1)


def run_guiding(args):
    """Learned guiding against a 16384-spp plain render of the same scene, by
    default the instancing config's 1024-instance field under the sun-and-sky
    env map at its 1920x1080 and 64 spp (or the volumes config's flame / water
    / glass scene at its 2560x1440 and 256 spp). Rare
    high-energy paths make one render's relMSE too noisy to rank two methods:
    each method renders the frame with K seeds, and its error at a given time
    is its mean relMSE over the seeds scaled by (its render time / that time)
    -- MSE falls as 1 / samples for an unbiased estimator. The guided time
    includes online training on the first 32 spp. `value` = equal-time relMSE
    ratio plain / guided over the whole image. Beside it: the same ratio over
    the image's bulk (per seed, the pixels below the 99th percentile of the
    larger of the two methods' errors) and of the median pixel error, and
    how much of the plain error sits in the top 0.1% of pixels and in those
    of them whose error is the same in both renders to 1% (one sample,
    drawn before any guided vertex, dominates both). Prints one JSON line."""
    from sundog_b200 import scene as sc
    from sundog_b200 import workloads
    if int(os.environ.get("RANK", "0")) != 0:
        return 0
    dw, dh, dspp = (2560, 1440, 256) if args.guide_scene == "volumes" else (1920, 1080, 64)
    w, h = args.guide_width or dw, args.guide_height or dh
    spp, ref_spp, seeds = args.guide_spp or dspp, args.guide_ref_spp, args.guide_seeds
    ad = asset_dir()
    if args.guide_scene == "volumes":
        make = lambda n: workloads.volumes(ad, width=w, height=h, spp=n)
        desc = ("flame + water + nested glass + rough panels + 2048-tri mesh light, %dx%d "
                "(the volumes config's scene)" % (w, h))
    else:
        make = lambda n: workloads.instancing(ad, width=w, height=h, spp=n)
        desc = ("1024 displaced icosphere instances, Lambert / metal / plastic, sun-and-sky "
                "env map, %dx%d (the instancing config's scene)" % (w, h))
    with sc.Session(make(ref_spp), base_dir=ad, seed=1000) as r:
        rr = r.render()
        ref = r.read()[..., :3].astype(np.float64)
    den = ref ** 2 + 1e-2
    s = make(spp)
    out, maps = {}, {}
    for name, guided in (("plain", False), ("guided", True)):
        errs, ms, kms, train_ms, rays, emaps = [], [], [], [], [], []
        for k in range(seeds):
            with sc.Session(s, base_dir=ad, seed=1 + k) as ses:
                if guided:
                    ses.set_guiding(True)
                if k == 0:
                    ses.render()  # warm-up: module load, first touch
                res = ses.render()
                img = ses.read()[..., :3].astype(np.float64)
                if guided:
                    train_ms.append(ses.guiding_stats().train_ms)
            em = ((img - ref) ** 2 / den).mean(-1)
            emaps.append(em)
            errs.append(float(em.mean()))
            ms.append(res.render_ms)
            kms.append(res.kernel_ms)
            rays.append(res.rays_traced)
        maps[name] = emaps
        out[name] = {"relmse_per_seed": errs, "relmse": float(np.mean(errs)),
                     "ms": float(np.mean(ms)), "path_kernel_ms": float(np.mean(kms)),
                     "rays": float(np.mean(rays))}
        if guided:
            out[name]["train_ms"] = float(np.mean(train_ms))
    bulk = {"plain": [], "guided": []}
    med = {"plain": [], "guided": []}
    for k in range(seeds):
        both = np.maximum(maps["plain"][k], maps["guided"][k])
        keep = both <= np.quantile(both, 0.99)
        for name in bulk:
            bulk[name].append(float(maps[name][k][keep].mean()))
            med[name].append(float(np.median(maps[name][k])))
    for name in bulk:
        out[name]["relmse_bulk"] = float(np.mean(bulk[name]))
        out[name]["median_pixel_relmse"] = float(np.mean(med[name]))
    ep, eg = maps["plain"][0], maps["guided"][0]
    top = ep >= np.quantile(ep, 0.999)
    shared = top & (np.abs(ep - eg) <= 0.01 * ep)
    p, g = out["plain"], out["guided"]
    tr = g["ms"] / p["ms"]
    line = {
        "metric": "equal-time relMSE ratio plain / guided",
        "value": p["relmse"] / (g["relmse"] * tr),
        "unit": "x", "higher_is_better": True, "n_gpus": 1,
        "dtype": "f32 render, bf16 network", "data": "synthetic",
        "config": {"workload": desc, "scene": args.guide_scene, "width": w, "height": h,
                   "spp": spp, "seeds": seeds, "reference_spp": ref_spp,
                   "relmse": "mean over pixels of (x - ref)^2 / (ref^2 + 0.01), RGB mean",
                   "equal_time": "relMSE x render time (MSE ~ 1/time for unbiased estimators)",
                   "bulk": "per seed, pixels below the 99th percentile of max(plain, guided) error"},
        "equal_spp_ratio": p["relmse"] / g["relmse"],
        "time_ratio": tr,
        "bulk_equal_time_ratio": p["relmse_bulk"] / (g["relmse_bulk"] * tr),
        "bulk_equal_spp_ratio": p["relmse_bulk"] / g["relmse_bulk"],
        "median_pixel_equal_time_ratio": p["median_pixel_relmse"] / (g["median_pixel_relmse"] * tr),
        "plain_error_in_top_0.1pct_pixels": float(ep[top].sum() / ep.sum()),
        "plain_error_in_top_pixels_shared_by_both": float(ep[shared].sum() / ep.sum()),
        "plain": p, "guided": g, "reference_ms": rr.render_ms,
    }
    print(json.dumps(line))
    return 0


# ---- serving: Poisson-arriving jobs, continuous batching ----------------------------------

def run_serving(args):
    """Render server under Poisson arrivals (default rate 20/s, seed 5): each job
    draws a scene from the Cornell / instancing / volumes configs, a square
    resolution log-uniform in 256..2048 and spp log-uniform in 4..256, and is
    submitted at its arrival time; the server batches 64x64 tile-passes of all
    admitted jobs into each persistent launch. Reports p50 / p99 job latency
    (submission -> film on the host) and aggregate Mrays/s over the run; then
    renders every job alone on a fresh server for its slowdown in the mix
    (latency in the mix / latency alone), and gives the server's capacity
    (camera paths per busy second) and the arrival rate it sustains (capacity
    / mean paths per job). Prints one JSON line."""
    from sundog_b200 import serve, workloads
    if int(os.environ.get("RANK", "0")) != 0:
        return 0
    ad = asset_dir()
    scenes = [workloads.cornell(), workloads.instancing(ad), workloads.volumes(ad)]
    rng = np.random.default_rng(5)
    n = args.serve_jobs
    gaps = rng.exponential(1.0 / args.serve_rate, n)
    arrivals = np.cumsum(gaps) - gaps[0]
    kinds = rng.integers(0, 3, n)
    sides = np.exp(rng.uniform(np.log(256), np.log(2048), n)).astype(int)
    spps = np.exp(rng.uniform(np.log(4), np.log(256), n)).round().astype(int)
    work = [(int(k), int(w), int(p)) for k, w, p in zip(kinds, sides, spps)]
    # Warm-up: every scene once (module load, scene builds), then a fresh
    # server for the timed run so no scene is resident when it starts.
    cfg = {"engine": args.serve_engine}
    if args.serve_batch > 0:
        cfg["iteration_paths"] = args.serve_batch
    with serve.Server(**cfg) as sv:
        for s in scenes:
            sv.submit(s, base_dir=ad, width=64, height=64, spp=1, film=False).wait()
    sampler = ClockSampler(int(os.environ.get("LOCAL_RANK", "0")))
    sampler.start()
    with serve.Server(**cfg) as sv:
        t0 = time.perf_counter()
        jobs = []
        for (k, side, spp), at in zip(work, arrivals):
            delay = t0 + at - time.perf_counter()
            if delay > 0:
                time.sleep(delay)
            jobs.append(sv.submit(scenes[k], base_dir=ad, width=side, height=side, spp=spp,
                                  seed=1 + len(jobs)))
        lat, queued, failed = [], [], 0
        for j in jobs:
            try:
                j.wait()
            except serve.JobError:
                failed += 1
            lat.append(j.last.latency_ms)
            queued.append(j.last.queued_ms)
            j.film = None
        wall = time.perf_counter() - t0
        st = sv.stats()
    clocks = sampler.stop()
    # Each job alone on an idle server, in arrival order: its latency in the
    # mix over its latency alone is the slowdown the other jobs caused.
    alone = []
    with serve.Server(**cfg) as sv:
        for i, (k, side, spp) in enumerate(work):
            j = sv.submit(scenes[k], base_dir=ad, width=side, height=side, spp=spp, seed=1 + i)
            try:
                j.wait()
            except serve.JobError:
                pass
            alone.append(j.last.latency_ms)
            j.film = None
    slow = np.array(lat) / np.maximum(np.array(alone), 1e-3)
    capacity = st.paths / (st.busy_ms / 1e3) if st.busy_ms else None
    mean_job_paths = float(np.mean([side * side * spp for _, side, spp in work]))
    paths_total = sum(side * side * spp for _, side, spp in work)
    line = {
        "metric": "serving: aggregate Mrays/s; p50/p99 job latency", "value": st.rays / wall / 1e6,
        "unit": "Mrays/s", "higher_is_better": True, "n_gpus": 1, "dtype": "f32",
        "data": "synthetic",
        "config": {"workload": "Poisson arrivals %g/s (seed 5) of Cornell / instancing / volumes "
                               "jobs, square 256..2048 px and 4..256 spp log-uniform, 64x64 "
                               "tile-passes of 8 spp batched across jobs" % args.serve_rate,
                   "jobs": n, "arrival_rate_per_s": args.serve_rate,
                   "max_jobs": sv.config.max_jobs,
                   "iteration_paths": sv.config.iteration_paths,
                   "engine": ["wavefront", "megakernel", "wavefront"][sv.config.engine]},
        "latency_ms": {"p50": float(np.percentile(lat, 50)), "p99": float(np.percentile(lat, 99)),
                       "mean": float(np.mean(lat)), "max": float(np.max(lat))},
        "queued_ms": {"p50": float(np.percentile(queued, 50)),
                      "p99": float(np.percentile(queued, 99))},
        "jobs_done": st.jobs_done, "jobs_failed": failed,
        "wall_s": wall, "gpu_busy_s": st.busy_ms / 1e3,
        "busy_mrays_per_s": st.rays / (st.busy_ms / 1e3) / 1e6 if st.busy_ms else None,
        "samples_per_sec": st.paths / wall,
        "offered_paths_per_s": paths_total / float(arrivals[-1] if n > 1 else 1.0),
        "capacity_paths_per_s": capacity,
        "sustainable_rate_per_s": capacity / mean_job_paths if capacity else None,
        "alone_latency_ms": {"p50": float(np.percentile(alone, 50)),
                             "p99": float(np.percentile(alone, 99))},
        "slowdown_vs_alone": {"p50": float(np.percentile(slow, 50)),
                              "p99": float(np.percentile(slow, 99)),
                              "max": float(np.max(slow))},
        "per_job": [{"scene": ["cornell", "instancing", "volumes"][k], "side": side, "spp": spp,
                     "arrival_ms": round(1e3 * float(at), 1), "latency_ms": round(l, 1),
                     "queued_ms": round(q, 1), "alone_ms": round(a, 1)}
                    for (k, side, spp), at, l, q, a in zip(work, arrivals, lat, queued, alone)],
        "iterations": st.iterations, "scenes_resident_at_end": st.scenes_resident,
        "clocks": clocks,
    }
    print(json.dumps(line))
    return 0


def main():
    args = parse_args()
    if args.impl == "reference":
        return run_reference(args)
    if args.guiding:
        return run_guiding(args)
    if args.serving:
        return run_serving(args)
    return run_ours(args)


if __name__ == "__main__":
    sys.exit(main())
