#!/usr/bin/env python
"""Benchmark: 1080p HEVC motion estimation on B200.

Workload (one step): a 1080p 8-bit HEVC sequence of 62 synthetic pictures
(sinusoids + noise, 64x64-region motion in +-40 px at quarter samples,
sigma-2 noise), of which the last 60 are searched, each against the two
pictures before it: 2Nx2N prediction units 8x8..64x64 (42,900 per
reference), +-64 whole-sample search, half- then quarter-sample SATD
refinement, lambda at QP 32 (medium tier: no widening rings, Tune::lambda
0.85), STANDALONE predictors. A step rebuilds the search planes of the 60
new references (HalfPlanes::new's work) and searches the 60 frames in one
persistent launch (the batched form). The working set (62 pictures x 16
planes, 2.6 GB) is far larger than L2, so no flush is needed between steps.

Lines printed (one JSON line each; rank 0 only):
  default            the batched form: value = frames/s on the device with
                     inputs resident; e2e = the same through the C ABI from
                     pinned host memory (uploads + plane builds + search +
                     results back inside the timed region, two steps in
                     flight); the plain
                     per-frame path (one frame per call) beside it, p50/p99.
                     `served`: the serving loop under Poisson load (30 fps
                     streams, 20..120 % of the batched capacity), p50/p99
                     per-frame latency per load.
  --impl reference   the reference's CPU path on the host cores: the
                     oracle's C++ restatement (AVX2 distortion rungs), since
                     the Rust crate cannot be built here.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

WIDTH, HEIGHT, NFRAMES, NREF, QP, RANGE = 1920, 1080, 60, 2, 32, 64
# The headline metric as stated for this path; `value` is the batched
# persistent launch the serving loop runs (its capacity), with the served
# sweep and the plain per-frame path (p50/p99) beside it in the same line.
METRIC = "1080p HEVC ME frames/s served vs plain per-frame GPU; p99 latency; bit-exact"


def log(*a):
    print(*a, file=sys.stderr, flush=True)


class ClockSampler:
    """nvidia-smi clocks and throttle reasons, sampled every 200 ms."""
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu: int):
        self.gpu, self.proc, self.lines = gpu, None, []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            threading.Thread(target=self._read, daemon=True).start()
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *exc):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self) -> dict:
        sm, mx, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx = max(mx, float(parts[2]))
            except ValueError:
                continue
            for name, v in zip(names, parts[5:9]):
                if v.lower() == "active":
                    reasons.add(name)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": mx or None,
                "reasons": sorted(reasons), "samples": len(sm)}


def make_workload(rank: int):
    from rivet_h26x_codecs_b200 import synth
    seq = synth.make_sequence(synth.HEVC, WIDTH, HEIGHT, 8, NFRAMES + NREF, synth.seed_for(1, rank), 64, 160, 2.0)
    return seq.frames


def hevc_params(oracle_mod=None):
    import rivet_h26x_codecs_b200.capi as capi
    p = capi.default_params(capi.RME_CODEC_HEVC, QP) if oracle_mod is None else oracle_mod.params(capi.RME_CODEC_HEVC, QP)
    p.hevc_search_range = RANGE
    return p


def cpu_model() -> str:
    """The host CPU's model name (/proc/cpuinfo), for the baseline's row."""
    try:
        for line in open("/proc/cpuinfo"):
            if line.startswith("model name"):
                return line.split(":", 1)[1].strip()
    except OSError:
        pass
    return "unknown"


def cpu_baseline(frames, threads: int, simd: int = 1, nframes: int | None = None):
    """The oracle (C++ restatement, AVX2 rungs for SAD, SATD and the HEVC
    interpolation) over `nframes` frames of the sequence (default: one per
    thread) on `threads` host threads. Each reference's phase planes are
    built once, as a streaming encoder builds them once per coded picture
    (retain_reference, h265.rs:1553-1589): about one plane build per frame.
    Returns (frames/s including those builds, frames, seconds, plane-build
    seconds)."""
    sys.path.insert(0, str(ROOT / "oracle"))
    import oracle
    import rivet_h26x_codecs_b200.capi as capi
    n = max(1, min(nframes or threads, len(frames) - NREF))
    srcs = [frames[NREF + i] for i in range(n)]
    refs = [[frames[NREF + i - 1 - r] for r in range(NREF)] for i in range(n)]
    p = hevc_params(oracle)
    _, secs, plane_secs = oracle.frames_search_mt(capi.RME_CODEC_HEVC, 8, srcs, refs, p, simd=simd, threads=threads)
    return n / secs, n, secs, plane_secs


def dist_setup(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import datetime

        import torch
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300),
                                device_id=torch.device("cuda", local))
    return world, rank, local


def max_over_ranks(x: float, world: int, device: str = "cuda") -> float:
    """The slowest rank's time: replicas are timed as a whole job."""
    if world == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def barrier(world: int, device: str = "cuda"):
    if world > 1:
        import torch
        import torch.distributed as dist
        dist.barrier()
        if device == "cuda":
            torch.cuda.synchronize()


def job_rate(world: int, frames_per_step: int, steps: int, seconds: float) -> float:
    """Whole-job frames/s: every rank searches its own frames (weak scaling)."""
    return world * frames_per_step * steps / seconds


def run_reference(args, world, rank):
    """The reference arm: the CPU restatement of the search on every host
    thread, each step the whole workload of our arm's step (the 60 frames of
    the 1080p sequence, each against its two previous pictures)."""
    if rank != 0:
        return
    frames = make_workload(0)
    threads = os.cpu_count() or 1
    nframes = min(args.ref_frames or NFRAMES, NFRAMES)
    for _ in range(args.warmup):
        cpu_baseline(frames, threads, nframes=nframes)
    t0 = time.perf_counter()
    done, plane_s = 0, 0.0
    for _ in range(args.steps):
        _, n, _, ps = cpu_baseline(frames, threads, nframes=nframes)
        done += n
        plane_s += ps
    secs = time.perf_counter() - t0
    fps = done / secs
    sample = (f"{done // args.steps} frames of the 1080p workload per step on {threads} host threads, AVX2 rungs "
              f"(SAD, SATD, HEVC interpolation), each reference's planes built once "
              f"({plane_s / secs * 100:.0f} % of the time)")
    print(json.dumps({
        "impl": "reference", "metric": METRIC, "value": fps, "unit": "frames/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": secs / args.steps * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u8", "data": "synthetic",
        "config": workload_config(done // args.steps, world),
        "cpu_baseline": {"value": fps, "unit": "frames/s", "cores": threads, "kind": "port", "cpu_model": cpu_model(),
                         "sample": sample, "plane_build_s_per_step": plane_s / args.steps},
        "e2e": {"value": fps, "unit": "frames/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }), flush=True)


def plain_latency(ms, frames, p, stream, nframes: int = 600, warm: int = 8) -> dict:
    """The plain per-frame path as an encoder drives it, one picture at a
    time: each timed call uploads the new picture from pinned host memory
    (its planes built on the device), searches it against the two pictures
    before it, and reads its results back into a pinned buffer the caller
    keeps. `nframes` calls over the sequence (cycled), after `warm` untimed
    ones; p50/p99 over the timed calls (host clock around the whole call)."""
    import torch
    import rivet_h26x_codecs_b200.capi as capi
    ring = 4  # picture slots: the new picture, its two references and one spare
    pinned = []
    for f in frames:
        t = torch.empty(f.shape, dtype=torch.uint8, pin_memory=True)
        t.numpy()[...] = f
        pinned.append(t.numpy())
    base = 5000
    for k in range(NREF):
        ms.upload(base + k, pinned[k], capi.RME_CODEC_HEVC, 8, as_ref=True, stream=stream)
    n = ms.result_count(base, [base + r for r in range(NREF)], p)
    bufs = []
    for _ in range(2):
        b = torch.empty(n * capi.RESULT_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)
        b.fill_(1)
        bufs.append(b.numpy().view(capi.RESULT_DTYPE))
    lat = []
    for i in range(NREF, NREF + warm + nframes):
        slot = base + i % ring
        refs = [base + (i - 1 - r) % ring for r in range(NREF)]
        a = time.perf_counter()
        ms.upload(slot, pinned[i % len(frames)], capi.RME_CODEC_HEVC, 8, as_ref=True, stream=stream)
        ms.search(slot, refs, p, stream=stream, out=bufs[i & 1])
        if i >= NREF + warm:
            lat.append(time.perf_counter() - a)
    for k in range(ring):
        ms.release(base + k)
    lat_ms = np.array(lat) * 1e3
    return {"value": len(lat) / float(np.sum(lat)), "unit": "frames/s", "frames": len(lat),
            "p50_ms": float(np.percentile(lat_ms, 50)), "p99_ms": float(np.percentile(lat_ms, 99)),
            "max_ms": float(lat_ms.max()),
            "call": "upload from pinned memory + plane build + search + results to pinned memory, one picture a call"}


def workload_config(frames_per_step: int, world: int) -> dict:
    """The bench's workload, named by what it is (both arms report it)."""
    return {"workload": "hevc-1080p-8bit-2ref-pu8to64-range64-qp32", "frames_per_step": frames_per_step,
            "width": WIDTH, "height": HEIGHT, "refs": NREF, "predictors": "standalone",
            "parallelism": f"replicas{world}", "l2": "inputs larger than L2 (2.6 GB of planes)"}


def run_ours(args, world, rank, local):
    import torch

    import rivet_h26x_codecs_b200 as rme
    import rivet_h26x_codecs_b200.capi as capi

    peaks = {}
    try:
        peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text())
    except (OSError, ValueError):
        pass
    t0 = time.perf_counter()
    frames = make_workload(rank)
    log(f"[rank {rank}] workload generated in {time.perf_counter() - t0:.1f}s")
    ms = rme.MotionSearch(local)
    p = hevc_params()
    ids = list(range(len(frames)))
    for i, f in zip(ids, frames):
        ms.upload(i, f, capi.RME_CODEC_HEVC, 8, as_ref=True)
    batch = [(t, [t - 1 - r for r in range(NREF)]) for t in range(NREF, len(frames))]
    stream = torch.cuda.Stream(device=local)
    sh = stream.cuda_stream

    # Results stay in device memory in the device-resident step.
    total = ms.batch_result_count(batch, p)
    dev_out = torch.empty(total * capi.RESULT_DTYPE.itemsize, dtype=torch.uint8, device=f"cuda:{local}")

    def step():
        for t, _ in batch:
            ms.build_planes(t, sh)
        return ms.search_batch(batch, p, sh, out=dev_out)

    def as_host(views):
        return [v.cpu().numpy().view(capi.RESULT_DTYPE) for v in views]

    # ---- plain per-frame GPU path (one frame per call) -----------------------
    # Each frame's results go to a buffer the caller keeps (as an encoder
    # keeps its motion field) in pinned memory, which the results' copy
    # fills directly; touched before the timing.
    # Warm-up: the first launches of this size allocate the buffers.
    for _ in range(18):
        ms.search(batch[0][0], batch[0][1], p, stream=sh)
    per_frame = ms.result_count(batch[0][0], batch[0][1], p)
    plain_bufs = []
    for _ in batch:
        b = torch.empty(per_frame * capi.RESULT_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)
        b.fill_(1)
        plain_bufs.append(b.numpy().view(capi.RESULT_DTYPE))
    lat = []
    plain_out = []
    for (t, refs), buf in zip(batch, plain_bufs):
        a = time.perf_counter()
        plain_out.append(ms.search(t, refs, p, stream=sh, out=buf))
        lat.append(time.perf_counter() - a)
    plain_fps = len(batch) / sum(lat)

    # ---- batched, device-resident -------------------------------------------
    # Warm-up: a launch's CUDA graph is captured the second time its shape
    # comes; a few more steps settle it before timing.
    warm = max(args.warmup, 3) + 5
    for _ in range(warm):
        outs = step()
    outs = as_host(outs)
    for o, q in zip(outs, plain_out):
        if not (o == q).all():
            raise SystemExit("batched results differ from the per-frame path")
    stats = ms.stats()
    kernel_ms_list = []
    barrier(world)
    torch.cuda.synchronize()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(local) as clk:
        ev0.record(stream)
        for _ in range(args.steps):
            step()
            kernel_ms_list.append(ms.stats().kernel_ms)
        ev1.record(stream)
        torch.cuda.synchronize()
    elapsed = ev0.elapsed_time(ev1) / 1e3
    barrier(world)
    elapsed = max_over_ranks(elapsed, world)
    frames_per_step = len(batch)
    value = job_rate(world, frames_per_step, args.steps, elapsed)
    clocks = clk.summary()

    # ---- end to end through the C ABI from pinned host memory --------------------
    pinned = []
    for f in frames:
        t = torch.empty(f.shape, dtype=torch.uint8, pin_memory=True)
        t.numpy()[...] = f
        pinned.append(t)
    h2d = sum(int(f.nbytes) for f in frames)
    d2h = sum(int(o.nbytes) for o in outs)
    rbytes = total * capi.RESULT_DTYPE.itemsize
    host_out = [torch.empty(rbytes, dtype=torch.uint8, pin_memory=True) for _ in range(2)]
    dev_out = [torch.empty(rbytes, dtype=torch.uint8, device=f"cuda:{local}") for _ in range(2)]

    # A pipeline of two steps in flight. The uploads alternate between two
    # streams, so one picture's copy runs while the previous picture's planes
    # are built; the search waits for both. (The previous step's search has
    # returned, so nothing still reads the pictures being refilled.) Each
    # step's results stay in one of two device buffers and are read back to
    # pinned memory on a copy stream while the next step's uploads run; a
    # search waits for the read-back of the step before last, which used the
    # same buffer. Every step's copies lie inside the timed region, which
    # ends with a device-wide synchronize.
    up = [torch.cuda.Stream(device=local) for _ in range(2)]
    up_done = [torch.cuda.Event() for _ in range(2)]
    cp = torch.cuda.Stream(device=local)
    searched, copied = torch.cuda.Event(), [torch.cuda.Event() for _ in range(2)]
    for e in copied:
        e.record(cp)

    def e2e_step(k):
        b = k & 1
        for j, (i, t) in enumerate(zip(ids, pinned)):
            ms.upload(i, t.numpy(), capi.RME_CODEC_HEVC, 8, as_ref=True, stream=up[j & 1].cuda_stream)
        for u, e in zip(up, up_done):
            e.record(u)
            stream.wait_event(e)
        stream.wait_event(copied[b])
        views = ms.search_batch(batch, p, sh, out=dev_out[b])
        searched.record(stream)
        cp.wait_event(searched)
        with torch.cuda.stream(cp):
            host_out[b].copy_(dev_out[b], non_blocking=True)
        copied[b].record(cp)
        base = dev_out[b].data_ptr()
        return [(b, v.data_ptr() - base, v.numel()) for v in views]

    for k in range(2):
        e2e_step(k)
    torch.cuda.synchronize()
    barrier(world)
    a = time.perf_counter()
    for k in range(args.steps):
        e2e_last = e2e_step(k)
    torch.cuda.synchronize()
    e2e_secs = max_over_ranks(time.perf_counter() - a, world)
    e2e_value = job_rate(world, frames_per_step, args.steps, e2e_secs)
    e2e_out = [host_out[b][o:o + n].numpy().view(capi.RESULT_DTYPE) for b, o, n in e2e_last]
    for o, q in zip(e2e_out, plain_out):
        if not (o == q).all():
            raise SystemExit("end-to-end results differ from the per-frame path")

    # ---- roofline ---------------------------------------------------------------
    st = ms.stats()
    kms = float(np.median(kernel_ms_list)) / 1e3
    int_ops = 2 * st.sad_samples + 7 * st.satd_samples + st.satd_samples // 16
    peak_ops = C_double = None
    import ctypes as C
    C_double = C.c_double()
    if capi.lib().rme_probe_int_peak(local, C.byref(C_double)) == 0:
        peak_ops = C_double.value
    plane_bytes = (WIDTH + 160 + 63) // 64 * 64 * (HEIGHT + 160)  # one padded plane, 8-bit
    alg_bytes = (len(frames) * 16 * plane_bytes + frames_per_step * WIDTH * HEIGHT
                 + sum(int(o.nbytes) for o in outs))
    hbm_peak = peaks.get("hbm_gbs", 6650.0)
    # The search kernel against HBM (the path's byte stream) and, beside it,
    # against the integer pipes; it reaches neither: a data-dependent descent
    # of short dependent steps, latency-bound (see the profiles).
    roof = {
        "bound": "hbm",
        "achieved": alg_bytes / kms / 1e9, "peak": hbm_peak, "unit": "GB/s",
        "frac": alg_bytes / kms / 1e9 / hbm_peak,
        "peak_source": "measured (MEASURED_PEAKS.json hbm_gbs)" if "hbm_gbs" in peaks else "fallback",
        "algorithmic_bytes_per_launch": alg_bytes,
        "kernel_ms": kms * 1e3,
        "traffic": None,
        "int_alu": {"achieved": int_ops / kms / 1e12, "peak": (peak_ops or 0) / 1e12, "unit": "Tops/s",
                    "frac": (int_ops / kms / peak_ops) if peak_ops else None,
                    "peak_source": "measured: rme_probe_int_peak (32-bit add/shift/xor chains, all SMs)",
                    "algorithmic_int_ops_per_launch": int(int_ops)},
        "note": "latency-bound: dependent search steps; neither HBM nor the integer pipes saturate",
    }
    traffic_file = ROOT / "profiles" / "search_kernel_traffic.json"
    if traffic_file.exists():
        try:
            tr = json.loads(traffic_file.read_text())
            roof["traffic"] = tr.get("bytes_per_launch_1080p")
            roof["traffic_source"] = ("scaled from profiles/search_kernel_traffic.json (ncu DRAM bytes of an "
                                      "8-frame launch, times 60/8), not measured in this run")
        except ValueError:
            pass

    # ---- plain per-frame path, one picture a call (upload inside) -------------------
    plain_stream = plain_latency(ms, frames, p, sh)

    # ---- serving loop under load (every rank serves its own streams) ---------------
    served = served_resident = None
    if not args.no_serve:
        served = run_served(frames, value / world, local=local)
        # The resident engine beside it (a shorter sweep: 500 requests a load).
        served_resident = run_served(frames, value / world, rates=(60, 150, 300), min_requests=500, local=local,
                                     resident=True)

    # ---- CPU baseline (bounded sample) ---------------------------------------------
    cpu = None
    others = None
    if rank == 0 and world == 1 and not args.no_serve:
        others = other_configs(local)
    if rank == 0 and world == 1 and not args.no_cpu:
        threads = os.cpu_count() or 1
        fps_all, n_all, secs_all, ps_all = cpu_baseline(frames, threads)
        fps_1, _, _, _ = cpu_baseline(frames, 1)
        cpu = {"value": fps_all, "unit": "frames/s", "cores": threads, "kind": "port",
               "sample": f"{n_all} frames of the workload, one per host thread, AVX2 rungs (SAD, SATD, HEVC "
                         "interpolation), each reference's planes built once",
               "plane_build_share": ps_all / secs_all,
               "value_1_thread": fps_1, "cpu_model": cpu_model()}

    # The headline: the served rate at the highest load kept up with (served
    # >= 0.97 x offered and p99 <= 8 ms), over all ranks; where no load met
    # the rule on every rank, the batched device-resident rate, and the line
    # says which.
    met = served is not None and served["met"]
    if world > 1:
        met = max_over_ranks(0.0 if met else 1.0, world) == 0.0
    served_total = (served["value"] if served else 0.0) * 1.0
    if world > 1:
        import torch
        import torch.distributed as dist
        tt = torch.tensor([served_total], dtype=torch.float64, device="cuda")
        dist.all_reduce(tt)
        served_total = float(tt.item())
    frame_in = WIDTH * HEIGHT
    frame_out = 42900 * NREF * capi.RESULT_DTYPE.itemsize
    if rank == 0:
        lat_ms = np.array(lat) * 1e3
        batched = {"value": value, "unit": "frames/s", "ms_per_step": elapsed / args.steps * 1e3,
                   "frames_per_step": frames_per_step, "timing": "CUDA events over the steps, max over ranks",
                   "e2e": {"value": e2e_value, "unit": "frames/s", "h2d_bytes_per_step": h2d,
                           "d2h_bytes_per_step": d2h}}
        e2e = ({"value": served_total, "unit": "frames/s", "h2d_bytes_per_step": frame_in,
                "d2h_bytes_per_step": frame_out, "step": "one served frame request, through rme_serve_*"}
               if met else batched["e2e"])
        print(json.dumps({
            "metric": METRIC, "value": served_total if met else value, "unit": "frames/s", "n_gpus": world,
            "steps": args.steps,
            "value_is": ("served frames/s at the highest Poisson load with served >= 0.97 x offered and p99 <= 8 ms"
                         if met else "batched device-resident frames/s: no served load met p99 <= 8 ms"),
            "warmup": warm, "ms_per_step": elapsed / args.steps * 1e3, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "u8", "data": "synthetic",
            "config": {"workload": "hevc-1080p-8bit-2ref-pu8to64-range64-qp32", "frames_per_step": frames_per_step,
                       "width": WIDTH, "height": HEIGHT, "refs": NREF, "pus_per_ref": int(stats.tasks // frames_per_step // NREF),
                       "predictors": "standalone", "parallelism": f"replicas{world}",
                       "l2": "inputs larger than L2 (2.6 GB of planes)"},
            "plain_per_frame": plain_stream,
            "plain_per_frame_resident": {"value": plain_fps, "unit": "frames/s", "frames": len(lat),
                                         "p50_ms": float(np.percentile(lat_ms, 50)),
                                         "p99_ms": float(np.percentile(lat_ms, 99)),
                                         "call": "search only, pictures already resident"},
            "batched": batched,
            "pu_cost_evals_per_s": (st.sad_candidates + st.satd_candidates) / kms * world,
            "e2e": e2e,
            "served": served,
            "served_resident_engine": served_resident,
            "other_configs": others,
            "roofline": roof,
            "cpu_baseline": cpu,
            "clocks": clocks,
            "gpu_launches": args.steps * (frames_per_step + 1),
        }), flush=True)
    ms.close()


P99_TARGET_MS = 8.0


# Offered rates of the served sweep (frames/s, 30 a stream), finest around
# the p99 knee; each is reported with its fraction of the batched capacity.
SERVED_RATES = (60, 90, 120, 150, 180, 210, 240, 270, 300, 360, 450, 630)


def run_served(frames, capacity_fps: float, loads=None, min_requests: int = 1000,
               warm_s: float = 0.5, local: int = 0, resident: bool = False, max_batch: int = 2,
               rates=SERVED_RATES) -> dict:
    """The serving loop under Poisson load: streams of the 1080p workload at
    30 frames/s each, the total rate a fraction of the measured batched
    capacity; per-frame latency is submit -> results in the client's buffer
    (host clock, request loop included), over at least `min_requests`
    requests submitted after `warm_s` of the same load. A load is kept up
    with when served >= 0.97 x offered and p99 <= 8 ms; the headline is the
    highest served rate that is. `resident`: the resident engine, else a
    launch per batch of arrivals (at most `max_batch` frames) with launches
    overlapping."""
    import torch
    import rivet_h26x_codecs_b200 as rme
    import rivet_h26x_codecs_b200.capi as capi
    p = hevc_params()
    sweep = []
    rng = np.random.default_rng(2024)
    per_stream = 4  # frames of a stream in flight at once (rme_serve_open_stream)
    count = 42900 * NREF
    points = [(l, l * capacity_fps) for l in loads] if loads is not None else [(r / capacity_fps, r) for r in rates]
    for load, rate in points:
        nstreams = max(1, int(round(rate / 30.0)))
        seconds = max(2.0, min_requests / (nstreams * 30.0))
        with rme.MotionSearch(local) as ms:
            srv = rme.Server(ms, hbm_budget_bytes=120 << 30, max_frames_per_launch=max_batch, max_streams=1024,
                             resident=resident)
            try:
                for sid in range(nstreams):
                    assert srv.open_stream(sid, capi.RME_CODEC_HEVC, 8, WIDTH, HEIGHT, p, NREF) == 0
                # Each stream's client reuses a ring of pinned result buffers
                # (as an encoder reuses its motion field), touched once here.
                bufs = {}
                for sid in range(nstreams):
                    bufs[sid] = []
                    for _ in range(8):
                        t = torch.empty(count * capi.RESULT_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)
                        t.fill_(1)
                        bufs[sid].append(t.numpy().view(capi.RESULT_DTYPE))
                # Fill every stream's picture ring once (allocations, not timed).
                nxt = {}
                for sid in range(nstreams):
                    for t in range(NREF + per_stream):
                        srv.submit(sid, frames[(sid * 7 + t) % len(frames)], out=bufs[sid][t % 8] if t else None)
                    nxt[sid] = NREF + per_stream
                pending = nstreams * (NREF + per_stream)
                while pending:
                    pending -= len(srv.poll())
                    time.sleep(0.0005)
                # Poisson arrivals, 30 frames/s per stream: a warm-up period,
                # then the measured window.
                events = []
                for sid in range(nstreams):
                    t = rng.exponential(1 / 30.0)
                    while t < warm_s + seconds:
                        events.append((t, sid))
                        t += rng.exponential(1 / 30.0)
                events.sort()
                measured, done = set(), []
                t0 = time.perf_counter()
                for at, sid in events:
                    while time.perf_counter() - t0 < at:
                        done += srv.poll()
                        time.sleep(0.0001)
                    rid = srv.submit(sid, frames[(sid * 7 + nxt[sid]) % len(frames)], out=bufs[sid][nxt[sid] % 8])
                    nxt[sid] += 1
                    if at >= warm_s:
                        measured.add(rid)
                deadline = time.perf_counter() + 60
                while len(done) < len(events) and time.perf_counter() < deadline:
                    done += srv.poll()
                    time.sleep(0.0002)
            finally:
                srv.stop()
        ok = [d for d in done if d["status"] == 0 and d["id"] in measured]
        lat = np.array([d["done_s"] - d["submit_s"] for d in ok]) * 1e3
        span = max(d["done_s"] for d in ok) - min(d["submit_s"] for d in ok) if ok else 1.0
        sweep.append({"load": load, "streams": nstreams, "offered_fps": len(measured) / seconds,
                      "served_fps": len(ok) / span, "completed": len(ok), "submitted": len(measured),
                      "p50_ms": float(np.percentile(lat, 50)) if len(lat) else None,
                      "p99_ms": float(np.percentile(lat, 99)) if len(lat) else None})
        log(f"served load {load:.2f}: {sweep[-1]}")
    rule = f"served >= 0.97 x offered and p99 <= {P99_TARGET_MS:g} ms"
    keeps_up = [x for x in sweep if x["served_fps"] >= 0.97 * x["offered_fps"] and x["p99_ms"] is not None
                and x["p99_ms"] <= P99_TARGET_MS]
    head = max(keeps_up, key=lambda x: x["served_fps"]) if keeps_up else None
    return {"value": head["served_fps"] if head else 0.0, "unit": "frames/s",
            "streams_at_30fps": head["streams"] if head else 0,
            "load": head["load"] if head else None, "p50_ms": head["p50_ms"] if head else None,
            "p99_ms": head["p99_ms"] if head else None, "capacity_fps": capacity_fps, "keeps_up": rule,
            "met": head is not None, "mode": "resident engine" if resident else f"overlapping launches of <= {max_batch} frames",
            "sweep": sweep,
            "latency": "submit to results in the client's pinned buffer, host clock, request loop included"}


def run_served_mix(local: int = 0, nstreams: int = 200, loads=(0.2, 0.5, 0.8, 1.0, 1.2), seconds: float = 3.0,
                   warm_s: float = 1.0, max_batch: int = 64):
    """The serving loop over a mixed population: `nstreams` streams, each of a
    size from {360p, 720p, 1080p, 2160p}, a depth from {8, 10} and a codec
    from {H.264, HEVC} drawn uniformly (seeded), admitted against a 120 GB
    HBM budget; Poisson arrivals over the admitted streams at a total rate of
    a fraction of the mix's batched capacity (a 64-frame launch drawn from
    the same population). One JSON line: admission, capacity, the sweep."""
    import torch
    import rivet_h26x_codecs_b200 as rme
    import rivet_h26x_codecs_b200.capi as capi
    from rivet_h26x_codecs_b200 import synth

    sizes = [(640, 360, 32), (1280, 720, 64), (1920, 1080, 64), (3840, 2160, 128)]
    kinds = [(c, w, h, bd, r) for (w, h, r) in sizes for bd in (8, 10) for c in (capi.RME_CODEC_H264,
                                                                                 capi.RME_CODEC_HEVC)]
    rng = np.random.default_rng(4)
    skind = rng.integers(len(kinds), size=nstreams)
    pools = {}
    for k in sorted(set(skind.tolist())):
        c, w, h, bd, _ = kinds[k]
        pools[k] = synth.stream_sequence(c, w, h, bd, 6, k, config=4).frames

    def params_of(k):
        c, w, h, bd, r = kinds[k]
        q = capi.default_params(c, 28 if c == capi.RME_CODEC_H264 else QP)
        if c == capi.RME_CODEC_H264:
            q.h264_range = min(r, 32)
        else:
            q.hevc_search_range = r
        return q

    # The mix's batched capacity: one launch of 64 frames drawn from the
    # population (device search time).
    with rme.MotionSearch(local) as ms:
        frames, params, pid = [], [], 9000
        for k in rng.choice(skind, size=max_batch):
            c, w, h, bd, _ = kinds[k]
            ids = []
            for f in pools[k][:3]:
                ms.upload(pid, f, c, bd, as_ref=True)
                ids.append(pid)
                pid += 1
            frames.append((ids[2], [ids[1], ids[0]]))
            params.append(params_of(k))
        total = ms.batch_result_count(frames, params)
        dev = torch.empty(total * capi.RESULT_DTYPE.itemsize, dtype=torch.uint8, device=f"cuda:{local}")
        ks = []
        for i in range(8):
            ms.search_batch(frames, params, 0, out=dev)
            if i >= 5:
                ks.append(ms.stats().kernel_ms)
        capacity = max_batch / float(np.median(ks)) * 1e3
    del dev
    torch.cuda.empty_cache()
    per_stream = 4
    sweep, admitted = [], 0
    for load in loads:
        with rme.MotionSearch(local) as ms:
            srv = rme.Server(ms, hbm_budget_bytes=120 << 30, max_frames_per_launch=max_batch, max_streams=1024)
            try:
                live = []
                for sid in range(nstreams):
                    c, w, h, bd, _ = kinds[skind[sid]]
                    if srv.open_stream(sid, c, bd, w, h, params_of(skind[sid]), NREF) == 0:
                        live.append(sid)
                admitted = len(live)
                bufs = {}
                nxt = {}
                for sid in live:
                    pool = pools[skind[sid]]
                    for t in range(NREF + per_stream):
                        srv.submit(sid, pool[t % len(pool)])
                    nxt[sid] = NREF + per_stream
                    n = srv.result_count(sid)
                    bufs[sid] = [np.zeros(n, capi.RESULT_DTYPE) for _ in range(4)]
                pending = len(live) * (NREF + per_stream)
                deadline = time.perf_counter() + 300
                while pending and time.perf_counter() < deadline:
                    pending -= len(srv.poll())
                    time.sleep(0.001)
                rate = load * capacity / len(live)
                events = []
                for sid in live:
                    t = rng.exponential(1 / rate)
                    while t < warm_s + seconds:
                        events.append((t, sid))
                        t += rng.exponential(1 / rate)
                events.sort()
                measured, done = set(), []
                t0 = time.perf_counter()
                for at, sid in events:
                    while time.perf_counter() - t0 < at:
                        done += srv.poll()
                        time.sleep(0.0002)
                    pool = pools[skind[sid]]
                    rid = srv.submit(sid, pool[nxt[sid] % len(pool)], out=bufs[sid][nxt[sid] % 4])
                    nxt[sid] += 1
                    if at >= warm_s:
                        measured.add(rid)
                deadline = time.perf_counter() + 120
                while len(done) < len(events) and time.perf_counter() < deadline:
                    done += srv.poll()
                    time.sleep(0.0005)
            finally:
                srv.stop()
        ok = [d for d in done if d["status"] == 0 and d["id"] in measured]
        lat = np.array([d["done_s"] - d["submit_s"] for d in ok]) * 1e3
        span = max(d["done_s"] for d in ok) - min(d["submit_s"] for d in ok) if ok else 1.0
        sweep.append({"load": load, "offered_fps": len(measured) / seconds, "served_fps": len(ok) / span,
                      "completed": len(ok), "submitted": len(measured),
                      "p50_ms": float(np.percentile(lat, 50)) if len(lat) else None,
                      "p99_ms": float(np.percentile(lat, 99)) if len(lat) else None})
        log(f"served mix load {load:.1f}: {sweep[-1]}")
    print(json.dumps({"workload": "serving mix: sizes 360p..2160p, 8/10-bit, H.264/HEVC, 2 refs",
                      "streams": nstreams, "admitted": admitted, "hbm_budget_gb": 120,
                      "capacity_fps": capacity, "sweep": sweep}), flush=True)


def run_rows(local: int = 0):
    """The rows built beside the headline path, measured on 1080p inputs: per
    row the synchronous C-ABI call timed on the host (its own copies
    included) and the oracle's single-thread time on the same input, one
    JSON line each. The oracle's calls build their reference planes inside;
    that share is timed on its own (an empty call) and taken out."""
    sys.path.insert(0, str(ROOT / "oracle"))
    import oracle
    import rivet_h26x_codecs_b200 as rme
    import rivet_h26x_codecs_b200.capi as capi
    from rivet_h26x_codecs_b200 import synth

    def per_call(fn, reps):
        fn()
        fn()
        a = time.perf_counter()
        for _ in range(reps):
            fn()
        return (time.perf_counter() - a) / reps

    def line(row, unit, n, gpu_s, cpu_s, note):
        print(json.dumps({"row": row, "unit": unit, "value": n / gpu_s, "cpu_value": n / cpu_s, "cpu_threads": 1,
                          "speedup": cpu_s / gpu_s, "gpu_ms_per_call": gpu_s * 1e3, "cpu_ms_per_call": cpu_s * 1e3,
                          "note": note}), flush=True)

    rng = np.random.default_rng(7)
    ms = rme.MotionSearch(local)
    for codec, name in ((capi.RME_CODEC_HEVC, "hevc"), (capi.RME_CODEC_H264, "h264")):
        seq = synth.make_sequence(codec, WIDTH, HEIGHT, 8, 3, synth.seed_for(1), 64, 160, 2.0)
        f0, f1, f2 = seq.frames
        base = 3000 if codec == capi.RME_CODEC_HEVC else 3100
        for i, f in enumerate((f0, f1, f2)):
            ms.upload(base + i, f, codec, 8, as_ref=True)
            ms.lowres_build(base + i)
        # The lookahead's work for one B picture: its plane, both searches,
        # the average of two.
        def gpu_la():
            ms.lowres_build(base + 2)
            _, m0, _ = ms.lowres_search(base + 2, base + 1)
            _, m1, _ = ms.lowres_search(base + 2, base + 0)
            ms.lowres_bi_cost(base + 2, base + 1, m0, base + 0, m1)

        def cpu_la():
            oracle.lowres(f2, 8, codec)
            _, m0, _ = oracle.lowres_search(f2, f1, 8, codec)
            _, m1, _ = oracle.lowres_search(f2, f0, 8, codec)
            oracle.lowres_bi_cost(f2, f1, m0, f0, m1, 8, codec)

        line(f"lookahead_{name}", "frames/s", 1, per_call(gpu_la, 20), per_call(cpu_la, 2),
             "half-resolution plane + intra costs, two block searches, the average-of-two cost "
             "(the oracle's searches rebuild both pictures' planes)")
        # A lookahead's depth at once: every picture against its two
        # predecessors, all pairs in one launch.
        more = synth.make_sequence(codec, WIDTH, HEIGHT, 8, 10, synth.seed_for(2), 64, 160, 2.0).frames
        for i, f in enumerate(more):
            ms.upload(base + 10 + i, f, codec, 8, as_ref=True)
            ms.lowres_build(base + 10 + i)
        pairs = [(base + 10 + t, base + 10 + t - d) for t in range(2, 10) for d in (1, 2)]

        def cpu_pairs():
            for t in range(2, 10):
                for d in (1, 2):
                    oracle.lowres_search(more[t], more[t - d], 8, codec)

        line(f"lookahead_search_batch_{name}", "pairs/s", len(pairs),
             per_call(lambda: ms.lowres_search_batch(pairs), 20), per_call(cpu_pairs, 1),
             "16 (picture, reference) block searches in one launch (the oracle's rebuild both planes)")
        for i in range(10):
            ms.release(base + 10 + i)
        for i in range(3):
            ms.release(base + i)

    # HEVC B: every 16x16 unit of a picture, a pair of vectors each.
    seq = synth.make_sequence(capi.RME_CODEC_HEVC, WIDTH, HEIGHT, 8, 3, synth.seed_for(1), 64, 160, 2.0)
    r0, r1, src = seq.frames
    for i, f in enumerate((src, r0, r1)):
        ms.upload(3200 + i, f, capi.RME_CODEC_HEVC, 8, as_ref=i > 0)
    ph = hevc_params(oracle)
    ph.predictor_mode = capi.RME_PRED_GIVEN
    xs, ys = np.meshgrid(np.arange(0, WIDTH - 15, 16), np.arange(0, HEIGHT - 15, 16))
    nb = xs.size
    bj = np.zeros(nb, capi.BI_JOB_DTYPE)
    bj["x"], bj["y"], bj["w"], bj["h"] = xs.ravel(), ys.ravel(), 16, 16
    bj["ref"] = (0, 1)
    bj["mv"] = rng.integers(-48, 49, size=(nb, 2, 2))
    bj["list"] = rng.integers(2, size=nb)
    bj["mvp"] = bj["mv"]
    empty = bj[:0]
    refs = [r0, r1]
    cpu_base = per_call(lambda: oracle.hevc_bi(8, src, refs, ph, empty, refine=False), 1)
    line("bi_satd_hevc", "units/s", nb, per_call(lambda: ms.bi_satd(3200, [3201, 3202], ph, bj), 20),
         per_call(lambda: oracle.hevc_bi(8, src, refs, ph, bj, refine=False), 1) - cpu_base,
         "satd_bi_at of every 16x16 unit of a 1080p picture")
    line("bi_refine_hevc", "units/s", nb, per_call(lambda: ms.bi_refine(3200, [3201, 3202], ph, bj), 10),
         per_call(lambda: oracle.hevc_bi(8, src, refs, ph, bj, refine=True), 1) - cpu_base,
         "refine_bi of every 16x16 unit (target build, search_full + refine_subpel at 2 lam)")
    for i in range(3):
        ms.release(3200 + i)

    # H.264 B: every macroblock's 16x16 pair, bi_refine's default 2 rounds.
    seq = synth.make_sequence(capi.RME_CODEC_H264, WIDTH, HEIGHT, 8, 3, synth.seed_for(1), 64, 160, 2.0)
    r0, r1, src = seq.frames
    for i, f in enumerate((src, r0, r1)):
        ms.upload(3300 + i, f, capi.RME_CODEC_H264, 8, as_ref=i > 0)
    p4 = oracle.params(capi.RME_CODEC_H264, 28, predictor_mode=capi.RME_PRED_GIVEN)
    xs, ys = np.meshgrid(np.arange(0, WIDTH, 16), np.arange(0, HEIGHT - 15, 16))
    nb = xs.size
    hj = np.zeros(nb, capi.H264_BI_JOB_DTYPE)
    hj["x"], hj["y"], hj["w"], hj["h"] = xs.ravel(), ys.ravel(), 16, 16
    hj["ref"] = (0, 1)
    hj["mv"] = rng.integers(-40, 41, size=(nb, 2, 2))
    hj["mvp"] = hj["mv"]
    hj["limit"] = 0xFFFFFFFF
    refs = [r0, r1]
    cpu_base = per_call(lambda: oracle.h264_bi_refine(8, src, refs, p4, hj[:0], 2), 1)
    line("bi_refine_h264", "macroblocks/s", nb,
         per_call(lambda: ms.h264_bi_refine(3300, [3301, 3302], p4, hj, 2), 20),
         per_call(lambda: oracle.h264_bi_refine(8, src, refs, p4, hj, 2), 1) - cpu_base,
         "b_mb's joint refinement of every macroblock's 16x16 pair, 2 rounds, square ring")

    # Weighted prediction: the weighted search plane (plane 0 and the
    # half-sample planes rebuilt), the fit's two passes.
    def cpu_plane():
        oracle.h264_planes(oracle.weighted_samples(capi.RME_CODEC_H264, 8, r0, 6, 72, -9), 8)

    import torch

    line("weighted_plane_h264", "pictures/s", 1, per_call(lambda: (ms.picture_weighted(3301, 3303, 6, 72, -9),
                                                                   torch.cuda.synchronize()), 50),
         per_call(cpu_plane, 3), "weighted search plane and its b, h, j planes (one 1080p reference)")
    line("wp_moments", "pictures/s", 1, per_call(lambda: ms.wp_moments(3300, 3301), 100),
         per_call(lambda: oracle.wp_moments(capi.RME_CODEC_H264, 8, src, r0), 5), "the fit's sums over a picture pair")
    line("weighted_sad", "pictures/s", 1, per_call(lambda: ms.weighted_sad(3300, 3301, 80, 6, -12), 100),
         per_call(lambda: oracle.weighted_sad(capi.RME_CODEC_H264, 8, src, r0, 80, 6, -12), 5),
         "the fit's weighted SAD over a picture pair")
    for i in range(4):
        ms.release(3300 + i)


def run_configs(local: int = 0):
    """The other workloads of the path, measured as the headline is (one JSON
    line each): the 2160p 10-bit four-reference stream (±128, AMP units) and
    the 64-stream mixed batch (one frame of every stream per launch). Each:
    the batched launch (device-resident, device time of its search) against
    the plain per-frame path (one synchronous call per frame, host clock),
    and whether the two agree bit for bit."""
    import torch
    import rivet_h26x_codecs_b200 as rme
    import rivet_h26x_codecs_b200.capi as capi
    from rivet_h26x_codecs_b200 import synth

    ms = rme.MotionSearch(local)

    def measure(name, frames, params, note):
        total = ms.batch_result_count(frames, params)
        dev = torch.empty(total * capi.RESULT_DTYPE.itemsize, dtype=torch.uint8, device=f"cuda:{local}")
        for _ in range(8):  # the first calls, the graph's capture, a few more
            outs = ms.search_batch(frames, params, 0, out=dev)
        torch.cuda.synchronize()
        ks = []
        for _ in range(5):
            ms.search_batch(frames, params, 0, out=dev)
            ks.append(ms.stats().kernel_ms)
        batched = [v.cpu().numpy().view(capi.RESULT_DTYPE) for v in outs]
        plain, lat = [], []
        for k, (src, refs) in enumerate(frames):
            ms.search(src, refs, params[k])  # warm each shape
        for k, (src, refs) in enumerate(frames):
            a = time.perf_counter()
            plain.append(ms.search(src, refs, params[k]))
            lat.append(time.perf_counter() - a)
        exact = all((b == q).all() for b, q in zip(batched, plain))
        kms = float(np.median(ks))
        print(json.dumps({"config": name, "frames_per_launch": len(frames), "batched_fps": len(frames) / kms * 1e3,
                          "batched_search_ms": kms, "plain_fps": len(frames) / sum(lat),
                          "plain_p50_ms": float(np.median(lat)) * 1e3, "batched_vs_plain": sum(lat) / kms * 1e3,
                          "bit_exact_batched_vs_plain": bool(exact), "note": note}), flush=True)

    # 2160p HEVC 10-bit, 4 references, ±128, AMP 2NxnU / nLx2N.
    seq = synth.config2(nframes=12)
    p2 = capi.default_params(capi.RME_CODEC_HEVC, QP)
    p2.hevc_search_range = 128
    p2.hevc_amp = 0b0101
    for i, f in enumerate(seq.frames):
        ms.upload(4000 + i, f, capi.RME_CODEC_HEVC, 10, as_ref=True)
    frames = [(4000 + t, [4000 + t - 1 - r for r in range(4)]) for t in range(4, 12)]
    measure("2160p HEVC 10-bit, 4 refs, range 128, PUs 8..64 + AMP 2NxnU/nLx2N", frames, [p2] * len(frames),
            "8 frames of the stream per launch (each against its 4 predecessors: source pictures, all known)")
    for i in range(len(seq.frames)):
        ms.release(4000 + i)
    del seq

    # The mixed batch: 64 streams, 2 references each, one frame of each.
    kinds = [(capi.RME_CODEC_H264, 640, 360, 8, 32, 16), (capi.RME_CODEC_HEVC, 1280, 720, 8, 64, 24),
             (capi.RME_CODEC_HEVC, 1920, 1080, 10, 64, 16), (capi.RME_CODEC_HEVC, 3840, 2160, 8, 128, 8)]
    frames, params, pid, stream = [], [], 5000, 0
    for codec, w, h, bd, rng_, count in kinds:
        for _ in range(count):
            seq = synth.stream_sequence(codec, w, h, bd, 3, stream, config=3)
            ids = []
            for f in seq.frames:
                ms.upload(pid, f, codec, bd, as_ref=True)
                ids.append(pid)
                pid += 1
            q = capi.default_params(codec, 28 if codec == capi.RME_CODEC_H264 else QP)
            if codec == capi.RME_CODEC_H264:
                q.h264_range = rng_
            else:
                q.hevc_search_range = rng_
            frames.append((ids[2], [ids[1], ids[0]]))
            params.append(q)
            stream += 1
    measure("64-stream mix: 16x360p H.264 8-bit, 24x720p HEVC 8-bit, 16x1080p HEVC 10-bit, 8x2160p HEVC 8-bit",
            frames, params, "one frame of every stream per launch, 2 references each; four kinds on forked streams")


def other_configs(local: int = 0) -> dict:
    """The path's other workloads, reported inside the headline line (a few
    seconds each): the H.264 CIF frame (frames/s of the plain path and parity
    with the oracle), the 2160p 10-bit four-reference stream (batched against
    plain, bit-exact between them) and the mixed serving population (how many
    30 frames/s streams drawn from it are served at p99 <= 8 ms)."""
    import torch
    import rivet_h26x_codecs_b200 as rme
    import rivet_h26x_codecs_b200.capi as capi
    from rivet_h26x_codecs_b200 import synth
    sys.path.insert(0, str(ROOT / "oracle"))
    import oracle
    out = {}
    with rme.MotionSearch(local) as ms:
        # H.264 CIF, one reference, QP 28, the medium MeCfg.
        seq = synth.config0()
        ms.upload(1, seq.frames[0], capi.RME_CODEC_H264, 8, as_ref=True)
        ms.upload(2, seq.frames[1], capi.RME_CODEC_H264, 8, as_ref=True)
        p4 = capi.default_params(capi.RME_CODEC_H264, 28)
        for _ in range(5):
            got = ms.search(2, [1], p4)
        lat = []
        for _ in range(200):
            a = time.perf_counter()
            ms.search(2, [1], p4)
            lat.append(time.perf_counter() - a)
        want = oracle.frame_search(capi.RME_CODEC_H264, 8, seq.frames[1], [seq.frames[0]], oracle.params(capi.RME_CODEC_H264, 28))
        lat_ms = np.array(lat) * 1e3
        out["h264_cif"] = {"value": len(lat) / float(np.sum(lat)), "unit": "frames/s", "p50_ms": float(np.median(lat_ms)),
                           "p99_ms": float(np.percentile(lat_ms, 99)), "macroblocks": int(len(got)),
                           "bit_exact_vs_oracle": bool((got == want).all()),
                           "call": "plain per-frame search, pictures resident, results to host"}
        # 2160p HEVC 10-bit, 4 references, +-128, PUs 8..64 + AMP 2NxnU / nLx2N.
        seq = synth.config2(nframes=12)
        p2 = capi.default_params(capi.RME_CODEC_HEVC, QP)
        p2.hevc_search_range = 128
        p2.hevc_amp = 0b0101
        for i, f in enumerate(seq.frames):
            ms.upload(100 + i, f, capi.RME_CODEC_HEVC, 10, as_ref=True)
        frames = [(100 + t, [100 + t - 1 - r for r in range(4)]) for t in range(4, 12)]
        total = ms.batch_result_count(frames, p2)
        dev = torch.empty(total * capi.RESULT_DTYPE.itemsize, dtype=torch.uint8, device=f"cuda:{local}")
        for _ in range(8):  # the first calls, the graph's capture, a few more
            outs = ms.search_batch(frames, p2, 0, out=dev)
        ks = []
        for _ in range(3):
            ms.search_batch(frames, p2, 0, out=dev)
            ks.append(ms.stats().kernel_ms)
        batched = [v.cpu().numpy().view(capi.RESULT_DTYPE) for v in outs]
        for _ in range(8):
            ms.search(*frames[0], p2)
        plain, lat = [], []
        for src, refs in frames:
            a = time.perf_counter()
            plain.append(ms.search(src, refs, p2))
            lat.append(time.perf_counter() - a)
        kms = float(np.median(ks))
        out["hevc_2160p10"] = {"batched_fps": len(frames) / kms * 1e3, "plain_fps": len(frames) / float(np.sum(lat)),
                               "plain_p50_ms": float(np.median(lat)) * 1e3, "plain_max_ms": float(np.max(lat)) * 1e3,
                               "bit_exact_batched_vs_plain": bool(all((b == q).all() for b, q in zip(batched, plain))),
                               "note": "8 frames a launch, each against its 4 predecessors; range 128; AMP 2NxnU/nLx2N"}
        del dev, seq
        for i in range(12):
            ms.release(100 + i)
    torch.cuda.empty_cache()
    out["served_mix"] = served_mix_streams(local)
    return out


def served_mix_streams(local: int = 0, counts=(8, 24, 48), seconds: float = 2.0) -> dict:
    """Streams drawn from the mixed population (sizes 360p..2160p, 8/10-bit,
    H.264/HEVC, 2 references each), each at 30 frames/s (Poisson), served by
    the resident engine: per stream count, p50/p99 over all frames and by
    size; the largest count with served >= 0.97 x offered and p99 <= 8 ms."""
    import torch
    import rivet_h26x_codecs_b200 as rme
    import rivet_h26x_codecs_b200.capi as capi
    from rivet_h26x_codecs_b200 import synth
    sizes = [(640, 360, 32), (1280, 720, 64), (1920, 1080, 64), (3840, 2160, 128)]
    kinds = [(c, w, h, bd, r) for (w, h, r) in sizes for bd in (8, 10) for c in (capi.RME_CODEC_H264, capi.RME_CODEC_HEVC)]
    rng = np.random.default_rng(4)
    skind = rng.integers(len(kinds), size=200)
    pools = {}

    def params_of(k):
        c, w, h, bd, r = kinds[k]
        q = capi.default_params(c, 28 if c == capi.RME_CODEC_H264 else QP)
        if c == capi.RME_CODEC_H264:
            q.h264_range = min(r, 32)
        else:
            q.hevc_search_range = r
        return q

    sweep = []
    for n in counts:
        for k in sorted(set(skind[:n].tolist())):
            if k not in pools:
                c, w, h, bd, _ = kinds[k]
                pools[k] = synth.stream_sequence(c, w, h, bd, 6, k, config=4).frames
        with rme.MotionSearch(local) as ms:
            srv = rme.Server(ms, hbm_budget_bytes=120 << 30, max_frames_per_launch=64, max_streams=1024)
            try:
                bufs, nxt = {}, {}
                for sid in range(n):
                    c, w, h, bd, _ = kinds[skind[sid]]
                    assert srv.open_stream(sid, c, bd, w, h, params_of(skind[sid]), NREF) == 0
                for sid in range(n):
                    pool = pools[skind[sid]]
                    codec, nb = srv._streams[sid][0], srv._streams[sid][1]
                    cnt = nb if codec == capi.RME_CODEC_H264 else nb * NREF
                    bufs[sid] = []
                    for _ in range(4):
                        tt = torch.empty(cnt * capi.RESULT_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)
                        bufs[sid].append(tt.numpy().view(capi.RESULT_DTYPE))
                    srv.submit(sid, pool[0])
                    for t in range(1, NREF + 4):
                        srv.submit(sid, pool[t % len(pool)], out=bufs[sid][t % 4])
                    nxt[sid] = NREF + 4
                pending = n * (NREF + 4)
                deadline = time.perf_counter() + 120
                while pending and time.perf_counter() < deadline:
                    pending -= len(srv.poll())
                    time.sleep(0.0005)
                events = []
                for sid in range(n):
                    t = rng.exponential(1 / 30.0)
                    while t < 0.5 + seconds:
                        events.append((t, sid))
                        t += rng.exponential(1 / 30.0)
                events.sort()
                measured, done, size_of = set(), [], {}
                t0 = time.perf_counter()
                for at, sid in events:
                    while time.perf_counter() - t0 < at:
                        done += srv.poll()
                        time.sleep(0.0001)
                    pool = pools[skind[sid]]
                    rid = srv.submit(sid, pool[nxt[sid] % len(pool)], out=bufs[sid][nxt[sid] % 4])
                    nxt[sid] += 1
                    if at >= 0.5:
                        measured.add(rid)
                        size_of[rid] = kinds[skind[sid]][2]
                deadline = time.perf_counter() + 60
                while len(done) < len(events) and time.perf_counter() < deadline:
                    done += srv.poll()
                    time.sleep(0.0002)
            finally:
                srv.stop()
        ok = [d for d in done if d["status"] == 0 and d["id"] in measured]
        lat = np.array([d["done_s"] - d["submit_s"] for d in ok]) * 1e3
        span = max(d["done_s"] for d in ok) - min(d["submit_s"] for d in ok) if ok else 1.0
        by_size = {}
        for hgt in sorted(set(size_of.values())):
            ls = np.array([d["done_s"] - d["submit_s"] for d in ok if size_of[d["id"]] == hgt]) * 1e3
            if len(ls):
                by_size[f"{hgt}p"] = {"frames": int(len(ls)), "p50_ms": float(np.median(ls)),
                                      "p99_ms": float(np.percentile(ls, 99))}
        sweep.append({"streams": n, "offered_fps": len(measured) / seconds, "served_fps": len(ok) / span,
                      "p50_ms": float(np.median(lat)) if len(lat) else None,
                      "p99_ms": float(np.percentile(lat, 99)) if len(lat) else None, "by_size": by_size})
        log(f"served mix {n} streams: {sweep[-1]}")
    good = [x for x in sweep if x["p99_ms"] is not None and x["p99_ms"] <= P99_TARGET_MS
            and x["served_fps"] >= 0.97 * x["offered_fps"]]
    return {"streams_at_30fps_p99_8ms": max((x["streams"] for x in good), default=0), "sweep": sweep,
            "population": "200 streams drawn uniformly over {360p, 720p, 1080p, 2160p} x {8, 10 bit} x {H.264, HEVC}; "
                          "the first n of them, 30 frames/s each"}


def profile_case(kind: str):
    """The cases the ncu captures of the search kernel run on: one 1080p
    frame (2 references, about 130 MB on the device) through the per-frame
    path, or 8 frames (10 pictures, about 420 MB) in one batched launch;
    each searched twice. Inputs are larger than L2 in both."""
    import rivet_h26x_codecs_b200 as rme
    import rivet_h26x_codecs_b200.capi as capi
    from rivet_h26x_codecs_b200 import synth
    n = 3 if kind == "frame" else 10
    seq = synth.make_sequence(synth.HEVC, WIDTH, HEIGHT, 8, n, synth.seed_for(1), 64, 160, 2.0)
    with rme.MotionSearch(0) as ms:
        for i, f in enumerate(seq.frames):
            ms.upload(i, f, capi.RME_CODEC_HEVC, 8, as_ref=True)
        p = hevc_params()
        for _ in range(2):
            if kind == "frame":
                ms.search(2, [1, 0], p)
            else:
                ms.search_batch([(t, [t - 1, t - 2]) for t in range(2, n)], p)
        st = ms.stats()
        print(f"profile case {kind}: kernel {st.kernel_ms:.3f} ms, tasks {st.tasks}")


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--ref-frames", type=int, default=None,
                    help="reference arm: frames per step (default: the whole 60-frame step of our arm)")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-serve", action="store_true", help="skip the serving-loop sweep")
    ap.add_argument("--served-mix", action="store_true",
                    help="the serving loop over the mixed 200-stream population instead")
    ap.add_argument("--configs", action="store_true",
                    help="measure the 2160p 10-bit stream and the 64-stream mixed batch instead")
    ap.add_argument("--rows", action="store_true",
                    help="measure the rows beside the headline path (lookahead, B, weighted) instead")
    ap.add_argument("--profile-case", choices=["frame", "batch"], default=None,
                    help="small case for ncu: one frame (3 pictures) or a batch of 8 frames, searched twice")
    args = ap.parse_args()
    world, rank, local = dist_setup(args)
    if args.profile_case:
        profile_case(args.profile_case)
        return
    if args.rows:
        run_rows(local)
        return
    if args.configs:
        run_configs(local)
        return
    if args.served_mix:
        run_served_mix(local)
        return
    try:
        if args.impl == "reference":
            run_reference(args, world, rank)
        else:
            run_ours(args, world, rank, local)
    finally:
        if world > 1:
            import torch.distributed as dist
            dist.destroy_process_group()


if __name__ == "__main__":
    main()
