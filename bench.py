#!/usr/bin/env python3
"""Benchmark of the per-frame hyperspectral detection hot path on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--workload sam|sam_cem]

One step = one pass of the hot path over one batch of synthetic frames:
64 frames of 1024x1024x113 float32 (the SAM+CEM video configuration), each
scored against an 8-target library (8 per-target SAM maps, best angle + id)
and thresholded into a raster-ordered detection list.  With
--workload sam_cem each frame also gets its scene correlation (tensor-core
stats pass), FP64 factorisation and 8 CEM maps from the same fused pass.

The JSON line reports whole-job Mpix/s with inputs resident in HBM (`value`),
the same metric end to end through the C ABI with host buffers and the
host<->device copies inside the timed region (`e2e`), the dominant kernel's
roofline fraction, and the reference's own CPU scorer timed on this host's
cores (`cpu_baseline`).  `--impl reference` times only that CPU scorer.

Multi-GPU (torchrun): frames are independent, so each rank scores its own 64
frames with no collective on the data path (weak scaling); the step time is
the max over ranks.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

REPO = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, REPO)
sys.path.insert(0, os.path.join(REPO, "hsi-detectors-cuda_b200"))

H, W, B = 1024, 1024, 113
FRAMES = 64
TARGETS = 8
THRESHOLD = 0.10
NMS_RADIUS = 2
CAPACITY = 4096
LOADING = 1e-6
CEM_THRESHOLD = 0.5


def max_over_ranks(dist, values, device):
    """Element-wise max of per-rank timings over all ranks (every rank gets it):
    the multi-GPU step time is the slowest rank's."""
    import torch
    if dist is None:
        return [float(v) for v in values]
    t = torch.tensor([float(v) for v in values], device=device, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return [float(v) for v in t]


def whole_job_mpix(world, pixels_per_rank, ms):
    """Whole-job throughput: every rank processes its own frames (weak scaling)."""
    return world * pixels_per_rank / (ms / 1e3) / 1e6


def rank_seed(base, rank, stride=1000):
    """Frame seeds per rank: ranks score different frames of the same scene model."""
    return base + stride * rank


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default=None, choices=["sam", "sam_cem", "rx_ace", "screen", "batch", "bip"])
    ap.add_argument("--train-frames", type=int, default=200)
    ap.add_argument("--frames", type=int, default=FRAMES)
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--profile-range", action="store_true",
                    help="bracket one untimed run (a batch graph replay; the first screen training frame and one screen step) with "
                         "cudaProfilerStart/Stop, for `ncu --profile-from-start off` launch lists")
    ap.add_argument("--no-extras", action="store_true",
                    help="skip the extra records of the default run (RX/ACE, screen, same-shape SAM scorer, "
                         "the reference's GPU SAM comparator)")
    return ap.parse_args()


# Both arms (ours and --impl reference) run this workload unless told otherwise.
DEFAULT_WORKLOAD = "sam_cem"


# ---------------------------------------------------------------------------
# CPU reference (the reference's own scorer, compiled from its sources)
# ---------------------------------------------------------------------------

def cpu_reference(workload, sample_rows, repeats, threads=None):
    """Run the reference CPU path on `threads` sample frames of 1024 x sample_rows
    at once, one frame per thread, `repeats` times.  Returns (Mpix/s, threads, seconds)."""
    import ctypes as C
    import oracle
    lib = oracle.ref_lib()
    threads = threads or len(os.sched_getaffinity(0))
    seed = 0x5EED2000 if workload == "rx_ace" else 0x5EED1000
    anomaly = 0.001 if workload == "rx_ace" else 0.0
    spec = oracle.scene(B, n_targets=TARGETS, target_frac=0.002, library_seed=seed)
    _, targets, _ = oracle.scene_spectra(spec.library_seed, B, 6, TARGETS)
    targets = np.ascontiguousarray(targets)
    norms = oracle.ref_norms(targets)
    P = W * sample_rows
    cubes = []
    for t in range(threads):
        s = oracle.scene(B, n_targets=TARGETS, target_frac=0.002, anomaly_frac=anomaly, library_seed=seed,
                         frame_seed=seed + 1 + t)
        cubes.append(oracle.generate(s, sample_rows, W)[0])
    f32, i32 = C.POINTER(C.c_float), C.POINTER(C.c_int32)

    def work(cube):
        maps = np.empty((TARGETS, P), np.float32)
        best = np.empty(P, np.float32)
        bt = np.empty(P, np.int32)
        cem = np.empty(P, np.float32)
        ct = np.empty(P, np.int32)
        dets = np.zeros(CAPACITY, oracle.DETECTION_DTYPE)
        cp = cube.ctypes.data_as(f32)
        if workload == "rx_ace":
            lib.ref_frame_rx_ace(cp, sample_rows, W, B, targets.ctypes.data_as(f32), TARGETS, LOADING,
                                 cem.ctypes.data_as(f32), ct.ctypes.data_as(i32), best.ctypes.data_as(f32))
        elif workload == "sam_cem":
            lib.ref_frame_sam_cem(cp, sample_rows, W, B, targets.ctypes.data_as(f32), TARGETS, LOADING,
                                  THRESHOLD, NMS_RADIUS, maps.ctypes.data_as(f32), best.ctypes.data_as(f32),
                                  bt.ctypes.data_as(i32), cem.ctypes.data_as(f32), ct.ctypes.data_as(i32),
                                  dets.ctypes.data, CAPACITY)
        else:
            lib.ref_sam_all(cp, sample_rows, W, B, targets.ctypes.data_as(f32), norms.ctypes.data_as(f32),
                            TARGETS, maps.ctypes.data_as(f32))
            lib.ref_sam_best(cp, sample_rows, W, B, targets.ctypes.data_as(f32), norms.ctypes.data_as(f32),
                             TARGETS, best.ctypes.data_as(f32), bt.ctypes.data_as(i32))
            lib.ref_detect(best.ctypes.data_as(f32), bt.ctypes.data_as(i32), sample_rows, W, THRESHOLD,
                           NMS_RADIUS, 0, dets.ctypes.data, CAPACITY)

    times = []
    for _ in range(repeats):
        ths = [threading.Thread(target=work, args=(c,)) for c in cubes]
        t0 = time.perf_counter()
        for t in ths:
            t.start()
        for t in ths:
            t.join()
        times.append(time.perf_counter() - t0)
    return times, threads, P


def cpu_baseline(workload, note=""):
    """The line's "cpu_baseline": the reference's CPU path on sample frames, or why its
    library (compiled from its sources by oracle/Makefile) is not there."""
    try:
        times, threads, P = cpu_reference(workload, 128, 2)
    except OSError as e:
        return {"unavailable": f"{type(e).__name__}: {e}"}
    t = float(np.mean(times))
    return {"value": round(threads * P / t / 1e6, 3), "unit": "Mpix/s", "cores": threads, "kind": "reference",
            "sample": f"{threads} frames of {W}x128x{B}, one per thread{note}, mean of 2 runs"}


# Shapes of the same-box GPU comparison of SAM scorers: the plain-SAM
# configuration (one target) and the SAM+CEM video frame (eight targets).
SAM_SHAPES = [(520, 696, 113, 1), (1024, 1024, 113, 8)]
BENCH_SAM = os.path.join(REPO, "oracle", "_ref", "bench_sam")


def reference_gpu_sam(timeout=300):
    """The reference's own GPU SAM kernels on this GPU: its unmodified
    bench/bench_sam.cu, built for sm_100a by oracle/Makefile, run at each of
    SAM_SHAPES.  Returns {shape: {variant: {"ms", "mpix_s"}}} from its
    throughput table (median of its timed passes, one resident cube), or a
    reason string."""
    if not os.path.exists(BENCH_SAM):
        return "oracle/_ref/bench_sam is not built"
    out = {}
    for h, w, b, t in SAM_SHAPES:
        cmd = [BENCH_SAM, f"--height={h}", f"--width={w}", f"--bands={b}", f"--targets={t}",
               "--iterations=50", "--warmup-ms=500", "--repeats=5"]
        r = subprocess.run(cmd, capture_output=True, text=True, timeout=timeout)
        rows, table, verdicts = {}, False, {}
        for line in r.stdout.splitlines():
            parts = line.split()
            if "Gpix/s" in line and parts and parts[0] == "variant":
                table = True
                continue
            if parts and parts[0] in ("baseline", "optimized", "half", "bip"):
                if table and len(parts) >= 8:
                    ms = float(parts[1])
                    rows[parts[0]] = {"ms": ms, "mpix_s": round(h * w / (ms / 1e3) / 1e6, 1)}
                elif not table and ("PASS" in parts or "FAIL" in parts):
                    verdicts[parts[0]] = "PASS" if "PASS" in parts else "FAIL"
            if line.startswith("optimized, pixels per thread"):
                table = False
        if r.returncode != 0 and not rows:
            return f"bench_sam exited {r.returncode}: {r.stderr.strip()[-200:]}"
        for k, v in verdicts.items():
            if k in rows:
                rows[k]["check_vs_cpu"] = v
        out[f"{h}x{w}x{b}, {t} target(s)"] = rows
    return out


def run_reference(args, workload):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    rows = 128
    times, threads, P = cpu_reference(workload, rows, args.warmup + args.steps)
    timed = times[args.warmup:]
    t = float(np.mean(timed))
    value = threads * P / t / 1e6
    gpu_cmp = None
    if not args.no_extras:
        try:
            gpu_cmp = reference_gpu_sam()
        except Exception as e:  # the comparator is extra information; the CPU arm stands without it
            gpu_cmp = f"{type(e).__name__}: {e}"
    config = workload_config(workload, args.frames, reference=True)
    config["deviation"] = (f"the CPU arm times {threads} sample frames of {W}x{rows}x{B} per step (one per host "
                           f"thread) and reports Mpix/s; the GPU arm's frames are {H}x{W}x{B}")
    line = {
        "impl": "reference", "metric": metric_name(workload), "value": round(value, 3), "unit": "Mpix/s",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(t * 1e3, 3),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic (seeded scene model, host-generated)",
        "config": config,
        "cpu_baseline": {"value": round(value, 3), "unit": "Mpix/s", "cores": threads, "kind": "reference",
                         "sample": f"{threads} frames of {W}x{rows}x{B} per step, one per thread"},
        "e2e": {"value": round(value, 3), "unit": "Mpix/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    if gpu_cmp is not None:
        line["gpu_comparator"] = {
            "what": "the reference's own GPU SAM kernels (src/sam.cu via its bench/bench_sam.cu, unmodified, "
                    "built for sm_100a) on this GPU: best angle + id, one resident cube, median of 5 passes of "
                    "50 launches; its own synthetic source",
            "results": gpu_cmp}
    print(json.dumps(line), flush=True)


def metric_name(workload):
    if workload == "batch":
        return "Mpix/s SAM+RX+ACE, 32 uneven frames (16/113/224 bands) in one CUDA graph"
    if workload == "screen":
        return "Mpix/s ACE with learned screen @224 bands"
    if workload == "rx_ace":
        return "Mpix/s RX+ACE @113 bands"
    return "Mpix/s SAM+CEM @113 bands" if workload == "sam_cem" else "Mpix/s SAM @113 bands"


def workload_config(workload, frames, reference=False):
    if workload == "rx_ace":
        return {"workload": f"one {RX_H}x{RX_W}x{B} f32 frame per GPU, {TARGETS} ACE targets: scene moments + "
                            "FP64 factor + whitening (RX + ACE maps + best)",
                "height": RX_H, "width": RX_W, "bands": B, "targets": TARGETS, "diagonal_loading": LOADING,
                "l2": "host CPU" if reference else "inputs larger than L2 (947.9 MB cube)"}
    cfg = {
        "workload": (f"{frames} frames {H}x{W}x{B} f32, {TARGETS} targets: "
                     + ("scene correlation + FP64 factor + fused SAM/CEM maps" if workload == "sam_cem"
                        else "SAM per-target maps + best")
                     + " + raster-ordered detection list"),
        "frames_per_step": frames, "height": H, "width": W, "bands": B, "targets": TARGETS,
        "threshold_rad": THRESHOLD, "nms_radius": NMS_RADIUS, "capacity": CAPACITY,
        "l2": "inputs larger than L2 (30.3 GB of cubes per GPU)",
    }
    if workload == "sam_cem":
        cfg["diagonal_loading"] = LOADING
    if reference:
        cfg["l2"] = "host CPU"
    return cfg


# ---------------------------------------------------------------------------
# GPU side
# ---------------------------------------------------------------------------

class ClockSampler:
    """SM clocks and throttle reasons sampled while the timed region runs: NVML
    read-only queries from a thread every 5 ms (a region of tens of ms still gets
    a dozen samples), else nvidia-smi every 200 ms.  Nothing is set."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
    REASONS = {"hw_slowdown": 0x8, "hw_thermal_slowdown": 0x40, "sw_thermal_slowdown": 0x20, "sw_power_cap": 0x4}

    def __init__(self, uuid):
        self.uuid = uuid
        self.proc = None
        self.file = None
        self.thread = None
        self.samples = []  # (sm MHz, reason bits)
        self.max_mhz = None

    def _nvml_start(self):
        import threading
        import pynvml
        pynvml.nvmlInit()
        h = (pynvml.nvmlDeviceGetHandleByUUID(self.uuid.encode()) if self.uuid
             else pynvml.nvmlDeviceGetHandleByIndex(0))
        self.max_mhz = float(pynvml.nvmlDeviceGetMaxClockInfo(h, pynvml.NVML_CLOCK_SM))
        self.stop = threading.Event()

        def run():
            while not self.stop.is_set():
                try:
                    self.samples.append((float(pynvml.nvmlDeviceGetClockInfo(h, pynvml.NVML_CLOCK_SM)),
                                         int(pynvml.nvmlDeviceGetCurrentClocksEventReasons(h))))
                except Exception:
                    pass
                self.stop.wait(0.005)

        self.thread = threading.Thread(target=run, daemon=True)
        self.thread.start()

    def __enter__(self):
        try:
            self._nvml_start()
            return self
        except Exception:
            self.thread = None
        try:
            self.file = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
            cmd = ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits", "-lms", "200"]
            if self.uuid:
                cmd += ["-i", self.uuid]
            self.proc = subprocess.Popen(cmd, stdout=self.file, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *exc):
        if self.thread is not None:
            self.stop.set()
            self.thread.join(timeout=5)
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        if self.thread is not None:
            if not self.samples:
                return None
            reasons = {n for n, bit in self.REASONS.items() if any(r & bit for _, r in self.samples)}
            return {"sm_mhz": float(np.median([m for m, _ in self.samples])), "sm_max_mhz": self.max_mhz,
                    "reasons": sorted(reasons), "samples": len(self.samples), "source": "nvml, 5 ms"}
        if self.file is None:
            return None
        try:
            rows = [l.split(",") for l in open(self.file.name).read().strip().splitlines() if l.strip()]
            os.unlink(self.file.name)
        except Exception:
            return None
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            try:
                sm.append(float(r[1]))
                mx = float(r[2])
                for i, n in enumerate(names):
                    if r[5 + i].strip() == "Active":
                        reasons.add(n)
            except (ValueError, IndexError):
                continue
        if not sm:
            return None
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm), "source": "nvidia-smi, 200 ms"}


class Workload:
    """Device-resident frames, libraries, outputs and the batched launch table."""

    def __init__(self, hsi, torch, frames, workload, device, seed_base, dtype=0):
        self.hsi, self.torch, self.n, self.kind = hsi, torch, frames, workload
        self.dtype = dtype  # 0: fp32 cubes, 1: fp16 cubes (accumulated in FP32)
        self.P = H * W
        self.stride = hsi.plane_stride(H, W)
        sc = hsi.scene(B, n_targets=TARGETS, target_frac=0.002, library_seed=0x5EED1000)
        self.targets_np = hsi.scene_targets(sc)
        self.targets = torch.from_numpy(self.targets_np).to(device)
        self.norms = torch.from_numpy(hsi.target_norms(self.targets_np)).to(device)
        self.cubes = []
        for f in range(frames):
            s = hsi.scene(B, n_targets=TARGETS, target_frac=0.002, library_seed=0x5EED1000,
                          frame_seed=seed_base + f)
            cube, _ = hsi.generate(s, H, W, dtype=dtype, truth=False, device=device)
            self.cubes.append(cube)
        P = self.P
        self.sam_maps = torch.empty((frames, TARGETS, P), device=device)
        self.sam_best = torch.empty((frames, P), device=device)
        self.sam_bt = torch.empty((frames, P), dtype=torch.int32, device=device)
        self.dets = torch.empty((frames, CAPACITY, 4), dtype=torch.int32, device=device)
        self.counts = torch.zeros((frames,), dtype=torch.int32, device=device)
        self.ws_bytes = hsi.detect_workspace_bytes(H, W)
        self.ws = torch.empty((frames, self.ws_bytes), dtype=torch.uint8, device=device)
        # one batched detection call for every frame's best-angle map
        self.jobs = [hsi.detect_job(self.sam_best[f], self.sam_bt[f], H, W, THRESHOLD, NMS_RADIUS,
                                    hsi.LOWER_IS_BETTER, CAPACITY, self.dets[f], self.counts[f:f + 1])
                     for f in range(frames)]
        self.det_ws = torch.empty(hsi.detect_batch_workspace_bytes(self.jobs), dtype=torch.uint8, device=device)
        self.cem = self.kind == "sam_cem"
        if self.cem:
            self.cem_w = torch.zeros((frames, TARGETS, B), device=device)
            self.cem_maps = torch.empty((frames, TARGETS, P), device=device)
            self.cem_best = torch.empty((frames, P), device=device)
            self.cem_bt = torch.empty((frames, P), dtype=torch.int32, device=device)
            self.moments = torch.zeros((frames, B + B * B + 1), dtype=torch.float64, device=device)
            self.status = torch.zeros(frames, dtype=torch.int32, device=device)
            # every frame's moments in one batched launch sequence
            jobs = [hsi.moments_job(self.cubes[f], H, W, B, self.moments[f], dtype=dtype, stride=self.stride)
                    for f in range(frames)]
            self.moment_jobs = (hsi.MomentsJob * frames)(*jobs)
            self.stats_bytes = hsi.lib().hsi_scene_moments_batch_workspace_bytes(self.moment_jobs, frames)
            self.stats_ws = torch.empty(self.stats_bytes, dtype=torch.uint8, device=device)
        self.table = self._table(self.cubes)
        self.launches_per_step = 0

    def _table(self, cubes):
        hsi = self.hsi
        frames = []
        for f, cube in enumerate(cubes):
            kw = dict(sam_targets=self.targets, sam_norms=self.norms, sam_maps=self.sam_maps[f],
                      sam_best=self.sam_best[f], sam_best_target=self.sam_bt[f], map_stride=self.P)
            if self.cem:
                kw.update(cem_weights=self.cem_w[f], cem_maps=self.cem_maps[f], cem_best=self.cem_best[f],
                          cem_best_target=self.cem_bt[f])
            frames.append(hsi.make_frame(cube, H, W, B, self.dtype, **kw))
        self.frames = frames  # host descriptors for hsi_score_frames_batch
        return hsi.frame_table(frames)

    def step(self, stream, events=None):
        """One pass of the hot path over all frames.  Returns kernel launches issued."""
        import ctypes as C
        hsi, torch = self.hsi, self.torch
        launches = 0
        L = hsi.lib()
        s = C.c_void_p(stream.cuda_stream)
        if events is not None:
            events[2].record(stream)
        if self.cem:
            hsi.check(L.hsi_scene_moments_batch(self.moment_jobs, self.n, C.c_void_p(self.stats_ws.data_ptr()),
                                                self.stats_bytes, s), "hsi_scene_moments_batch")
            launches += moments_launches([(H * W, B)] * self.n)
            # one launch factors every frame (one CTA per frame, FP64)
            hsi.check(L.hsi_build_statistics(self.n, B, TARGETS, LOADING, C.c_void_p(self.moments.data_ptr()),
                                             C.c_void_p(self.targets.data_ptr()), 0, None, None,
                                             C.c_void_p(self.cem_w.data_ptr()), C.c_void_p(self.status.data_ptr()),
                                             None, 0, s), "hsi_build_statistics")
            launches += 1
        if events is not None:
            events[0].record(stream)
        hsi.score_frames_batch(self.frames, stream=stream)
        launches += 1
        if events is not None:
            events[1].record(stream)
        self.counts.zero_()
        hsi.detect_batch(self.jobs, self.det_ws, stream=stream)
        launches += detect_launches(len(self.jobs))
        if events is not None and len(events) > 3:
            events[3].record(stream)
        return launches


# ---------------------------------------------------------------------------
# Kernel launches of the library's calls (the lines' "gpu_launches"; copies and
# fills are not counted)
# ---------------------------------------------------------------------------

def moments_launches(frames):
    """hsi_scene_moments(_batch) over FP32 or FP16 frames of one element type, (pixels, bands) each."""
    tensor = sum(1 for p, b in frames if p >= 32768 and b <= 127)
    # groups of up to 64 tensor-path frames: subsample, its reduction, GEMM, range
    # check, rescale, conditional GEMM re-run, reduce, finalize
    n = 8 * ((tensor + 63) // 64)
    for p, b in frames:
        if p >= 32768 and 127 < b <= 252:
            n += 9  # the same over six views, and their assembly
        elif p >= 32768 and 252 < b <= 254:
            n += 10  # the same over two views, the cross product and the assembly
        elif p < 32768 or b > 254:
            n += 6  # plain: three for the reference point, product, reduce, finalize
    return n


def rx_ace_launches(bands, targets, tensor_cores):
    """Preparation and scorer per pass over the targets."""
    return 2 * (max(1, -(-targets // min(16, 128 - bands))) if tensor_cores else 1)


def detect_launches(maps=1):
    """Two per 64 maps (of up to 16384 row segments each)."""
    return 2 * ((maps + 63) // 64)


def batch_launches(specs):
    """One run of the batch runner over (height, width, bands, targets, mosaic) FP32 frames,
    RX/ACE on the tensor cores up to 127 bands: one scorer launch, the moments, a
    factorisation and RX/ACE per frame, demosaics, three lists per frame."""
    n = 1 + moments_launches([(h * w, b) for h, w, b, _, _ in specs]) + detect_launches(3 * len(specs))
    for _, _, b, t, mosaic in specs:
        n += (1 if mosaic else 0) + 1 + rx_ace_launches(b, t, b <= 127)
    return n


def algorithmic_bytes_score(frames, cem, esize=4):
    """Bytes the fused scoring pass must move: the cube once (esize bytes per
    element), every map and the best/id outputs written once."""
    per_px = esize * B + 4 * TARGETS + 8
    if cem:
        per_px += 4 * TARGETS + 8
    return frames * H * W * per_px


def algorithmic_bytes_step(frames, cem):
    """Whole step: + the stats pass (cube read again) and the detection pass
    (best score + id read, 8 B/px)."""
    b = algorithmic_bytes_score(frames, cem) + frames * H * W * 8
    if cem:
        b += frames * H * W * 4 * B
    return b


def run_ours(args, workload):
    import torch
    import torch.distributed as dist
    import hsi_b200 as hsi

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", init_method="env://",
                                timeout=__import__("datetime").timedelta(seconds=300))
    device = torch.device("cuda", local if world > 1 else 0)
    torch.cuda.set_device(device)
    hsi.lib()

    wl = Workload(hsi, torch, args.frames, workload, device, seed_base=rank_seed(0x5EED1000, rank))
    stream = torch.cuda.current_stream(device)

    def barrier():
        if world > 1:
            dist.barrier()

    for _ in range(args.warmup):
        wl.step(stream)
    torch.cuda.synchronize()

    props = torch.cuda.get_device_properties(device)
    uuid = getattr(props, "uuid", None)
    uuid = f"GPU-{uuid}" if uuid is not None and not str(uuid).startswith("GPU-") else (str(uuid) if uuid else None)

    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    kev = [tuple(torch.cuda.Event(enable_timing=True) for _ in range(4)) for _ in range(args.steps)]
    barrier()
    torch.cuda.synchronize()
    launches = 0
    with ClockSampler(uuid) as clocks:
        start.record(stream)
        for k in range(args.steps):
            launches += wl.step(stream, kev[k])
        end.record(stream)
        torch.cuda.synchronize()
    barrier()
    ms = start.elapsed_time(end) / args.steps
    kernel_ms = float(np.mean([e[0].elapsed_time(e[1]) for e in kev]))
    stats_ms = float(np.mean([e[2].elapsed_time(e[0]) for e in kev]))
    detect_ms = float(np.mean([e[1].elapsed_time(e[3]) for e in kev]))
    ms, kernel_ms, stats_ms, detect_ms = max_over_ranks(dist if world > 1 else None,
                                                        [ms, kernel_ms, stats_ms, detect_ms], device)
    pixels_step = args.frames * H * W
    value = whole_job_mpix(world, pixels_step, ms)
    # detections found per frame in the last step (the detection workload's density)
    found = wl.counts.double().mean().item()

    # dominant kernel: the fused scoring pass
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(REPO, "MEASURED_PEAKS.json")))
    except Exception:
        pass
    hbm = float(peaks.get("hbm_gbs", 6650.0))
    achieved = algorithmic_bytes_score(args.frames, wl.cem) / (kernel_ms / 1e3) / 1e9
    traffic = load_traffic(workload, args.frames)
    roofline = {"kernel": "score_kernel (fused SAM/CEM filter bank)", "bound": "hbm",
                "achieved": round(achieved, 1), "peak": hbm, "unit": "GB/s", "frac": round(achieved / hbm, 4),
                "peak_source": "measured (MEASURED_PEAKS.json hbm_gbs)" if "hbm_gbs" in peaks else "fallback",
                "traffic": traffic, "kernel_ms": round(kernel_ms, 3),
                "algorithmic_bytes_per_launch": algorithmic_bytes_score(args.frames, wl.cem)}
    step_bytes = algorithmic_bytes_step(args.frames, wl.cem)
    roofline_stats = None
    if wl.cem:
        sb = args.frames * H * W * 4 * B
        ach = sb / (stats_ms / 1e3) / 1e9
        roofline_stats = {"kernel": "scene moments (INT8-limb tcgen05 GEMM) + FP64 factor, all frames",
                          "bound": "hbm", "achieved": round(ach, 1), "peak": hbm, "unit": "GB/s",
                          "frac": round(ach / hbm, 4), "ms": round(stats_ms, 3), "algorithmic_bytes": sb}

    e2e = None
    if not args.no_e2e:
        e2e = run_e2e(hsi, torch, wl, stream, args, world)

    del wl
    torch.cuda.empty_cache()

    # the configuration's fp16 variant of the same frames (FP32 accumulation)
    f16 = None
    if workload in ("sam", "sam_cem"):
        wl16 = Workload(hsi, torch, args.frames, workload, device, seed_base=rank_seed(0x5EED1000, rank), dtype=1)
        for _ in range(args.warmup):
            wl16.step(stream)
        ev = [tuple(torch.cuda.Event(enable_timing=True) for _ in range(4)) for _ in range(args.steps)]
        a16, b16 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        barrier()
        torch.cuda.synchronize()
        a16.record(stream)
        for k in range(args.steps):
            wl16.step(stream, ev[k])
        b16.record(stream)
        torch.cuda.synchronize()
        barrier()
        ms16 = a16.elapsed_time(b16) / args.steps
        k16 = float(np.mean([e[0].elapsed_time(e[1]) for e in ev]))
        s16 = float(np.mean([e[2].elapsed_time(e[0]) for e in ev]))
        d16 = float(np.mean([e[1].elapsed_time(e[3]) for e in ev]))
        ms16, k16, s16, d16 = max_over_ranks(dist if world > 1 else None, [ms16, k16, s16, d16], device)
        ach16 = algorithmic_bytes_score(args.frames, wl16.cem, esize=2) / (k16 / 1e3) / 1e9
        f16 = {"value": round(whole_job_mpix(world, pixels_step, ms16), 2), "unit": "Mpix/s",
               "ms_per_step": round(ms16, 3), "dtype": "f16 storage, f32 accumulation",
               "step_split_ms": {"statistics": round(s16, 3), "scoring": round(k16, 3), "detection": round(d16, 3)},
               "scoring_roofline_frac": round(ach16 / hbm, 4)}
        if not args.no_e2e:
            # the same end-to-end path with FP16 host cubes: half the bytes over PCIe
            f16["e2e"] = run_e2e(hsi, torch, wl16, stream, args, world)
        del wl16
        torch.cuda.empty_cache()

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        cpu = cpu_baseline(workload)

    if rank == 0:
        line = {
            "metric": metric_name(workload), "value": round(value, 2), "unit": "Mpix/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms, 3), "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic (seeded scene model generated on the device)",
            "config": dict(workload_config(workload, args.frames), parallelism=f"frames sharded over {world} GPU(s)"),
            "roofline": roofline,
            "roofline_stats": roofline_stats,
            "step_hbm_fraction": round(step_bytes / (ms / 1e3) / 1e9 / hbm, 4),
            "detections_per_frame": round(found, 1),
            "step_split_ms": {"statistics": round(stats_ms, 3), "scoring": round(kernel_ms, 3),
                              "detection": round(detect_ms, 3)},
            "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": launches, "clocks": clocks.summary(),
        }
        if f16 is not None:
            line["f16_variant"] = f16
        if world == 1 and not args.no_extras:
            extra_records(args, device, line)
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


def same_shape_scorer(hsi, torch, device, passes=5, iterations=50, warm_s=0.5):
    """This library's SAM scorer (best angle + id, no per-target maps) at the
    shapes the reference's bench_sam is run at (SAM_SHAPES), timed the way
    bench_sam times its kernels: one resident cube, CUDA events around
    `iterations` launches, the median of `passes` passes, after a warm-up in
    wall time.  FP32 and FP16 cubes."""
    out = {}
    stream = torch.cuda.current_stream(device)
    for h, w, b, t in SAM_SHAPES:
        P = h * w
        rec = {}
        sc = hsi.scene(b, n_targets=t, target_frac=0.005 if t == 1 else 0.002, library_seed=0x5EED0000)
        targets = hsi.scene_targets(sc)
        tg = torch.from_numpy(targets).to(device)
        nr = torch.from_numpy(hsi.target_norms(targets)).to(device)
        best = torch.empty(P, device=device)
        bt = torch.empty(P, dtype=torch.int32, device=device)
        for dt, name, esize in ((hsi.F32, "f32", 4), (hsi.F16, "f16", 2)):
            cube, _ = hsi.generate(sc, h, w, dtype=dt, truth=False, device=device)
            frames = [hsi.make_frame(cube, h, w, b, dt, sam_targets=tg, sam_norms=nr, sam_best=best,
                                     sam_best_target=bt, map_stride=P)]
            t0 = time.perf_counter()
            while time.perf_counter() - t0 < warm_s:
                for _ in range(16):
                    hsi.score_frames_batch(frames, stream=stream)
                torch.cuda.synchronize()
            samples = []
            for _ in range(passes):
                a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(stream)
                for _ in range(iterations):
                    hsi.score_frames_batch(frames, stream=stream)
                e.record(stream)
                torch.cuda.synchronize()
                samples.append(a.elapsed_time(e) / iterations)
            ms = float(np.median(samples))
            rec[name] = {"ms": round(ms, 4), "mpix_s": round(P / (ms / 1e3) / 1e6, 1),
                         "gb_s": round(P * (esize * b + 8) / (ms / 1e3) / 1e9, 1)}
            del cube
        out[f"{h}x{w}x{b}, {t} target(s)"] = rec
        del best, bt
    torch.cuda.empty_cache()
    return {"what": "hsi_score_frames_batch (score_kernel for f32, score_h_kernel for f16): best angle + id, "
                    "one resident cube, median of 5 passes of 50 launches, as the reference's bench_sam times its "
                    "kernels (its figures: the reference arm's gpu_comparator)",
            "results": out}


def lagged_record(hsi, torch, device, frames=16, warm=3):
    """The SAM+CEM video step of the headline workload in the lagged-statistics
    mode (include/hsi_lagged.h): each 1024x1024x113 frame is scored with the
    previous frame's statistics while its own are built on a second stream,
    against the same frames each scored with its own statistics, one frame at
    a time on one stream.  Per-frame time in steady state, and the latency of
    a frame (its work on the scoring stream: statistics first, or not)."""
    import ctypes as C
    L = hsi.lib()
    sc = hsi.scene(B, n_targets=TARGETS, target_frac=0.002, library_seed=0x5EED1000)
    targets_np = hsi.scene_targets(sc)
    cubes = []
    for f in range(frames):
        s_ = hsi.scene(B, n_targets=TARGETS, target_frac=0.002, library_seed=0x5EED1000, frame_seed=0x5EED1000 + f)
        cubes.append(hsi.generate(s_, H, W, truth=False, device=device)[0])
    stream = torch.cuda.current_stream(device)
    run = hsi.Lagged(H, W, B, targets_np, detectors=hsi.LAGGED_SAM_CEM, loading=LOADING, sam_threshold=THRESHOLD,
                     cem_threshold=CEM_THRESHOLD, nms_radius=NMS_RADIUS, capacity=CAPACITY)

    def timed(push):
        for f in range(warm):
            push(cubes[f])
        torch.cuda.synchronize()
        ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(frames)]
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for f in range(frames):
            ev[f][0].record(stream)
            push(cubes[f])
            ev[f][1].record(stream)
        b.record(stream)
        torch.cuda.synchronize()
        ms = a.elapsed_time(b) / frames
        lat = float(np.median([x.elapsed_time(y) for x, y in ev]))
        return ms, lat

    lag_ms, lag_lat = timed(lambda c: run.push(c, stream))
    # the same frames, each on its own statistics, one frame at a time
    P = H * W
    tg = torch.from_numpy(targets_np).to(device)
    nr = torch.from_numpy(hsi.target_norms(targets_np)).to(device)
    moments = torch.zeros(B + B * B + 1, dtype=torch.float64, device=device)
    cem_w = torch.zeros((TARGETS, B), device=device)
    status = torch.zeros(1, dtype=torch.int32, device=device)
    sws_b = L.hsi_stats_workspace_bytes(H, W, B)
    sws = torch.empty(sws_b, dtype=torch.uint8, device=device)
    smaps = torch.empty((TARGETS, P), device=device)
    cmaps = torch.empty((TARGETS, P), device=device)
    best = [torch.empty(P, device=device) for _ in range(2)]
    bt = [torch.empty(P, dtype=torch.int32, device=device) for _ in range(2)]
    dets = torch.empty((2, CAPACITY, 4), dtype=torch.int32, device=device)
    counts = torch.zeros(2, dtype=torch.int32, device=device)
    jobs = [hsi.detect_job(best[0], bt[0], H, W, THRESHOLD, NMS_RADIUS, hsi.LOWER_IS_BETTER, CAPACITY, dets[0],
                           counts[0:1]),
            hsi.detect_job(best[1], bt[1], H, W, CEM_THRESHOLD, NMS_RADIUS, hsi.HIGHER_IS_BETTER, CAPACITY, dets[1],
                           counts[1:2])]
    dws = torch.empty(hsi.detect_batch_workspace_bytes(jobs), dtype=torch.uint8, device=device)
    s = C.c_void_p(stream.cuda_stream)
    vp = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731

    def own(cube):
        stride = cube.shape[-1]
        hsi.check(L.hsi_scene_moments(vp(cube), H, W, B, 0, stride, vp(moments), None, vp(sws), sws_b, s), "moments")
        hsi.check(L.hsi_build_statistics(1, B, TARGETS, LOADING, vp(moments), vp(tg), 0, None, None, vp(cem_w),
                                         vp(status), None, 0, s), "statistics")
        hsi.score_frames([hsi.make_frame(cube, H, W, B, 0, sam_targets=tg, sam_norms=nr, cem_weights=cem_w,
                                         sam_maps=smaps, sam_best=best[0], sam_best_target=bt[0], cem_maps=cmaps,
                                         cem_best=best[1], cem_best_target=bt[1], map_stride=P)], stream=stream)
        counts.zero_()
        hsi.detect_batch(jobs, dws, stream=stream)

    own_ms, own_lat = timed(own)
    run.close()
    del cubes, sws, smaps, cmaps, best, bt, dets, dws
    torch.cuda.empty_cache()
    return {"what": f"{frames} frames of {H}x{W}x{B} f32, {TARGETS} targets, SAM+CEM maps and both lists, pushed "
                    "one at a time (median latency = the frame's work on the scoring stream)",
            "lagged": {"ms_per_frame": round(lag_ms, 3), "mpix_s": round(P / (lag_ms / 1e3) / 1e6, 1),
                       "latency_ms": round(lag_lat, 3)},
            "own_statistics": {"ms_per_frame": round(own_ms, 3), "mpix_s": round(P / (own_ms / 1e3) / 1e6, 1),
                               "latency_ms": round(own_lat, 3)}}


def extra_records(args, device, line):
    """The default run's other records, each measured after the headline
    (single GPU only): the RX+ACE precision workload, the learned screen, the
    SAM scorer at the shapes of the reference's GPU comparator, and the
    SAM+CEM video in the lagged-statistics mode."""
    import torch
    import hsi_b200 as hsi
    sub = argparse.Namespace(**vars(args))
    sub.steps, sub.warmup, sub.no_e2e = min(max(args.steps, 3), 10), 3, True
    for key, fn in (("rx_ace", measure_rxace), ("screen", measure_screen)):
        try:
            rec = fn(sub, None, 1, 0, device)
            rec.pop("e2e", None)
            line[key] = rec
        except Exception as e:  # reported, never hidden
            line[key] = {"error": f"{type(e).__name__}: {e}"}
        torch.cuda.empty_cache()
    try:
        line["same_shape_scorer"] = same_shape_scorer(hsi, torch, device)
    except Exception as e:
        line["same_shape_scorer"] = {"error": f"{type(e).__name__}: {e}"}
    try:
        line["lagged_statistics"] = lagged_record(hsi, torch, device)
    except Exception as e:
        line["lagged_statistics"] = {"error": f"{type(e).__name__}: {e}"}


# DRAM bytes (read + write) per frame of the scoring kernel, from the ncu
# captures summarised in profiles/ (score_kernel_samcem8_f32_4x1024x1024x113.md:
# 2.216 GB for a 4-frame launch; rxace_tc_kernel_f32_2048x1024x113.md: one
# frame).  The scorer's traffic grows with the frames in the launch.
TRAFFIC_PER_FRAME = {"sam_cem": 554.08e6, "rx_ace": 1035.63e6}


def load_traffic(workload, frames):
    """DRAM bytes per launch of the dominant kernel, scaled from the capture."""
    per = TRAFFIC_PER_FRAME.get(workload)
    return None if per is None else round(per * frames)


def run_e2e(hsi, torch, wl, stream, args, world):
    """Same step through the C ABI with host buffers: each frame's cube is copied
    from pinned host memory, scored and thresholded, and its detection list and
    count read back, with copies on a second stream overlapping the scoring."""
    nslots = 3
    host = [torch.empty_like(wl.cubes[i], device="cpu").pin_memory() for i in range(nslots)]
    for i in range(nslots):
        host[i].copy_(wl.cubes[i])
    dev = [torch.empty_like(wl.cubes[0]) for _ in range(nslots)]
    copy_stream = torch.cuda.Stream(device=stream.device)
    out_host = torch.empty((args.frames, CAPACITY, 4), dtype=torch.int32).pin_memory()
    count_host = torch.empty((args.frames,), dtype=torch.int32).pin_memory()
    copied = [torch.cuda.Event() for _ in range(nslots)]
    freed = [torch.cuda.Event() for _ in range(nslots)]
    frames = []
    for i in range(nslots):
        kw = dict(sam_targets=wl.targets, sam_norms=wl.norms, sam_maps=wl.sam_maps[i], sam_best=wl.sam_best[i],
                  sam_best_target=wl.sam_bt[i], map_stride=wl.P)
        if wl.cem:
            kw.update(cem_weights=wl.cem_w[i], cem_maps=wl.cem_maps[i], cem_best=wl.cem_best[i],
                      cem_best_target=wl.cem_bt[i])
        frames.append(hsi.make_frame(dev[i], H, W, B, wl.dtype, **kw))
    import ctypes as C
    L = hsi.lib()
    s = C.c_void_p(stream.cuda_stream)

    def one_step():
        launches = 0
        for f in range(args.frames):
            i = f % nslots
            with torch.cuda.stream(copy_stream):
                copy_stream.wait_event(freed[i])
                dev[i].copy_(host[i], non_blocking=True)
                copied[i].record(copy_stream)
            stream.wait_event(copied[i])
            if wl.cem:
                hsi.check(L.hsi_scene_moments(C.c_void_p(dev[i].data_ptr()), H, W, B, wl.dtype, wl.stride,
                                              C.c_void_p(wl.moments[i].data_ptr()), None,
                                              C.c_void_p(wl.stats_ws.data_ptr()), wl.stats_bytes, s), "moments")
                hsi.check(L.hsi_build_statistics(1, B, TARGETS, LOADING, C.c_void_p(wl.moments[i].data_ptr()),
                                                 C.c_void_p(wl.targets.data_ptr()), 0, None, None,
                                                 C.c_void_p(wl.cem_w[i].data_ptr()),
                                                 C.c_void_p(wl.status[i:i + 1].data_ptr()), None, 0, s), "stats")
                launches += moments_launches([(H * W, B)]) + 1
            hsi.score_frames([frames[i]], stream=stream)
            freed[i].record(stream)
            wl.counts[f:f + 1].zero_()
            hsi.detect(wl.sam_best[i], wl.sam_bt[i], H, W, THRESHOLD, NMS_RADIUS, hsi.LOWER_IS_BETTER, CAPACITY,
                       out=wl.dets[f], count=wl.counts[f:f + 1], workspace=wl.ws[f], stream=stream)
            launches += 1 + detect_launches()
        out_host.copy_(wl.dets, non_blocking=True)
        count_host.copy_(wl.counts, non_blocking=True)
        return launches

    for _ in range(max(1, args.warmup)):
        one_step()
    torch.cuda.synchronize()
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record(stream)
    for _ in range(args.steps):
        one_step()
    end.record(stream)
    torch.cuda.synchronize()
    ms = start.elapsed_time(end) / args.steps
    if world > 1:
        import torch.distributed as dist
        ms = max_over_ranks(dist, [ms], stream.device)[0]
    value = world * args.frames * H * W / (ms / 1e3) / 1e6
    h2d = args.frames * host[0].numel() * host[0].element_size()
    d2h = out_host.numel() * 4 + count_host.numel() * 4
    return {"value": round(value, 2), "unit": "Mpix/s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
            "ms_per_step": round(ms, 3), "path": "C ABI (hsi_score_frames + hsi_detect) from pinned host cubes"}


# ---------------------------------------------------------------------------
# RX + ACE precision workload: one 2048 x 1024 x 113 frame, 8 ACE targets
# ---------------------------------------------------------------------------

RX_H, RX_W = 2048, 1024


def _fp64_reference(torch, cube, H, Wd, lib, rows):
    """Plain torch FP64 RX/ACE on the first `rows` rows, from FP64 statistics of
    the whole frame (the error reference; not the measured path)."""
    P = H * Wd
    x = cube[:, :P].double()
    mu = x.mean(dim=1)
    xc = x - mu[:, None]
    S = (xc @ xc.T) / P + LOADING * torch.eye(B, dtype=torch.float64, device=cube.device)
    Lc = torch.linalg.cholesky(S)
    Wm = torch.linalg.solve_triangular(Lc, torch.eye(B, dtype=torch.float64, device=cube.device), upper=False)
    U = Wm @ (lib.double() - mu[None, :]).T          # B x T
    uu = (U * U).sum(dim=0)
    z = Wm @ xc[:, :rows * Wd]
    rx = (z * z).sum(dim=0)
    maps = (U.T @ z) ** 2 / (uu[:, None] * rx[None, :])
    return rx, maps


def init_ranks(timeout_s=300):
    """(torch, dist or None, world, rank, device) for a one-process-per-GPU run."""
    import torch
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", init_method="env://",
                                timeout=__import__("datetime").timedelta(seconds=timeout_s))
    device = torch.device("cuda", local if world > 1 else 0)
    torch.cuda.set_device(device)
    return torch, dist, world, rank, device


def run_rxace(args):
    torch, dist, world, rank, device = init_ranks()
    line = measure_rxace(args, dist, world, rank, device)
    if rank == 0:
        print(json.dumps(line), flush=True)
    if dist:
        dist.destroy_process_group()


def measure_rxace(args, dist, world, rank, device):
    """The RX+ACE precision workload; returns its JSON record."""
    import ctypes as C
    import torch
    import hsi_b200 as hsi

    L = hsi.lib()
    H, Wd, T = RX_H, RX_W, TARGETS
    P = H * Wd
    sc = hsi.scene(B, n_targets=T, target_frac=0.002, anomaly_frac=0.001, library_seed=0x5EED2000,
                   frame_seed=rank_seed(0x5EED2001, rank))
    cube, _ = hsi.generate(sc, H, Wd, truth=False, device=device)
    stride = hsi.plane_stride(H, Wd)
    lib = torch.from_numpy(hsi.scene_targets(sc)).to(device)
    moments = torch.zeros(B + B * B + 1, dtype=torch.float64, device=device)
    stats64 = torch.zeros(L.hsi_statistics_elements(B, T), dtype=torch.float64, device=device)
    status = torch.zeros(1, dtype=torch.int32, device=device)
    sws_b = L.hsi_stats_workspace_bytes(H, Wd, B)
    sws = torch.empty(sws_b, dtype=torch.uint8, device=device)
    rx = torch.empty(P, device=device)
    ab = torch.empty(P, device=device)
    at = torch.empty(P, dtype=torch.int32, device=device)
    maps = torch.empty((T, P), device=device)
    tws_b = L.hsi_rx_ace_workspace_bytes(B, T)
    tws = torch.empty(tws_b, dtype=torch.uint8, device=device)
    pws_b = L.hsi_rx_ace_simt_workspace_bytes(B, T)
    pws = torch.empty(pws_b, dtype=torch.uint8, device=device)
    stream = torch.cuda.current_stream(device)
    s = C.c_void_p(stream.cuda_stream)
    vp = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731

    def statistics(src):
        hsi.check(L.hsi_scene_moments(vp(src), H, Wd, B, 0, stride, vp(moments), None, vp(sws), sws_b, s), "moments")
        hsi.check(L.hsi_build_statistics(1, B, T, LOADING, vp(moments), vp(lib), 0, vp(stats64), None, None,
                                         vp(status), None, 0, s), "statistics")

    def score(src, plain):
        fn = L.hsi_rx_ace_simt if plain else L.hsi_rx_ace
        ws, wb = (pws, pws_b) if plain else (tws, tws_b)
        hsi.check(fn(vp(src), H, Wd, B, 0, stride, vp(stats64), T, vp(rx), vp(ab), vp(at), vp(maps), P, vp(ws), wb,
                     s), "rx_ace")

    def timed(plain, steps, warmup):
        ev = [tuple(torch.cuda.Event(enable_timing=True) for _ in range(3)) for _ in range(steps)]
        for _ in range(warmup):
            statistics(cube)
            score(cube, plain)
        torch.cuda.synchronize()
        if dist:
            dist.barrier()
        torch.cuda.synchronize()
        for k in range(steps):
            ev[k][0].record(stream)
            statistics(cube)
            ev[k][1].record(stream)
            score(cube, plain)
            ev[k][2].record(stream)
        torch.cuda.synchronize()
        step = float(np.mean([a.elapsed_time(c) for a, _, c in ev]))
        kern = float(np.mean([b.elapsed_time(c) for _, b, c in ev]))
        return step, kern

    props = torch.cuda.get_device_properties(device)
    uuid = getattr(props, "uuid", None)
    uuid = f"GPU-{uuid}" if uuid is not None and not str(uuid).startswith("GPU-") else (str(uuid) if uuid else None)
    with ClockSampler(uuid) as clocks:
        ms, kern_ms = timed(False, args.steps, args.warmup)
    plain_ms, plain_kern = timed(True, max(2, args.steps // 2), 1)
    ms, kern_ms, plain_ms, plain_kern = max_over_ranks(dist, [ms, kern_ms, plain_ms, plain_kern], device)

    # error of the measured path against a torch FP64 reference on every pixel
    statistics(cube)
    score(cube, False)
    torch.cuda.synchronize()
    rows = H
    rx64, maps64 = _fp64_reference(torch, cube, H, Wd, lib, rows)
    n = rows * Wd
    rx_err = ((rx[:n].double() - rx64).abs() / rx64.abs().clamp(min=1.0))
    map_err = (maps[:, :n].double() - maps64).abs()
    best64 = maps64.clamp(0, 1).max(dim=0).values
    ace_err = (ab[:n].double() - best64).abs()
    del rx64, maps64, best64
    errors = {"reference": f"torch FP64 statistics and FP64 scores of the whole frame ({n} px, every pixel)",
              "rx_rel": {"max": float(rx_err.max()), "mean": float(rx_err.mean())},
              "ace_best_abs": {"max": float(ace_err.max()), "mean": float(ace_err.mean())},
              "ace_maps_abs": {"max": [float(v) for v in map_err.max(dim=1).values],
                               "mean": [float(v) for v in map_err.mean(dim=1)]}}

    e2e = None
    dev = None
    if not args.no_e2e:
        host = torch.empty_like(cube, device="cpu").pin_memory()
        host.copy_(cube)
        dev = torch.empty_like(cube)
        out_host = torch.empty((2, P), dtype=torch.float32).pin_memory()

        def e2e_step():
            dev.copy_(host, non_blocking=True)
            statistics(dev)
            score(dev, False)
            out_host[0].copy_(rx, non_blocking=True)
            out_host[1].copy_(ab, non_blocking=True)
        e2e_step()
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for _ in range(args.steps):
            e2e_step()
        b.record(stream)
        torch.cuda.synchronize()
        e_ms = a.elapsed_time(b) / args.steps
        e2e = {"value": round(world * P / (e_ms / 1e3) / 1e6, 2), "unit": "Mpix/s",
               "h2d_bytes_per_step": host.numel() * host.element_size(), "d2h_bytes_per_step": out_host.numel() * 4,
               "ms_per_step": round(e_ms, 3), "path": "C ABI (hsi_scene_moments + hsi_build_statistics + hsi_rx_ace)"}

    del cube, dev
    torch.cuda.empty_cache()
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        cpu = cpu_baseline("rx_ace", " (moments + statistics + ace_best_cpu with RX)")
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(REPO, "MEASURED_PEAKS.json")))
    except Exception:
        pass
    hbm = float(peaks.get("hbm_gbs", 6650.0))
    per_px = 4 * B + 4 + 4 * T + 8  # cube + RX + ACE maps + best score / id
    ach = P * per_px / (kern_ms / 1e3) / 1e9
    if rank == 0:
        line = {
            "metric": metric_name("rx_ace"), "value": round(world * P / (ms / 1e3) / 1e6, 2), "unit": "Mpix/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms, 3),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int8-limb/f32",
            "data": "synthetic (seeded scene model generated on the device, 0.1% anomalies)",
            "config": dict(workload_config("rx_ace", 1), parallelism=f"one frame per GPU over {world} GPU(s)"),
            "roofline": {"kernel": "rxace_tc_kernel (+ its prep)", "bound": "hbm", "achieved": round(ach, 1),
                         "peak": hbm, "unit": "GB/s", "frac": round(ach / hbm, 4),
                         "traffic": load_traffic("rx_ace", 1),
                         "kernel_ms": round(kern_ms, 3), "algorithmic_bytes_per_launch": P * per_px},
            "plain_fp32": {"step_ms": round(plain_ms, 3), "kernel_ms": round(plain_kern, 3),
                           "step_mpix_s": round(world * P / (plain_ms / 1e3) / 1e6, 2),
                           "kernel_mpix_s": round(P / (plain_kern / 1e3) / 1e6, 1),
                           "tensor_core_speedup": round(plain_kern / kern_ms, 2),
                           "step_speedup": round(plain_ms / ms, 2)},
            "errors_vs_fp64": errors,
            "cpu_baseline": cpu, "e2e": e2e,
            "gpu_launches": args.steps * (moments_launches([(P, B)]) + 1 + rx_ace_launches(B, T, True)), "clocks": clocks.summary(),
        }
    del rx, ab, at, maps, sws, tws, pws
    torch.cuda.empty_cache()
    return line if rank == 0 else None


# ---------------------------------------------------------------------------
# Learned screen: train on 512 x 512 x 224 frames, infer on 2048 x 2048 x 224 fp16
# ---------------------------------------------------------------------------

SCR_B, SCR_T = 224, 16
SCR_TRAIN_HW = 512
SCR_H = SCR_W = 2048
SCR_ACE = 0.5          # plain ACE decision threshold (fixed; the configuration gives none)
SCR_RECALL = 0.9995    # calibration target on the last 20 training frames
SCR_CAP = 1 << 18      # compact re-score capacity; beyond it the plain detector runs on the whole frame


def run_screen(args):
    torch, dist, world, rank, device = init_ranks(600)
    line = measure_screen(args, dist, world, rank, device)
    if rank == 0:
        print(json.dumps(line), flush=True)
    if dist:
        dist.destroy_process_group()


def measure_screen(args, dist, world, rank, device):
    """The learned-screen workload (training, then inference against plain ACE);
    returns its JSON record."""
    import ctypes as C
    import torch
    import hsi_b200 as hsi

    L = hsi.lib()
    Bs, T = SCR_B, SCR_T
    lib_seed = 0x5EED5000
    lib_t = torch.from_numpy(hsi.scene_targets(hsi.scene(Bs, n_targets=T, library_seed=lib_seed))).to(device)
    vp = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731

    def frame_stats(cube, h, w):
        gm = hsi.scene_moments(cube, h, w, Bs, dtype=1)
        s64, _, st = hsi.build_statistics(gm, Bs, lib_t, loading=LOADING)
        return gm, s64[0], st

    def plain_ace(cube, h, w, s64, out):
        hsi.rx_ace(cube, h, w, Bs, s64, T, dtype=1, ace_best=out, simt=True)

    # ---- training (not timed as a step; its wall time is reported) ----
    screen = hsi.Screen(Bs, seed=1, device=device)
    t0 = time.perf_counter()
    calib = []
    hw = SCR_TRAIN_HW
    ace_tr = torch.zeros(hw * hw, device=device)
    for f in range(args.train_frames):
        sc = hsi.scene(Bs, n_targets=T, target_frac=0.002, anomaly_frac=0.001, library_seed=lib_seed,
                       frame_seed=0x5EED5100 + f)
        cube, _ = hsi.generate(sc, hw, hw, dtype=1, truth=False, device=device)
        gm, s64, _ = frame_stats(cube, hw, hw)
        plain_ace(cube, hw, hw, s64, ace_tr)
        norm = hsi.screen_normaliser(gm, Bs)
        if args.profile_range and f == 0:
            torch.cuda.synchronize()
            torch.cuda.profiler.start()
        screen.train_on(cube, hw, hw, 1, norm, ace_tr, SCR_ACE, steps=20, batch=8192, seed=f, lr=1e-3)
        if args.profile_range and f == 0:
            torch.cuda.synchronize()
            torch.cuda.profiler.stop()
        if f >= args.train_frames - 20:
            lg = screen.logits(cube, hw, hw, norm)
            calib.append((lg[ace_tr >= SCR_ACE]).clone())
    pos = torch.cat(calib).sort().values
    thr = float(pos[int(np.floor((1.0 - SCR_RECALL) * pos.numel()))].item()) - 1e-3
    torch.cuda.synchronize()
    train_s = time.perf_counter() - t0
    del calib, pos

    # ---- inference frame ----
    H, Wd = SCR_H, SCR_W
    P = H * Wd
    sc = hsi.scene(Bs, n_targets=T, target_frac=0.002, anomaly_frac=0.001, library_seed=lib_seed,
                   frame_seed=rank_seed(0x5EED5900, rank))
    cube, _ = hsi.generate(sc, H, Wd, dtype=1, truth=False, device=device)
    stride = cube.shape[-1]
    moments = torch.zeros(Bs + Bs * Bs + 1, dtype=torch.float64, device=device)
    stats64 = torch.zeros(L.hsi_statistics_elements(Bs, T), dtype=torch.float64, device=device)
    status = torch.zeros(1, dtype=torch.int32, device=device)
    sws_b = L.hsi_stats_workspace_bytes(H, Wd, Bs)
    sws = torch.empty(sws_b, dtype=torch.uint8, device=device)
    fws_b = L.hsi_factor_workspace_bytes(1, Bs)
    fws = torch.empty(max(fws_b, 256), dtype=torch.uint8, device=device)
    norm = torch.zeros(2 * 256, device=device)
    logits = torch.empty(P, device=device)
    ace_full = torch.empty(P, device=device)
    cand = torch.zeros((SCR_CAP, 4), dtype=torch.int32, device=device)
    ccount = torch.zeros(1, dtype=torch.int32, device=device)
    dws = torch.empty(L.hsi_detect_workspace_bytes(H, Wd), dtype=torch.uint8, device=device)
    compact = torch.empty((Bs, SCR_CAP), dtype=torch.float16, device=device)
    ace_c = torch.empty(SCR_CAP, device=device)
    pws_b = L.hsi_rx_ace_simt_workspace_bytes(Bs, T)
    pws = torch.empty(pws_b, dtype=torch.uint8, device=device)
    iws = torch.empty(L.hsi_screen_infer_workspace_bytes(Bs), dtype=torch.uint8, device=device)
    dets = torch.zeros((SCR_CAP, 4), dtype=torch.int32, device=device)
    slot = torch.arange(SCR_CAP, dtype=torch.int32, device=device)
    dcount = torch.zeros(1, dtype=torch.int32, device=device)
    stream = torch.cuda.current_stream(device)
    s = C.c_void_p(stream.cuda_stream)

    # the screen needs only the moments (its normaliser): the FP64 factorisation,
    # which the re-scoring needs, runs on a side stream under the inference
    side = torch.cuda.Stream(device=device, priority=-1)  # the factorisation's cluster dispatches first
    # the screen kernel one CTA short per SM of that cluster, so the two run side by side
    screen_ctas = torch.cuda.get_device_properties(device).multi_processor_count - 2
    s_side = C.c_void_p(side.cuda_stream)
    moments_done, factor_done = torch.cuda.Event(), torch.cuda.Event()

    def factor(on):
        hsi.check(L.hsi_build_statistics(1, Bs, T, LOADING, vp(moments), vp(lib_t), 0, vp(stats64), None, None,
                                         vp(status), vp(fws), fws_b, on), "statistics")

    def statistics(src):
        hsi.check(L.hsi_scene_moments(vp(src), H, Wd, Bs, 1, stride, vp(moments), None, vp(sws), sws_b, s), "moments")
        factor(s)

    def screen_step(src, ev=None):
        """moments; then the screen, its compaction and the proposals' gather, with the
        factorisation beside them on a side stream; plain ACE on the proposals; final list"""
        if ev:
            ev[0].record(stream)
        hsi.check(L.hsi_scene_moments(vp(src), H, Wd, Bs, 1, stride, vp(moments), None, vp(sws), sws_b, s), "moments")
        moments_done.record(stream)
        side.wait_event(moments_done)
        factor(s_side)
        factor_done.record(side)
        if ev:
            ev[1].record(stream)
        hsi.check(L.hsi_screen_normaliser(vp(moments), Bs, vp(norm), s), "normaliser")
        hsi.check(L.hsi_screen_infer_ctas(vp(src), H, Wd, Bs, 1, stride, vp(norm), vp(screen.params), vp(logits),
                                          vp(iws), iws.numel(), screen_ctas, s), "screen")
        ccount.zero_()
        hsi.check(L.hsi_detect(vp(logits), None, H, Wd, C.c_float(thr), 0, hsi.HIGHER_IS_BETTER, SCR_CAP, vp(cand),
                               vp(ccount), vp(dws), dws.numel(), s), "proposals")
        hsi.check(L.hsi_gather_candidates(vp(src), 1, stride, Bs, Wd, vp(cand), vp(ccount), SCR_CAP, vp(compact),
                                          SCR_CAP, s), "gather")
        stream.wait_event(factor_done)
        hsi.check(L.hsi_rx_ace_simt(vp(compact), 1, SCR_CAP, Bs, 1, SCR_CAP, vp(stats64), T, None, vp(ace_c), None,
                                    None, SCR_CAP, vp(pws), pws_b, s), "rescore")
        ace_c.masked_fill_(slot >= ccount, 0.0)  # slots past the proposal count are padding
        dcount.zero_()
        hsi.check(L.hsi_detect(vp(ace_c), None, 1, SCR_CAP, C.c_float(SCR_ACE), 0, hsi.HIGHER_IS_BETTER, SCR_CAP,
                               vp(dets), vp(dcount), vp(dws), dws.numel(), s), "final list")
        if ev:
            ev[2].record(stream)
        # moments, factorisation, normaliser, screen (pack + inference), proposals, gather, re-scoring, final list
        return moments_launches([(P, Bs)]) + 1 + 1 + 2 + detect_launches() + 1 + 2 + detect_launches()

    def plain_step(src, ev=None):
        if ev:
            ev[0].record(stream)
        statistics(src)
        if ev:
            ev[1].record(stream)
        hsi.check(L.hsi_rx_ace_simt(vp(src), H, Wd, Bs, 1, stride, vp(stats64), T, None, vp(ace_full), None, None, P,
                                    vp(pws), pws_b, s), "plain ace")
        if ev:
            ev[2].record(stream)
        return moments_launches([(P, Bs)]) + 1 + 2

    def timed(fn, steps, warmup):
        """(ms per step, ms per step after the shared statistics, launches)"""
        for _ in range(warmup):
            fn(cube)
        torch.cuda.synchronize()
        if dist:
            dist.barrier()
        ev = [tuple(torch.cuda.Event(enable_timing=True) for _ in range(3)) for _ in range(steps)]
        n = 0
        for k in range(steps):
            n += fn(cube, ev[k])
        torch.cuda.synchronize()
        return (float(np.mean([a.elapsed_time(c) for a, _, c in ev])),
                float(np.mean([b.elapsed_time(c) for _, b, c in ev])), n)

    props = torch.cuda.get_device_properties(device)
    uuid = getattr(props, "uuid", None)
    uuid = f"GPU-{uuid}" if uuid is not None and not str(uuid).startswith("GPU-") else (str(uuid) if uuid else None)
    if args.profile_range:
        screen_step(cube)
        torch.cuda.synchronize()
        torch.cuda.profiler.start()
        screen_step(cube)
        torch.cuda.synchronize()
        torch.cuda.profiler.stop()
    with ClockSampler(uuid) as clocks:
        ms, score_ms, launches = timed(screen_step, args.steps, args.warmup)
    plain_ms, plain_score_ms, _ = timed(plain_step, max(2, args.steps // 2), 1)
    # screen-only kernel time
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    ev[0].record(stream)
    hsi.check(L.hsi_screen_infer(vp(cube), H, Wd, Bs, 1, stride, vp(norm), vp(screen.params), vp(logits), vp(iws),
                                 iws.numel(), s), "screen")
    ev[1].record(stream)
    torch.cuda.synchronize()
    screen_ms = ev[0].elapsed_time(ev[1])
    ms, plain_ms, screen_ms, score_ms, plain_score_ms = max_over_ranks(
        dist, [ms, plain_ms, screen_ms, score_ms, plain_score_ms], device)

    # quality against plain ACE on the whole frame
    screen_step(cube)
    plain_step(cube)
    torch.cuda.synchronize()
    nprop = int(ccount.item())
    plain_pos = ace_full >= SCR_ACE
    proposed = logits >= thr
    n_plain = int(plain_pos.sum())
    missed = int((plain_pos & ~proposed).sum())
    false_prop = int((proposed & ~plain_pos).sum())
    # the screen path's own detections equal plain ACE on every proposed pixel
    n_keep = min(nprop, SCR_CAP)
    cc = cand[:n_keep].long()
    agree = bool(torch.equal(ace_c[:n_keep], ace_full[cc[:, 1] * Wd + cc[:, 0]])) if n_keep else True

    peaks = {}
    try:
        peaks = json.load(open(os.path.join(REPO, "MEASURED_PEAKS.json")))
    except Exception:
        pass
    hbm = float(peaks.get("hbm_gbs", 6650.0))
    per_px = 2 * Bs + 4  # fp16 cube read once + one logit
    ach = P * per_px / (screen_ms / 1e3) / 1e9
    if rank == 0:
        line = {
            "metric": metric_name("screen"), "value": round(world * P / (ms / 1e3) / 1e6, 2), "unit": "Mpix/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms, 3),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f16/bf16",
            "data": "synthetic (seeded scene model generated on the device)",
            "config": {"workload": f"one {H}x{Wd}x{Bs} fp16 frame per GPU, {T} ACE targets: statistics + learned "
                                   "screen (tcgen05) + plain ACE re-scoring of the proposals + detection list",
                       "height": H, "width": Wd, "bands": Bs, "targets": T, "ace_threshold": SCR_ACE,
                       "training": f"{args.train_frames} frames of {SCR_TRAIN_HW}x{SCR_TRAIN_HW}x{Bs}, 20 Adam "
                                   "steps of 8192 pixels each, labels = plain ACE >= 0.5",
                       "proposal_threshold": round(thr, 4), "calibrated_recall": SCR_RECALL,
                       "l2": "inputs larger than L2 (1.88 GB cube)",
                       "parallelism": f"one frame per GPU over {world} GPU(s)"},
            "roofline": {"kernel": "screen_tc_kernel", "bound": "hbm", "achieved": round(ach, 1), "peak": hbm,
                         "unit": "GB/s", "frac": round(ach / hbm, 4), "traffic": None,
                         "kernel_ms": round(screen_ms, 3), "algorithmic_bytes_per_launch": P * per_px},
            "plain_ace": {"step_ms": round(plain_ms, 3), "mpix_s": round(world * P / (plain_ms / 1e3) / 1e6, 2),
                          "speedup_with_screen": round(plain_ms / ms, 2),
                          "statistics_ms_shared": round(plain_ms - plain_score_ms, 3),
                          "moments_ms_screen_arm": round(ms - score_ms, 3),
                          "scoring_ms": {"screen_path": round(score_ms, 3), "plain": round(plain_score_ms, 3)},
                          "scoring_speedup_with_screen": round(plain_score_ms / score_ms, 2),
                          "note": "both arms compute the same moments and FP64 statistics; the screen arm runs "
                                  "the factorisation on a side stream under the screen (the screen needs only the "
                                  "moments) and joins before the re-scoring, so its screen_path time after the "
                                  "moments includes what of the factorisation the screen did not hide"},
            "quality_vs_plain_ace": {"plain_detections": n_plain, "missed": missed,
                                     "miss_rate": round(missed / max(n_plain, 1), 6),
                                     "proposals": int(proposed.sum()), "proposal_share": round(int(proposed.sum()) / P, 5),
                                     "false_proposal_rate": round(false_prop / max(int(proposed.sum()), 1), 5),
                                     "rescored_equals_plain": agree, "fallback": nprop > SCR_CAP},
            "train_seconds": round(train_s, 2),
            "cpu_baseline": None, "e2e": None, "gpu_launches": launches, "clocks": clocks.summary(),
        }
    del cube, logits, ace_full, compact, screen
    torch.cuda.empty_cache()
    return line if rank == 0 else None


# ---------------------------------------------------------------------------
# Batched stream: 32 uneven frames, band counts 16 (mosaic) / 113 / 224
# ---------------------------------------------------------------------------

BATCH_FRAMES = 32


def batch_specs(seed=0x5EED7000):
    """(height, width, bands, targets, mosaic) of the 32 frames: sides log-uniform
    in [256, 2048] x [256, 1024], bands cycling 16 (4x4 mosaic) / 113 / 224,
    1..16 targets."""
    rng = np.random.default_rng(seed)
    specs = []
    for i in range(BATCH_FRAMES):
        h = int(np.exp(rng.uniform(np.log(256), np.log(2048)))) // 8 * 8
        w = int(np.exp(rng.uniform(np.log(256), np.log(1024)))) // 8 * 8
        b = (16, 113, 224)[i % 3]
        specs.append((h, w, b, int(rng.integers(1, 17)), b == 16))
    return specs


def run_batch(args):
    import torch
    import hsi_b200 as hsi

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", init_method="env://", timeout=__import__("datetime").timedelta(seconds=600))
    device = torch.device("cuda", local if world > 1 else 0)
    torch.cuda.set_device(device)
    specs = batch_specs(0x5EED7000 + rank)
    frames, pixels, cube_bytes = [], 0, 0
    for i, (h, w, b, t, mosaic) in enumerate(specs):
        sc = hsi.scene(b, n_targets=t, target_frac=0.003, anomaly_frac=0.001, library_seed=0x5EED7100 + i,
                       frame_seed=rank_seed(0x5EED7200, rank) + i)
        cube, _ = hsi.generate(sc, h, w, truth=False, device=device)
        targets = hsi.scene_targets(sc)
        if mosaic:
            c = cube[:, :h * w].reshape(b, h, w)
            raw = torch.zeros((4 * h, 4 * w), device=device)
            for k in range(b):
                oy, ox = divmod(k, 4)
                raw[oy::4, ox::4] = c[k]
            frames.append(dict(raw=raw, period=4, bands=b, targets=targets))
            del cube
        else:
            frames.append(dict(cube=cube, height=h, width=w, bands=b, dtype=0, targets=targets))
        pixels += h * w
        cube_bytes += h * w * b * 4
    t0 = time.perf_counter()
    batch = hsi.Batch(frames, sam_threshold=THRESHOLD, capacity=CAPACITY, autotune=True)
    create_s = time.perf_counter() - t0
    stream = torch.cuda.Stream(device=device)
    batch.run(stream)
    batch.capture(stream)
    for _ in range(args.warmup):
        batch.launch(stream)
    stream.synchronize()
    if args.profile_range:
        torch.cuda.profiler.start()
        batch.launch(stream)
        stream.synchronize()
        torch.cuda.profiler.stop()
    if dist:
        dist.barrier()

    def timed(fn, steps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for _ in range(steps):
            fn(stream)
        b.record(stream)
        stream.synchronize()
        return a.elapsed_time(b) / steps

    props = torch.cuda.get_device_properties(device)
    uuid = getattr(props, "uuid", None)
    uuid = f"GPU-{uuid}" if uuid is not None and not str(uuid).startswith("GPU-") else (str(uuid) if uuid else None)
    with ClockSampler(uuid) as clocks:
        ms = timed(batch.launch, args.steps)
    eager_ms = timed(batch.run, max(2, args.steps // 2))
    ms, eager_ms = max_over_ranks(dist, [ms, eager_ms], device)
    tuning = batch.tuning()
    launches = args.steps * batch_launches(specs)
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(REPO, "MEASURED_PEAKS.json")))
    except Exception:
        pass
    hbm = float(peaks.get("hbm_gbs", 6650.0))
    # algorithmic bytes: each cube read by the moments, SAM and RX/ACE passes + five maps written
    step_bytes = 3 * cube_bytes + 20 * pixels
    if rank == 0:
        line = {
            "metric": metric_name("batch"), "value": round(world * pixels / (ms / 1e3) / 1e6, 2), "unit": "Mpix/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms, 3),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic (seeded scene model generated on the device; 16-band frames as 4x4 mosaics)",
            "config": {"workload": f"{BATCH_FRAMES} frames of uneven sizes (256..2048 x 256..1024), bands 16 "
                                   "(mosaic, demosaiced in the run) / 113 / 224, 1-16 targets each: demosaic, "
                                   "statistics, SAM (one persistent launch), RX + ACE, three detection lists per "
                                   "frame, replayed as one CUDA graph",
                       "frames": BATCH_FRAMES, "pixels_per_step": pixels, "cube_bytes": cube_bytes,
                       "l2": f"inputs larger than L2 ({cube_bytes / 1e9:.1f} GB of cubes)",
                       "parallelism": f"one batch per GPU over {world} GPU(s)"},
            "roofline": {"kernel": "whole step (moments, SAM, RX/ACE passes over each cube)", "bound": "hbm",
                         "achieved": round(step_bytes / (ms / 1e3) / 1e9, 1), "peak": hbm, "unit": "GB/s",
                         "frac": round(step_bytes / (ms / 1e3) / 1e9 / hbm, 4), "traffic": None},
            "eager": {"ms_per_step": round(eager_ms, 3), "graph_speedup": round(eager_ms / ms, 3)},
            "autotune": dict(tuning, create_seconds=round(create_s, 2)),
            "cpu_baseline": None, "e2e": None, "gpu_launches": launches, "clocks": clocks.summary(),
        }
        print(json.dumps(line), flush=True)
    batch.close()
    if dist:
        dist.destroy_process_group()


def run_bip(args):
    """SAM of BIP (pixel-interleaved) frames with the transpose fused into the
    scorer (hsi_sam_bip): 16 frames of 1024x1024x113 f32, 8 targets, best angle
    + id + 8 maps, against the standalone transpose followed by the BSQ scorer."""
    import ctypes as C
    torch, dist, world, rank, device = init_ranks()
    import hsi_b200 as hsi
    L = hsi.lib()
    frames = 16
    P = H * W
    sc = hsi.scene(B, n_targets=TARGETS, target_frac=0.002, library_seed=0x5EED1000)
    tnp = hsi.scene_targets(sc)
    tg = torch.from_numpy(tnp).to(device)
    nr = torch.from_numpy(hsi.target_norms(tnp)).to(device)
    bips = []
    for f in range(frames):
        s_ = hsi.scene(B, n_targets=TARGETS, target_frac=0.002, library_seed=0x5EED1000,
                       frame_seed=rank_seed(0x5EED1000, rank) + f)
        cube, _ = hsi.generate(s_, H, W, truth=False, device=device)
        bips.append(cube[:, :P].t().contiguous())
        del cube
    maps = torch.empty((TARGETS, P), device=device)
    best = torch.empty(P, device=device)
    bt = torch.empty(P, dtype=torch.int32, device=device)
    stride = hsi.plane_stride(H, W)
    bsq = torch.empty((B, stride), device=device)
    stream = torch.cuda.current_stream(device)
    s = C.c_void_p(stream.cuda_stream)
    vp = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731

    def fused(k):
        hsi.check(L.hsi_sam_bip(vp(bips[k]), H, W, B, vp(tg), vp(nr), TARGETS, vp(maps), P, vp(best), vp(bt), s),
                  "sam_bip")

    def two_pass(k):
        hsi.check(L.hsi_transpose_bip_to_bsq(vp(bips[k]), vp(bsq), H, W, B, stride, s), "transpose")
        hsi.score_frames([hsi.make_frame(bsq, H, W, B, 0, sam_targets=tg, sam_norms=nr, sam_maps=maps, sam_best=best,
                                         sam_best_target=bt, map_stride=P)], stream=stream)

    def timed(fn, steps, warmup):
        for k in range(warmup):
            fn(k % frames)
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for k in range(steps * frames):
            fn(k % frames)
        b.record(stream)
        torch.cuda.synchronize()
        return a.elapsed_time(b) / steps

    props = torch.cuda.get_device_properties(device)
    uuid = getattr(props, "uuid", None)
    uuid = f"GPU-{uuid}" if uuid is not None and not str(uuid).startswith("GPU-") else (str(uuid) if uuid else None)
    with ClockSampler(uuid) as clocks:
        ms = timed(fused, args.steps, args.warmup)
    ms2 = timed(two_pass, max(1, args.steps // 2), 1)
    ms, ms2 = max_over_ranks(dist, [ms, ms2], device)
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(REPO, "MEASURED_PEAKS.json")))
    except Exception:
        pass
    hbm = float(peaks.get("hbm_gbs", 6650.0))
    per_px = 4 * B + 4 * TARGETS + 8
    ach = frames * P * per_px / (ms / 1e3) / 1e9
    if rank == 0:
        print(json.dumps({
            "metric": "Mpix/s SAM of BIP cubes @113 bands", "value": round(world * frames * P / (ms / 1e3) / 1e6, 2),
            "unit": "Mpix/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": round(ms, 3), "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32", "data": "synthetic (seeded scene model generated on the device, stored pixel-major)",
            "config": {"workload": f"{frames} BIP frames {H}x{W}x{B} f32, {TARGETS} targets: SAM maps + best + id",
                       "l2": "inputs larger than L2 (7.6 GB of cubes)", "parallelism": f"{world} GPU(s)"},
            "roofline": {"kernel": "sam_bip_kernel", "bound": "hbm", "achieved": round(ach, 1), "peak": hbm,
                         "unit": "GB/s", "frac": round(ach / hbm, 4), "traffic": None,
                         "algorithmic_bytes_per_launch": P * per_px},
            "transpose_then_bsq": {"ms_per_step": round(ms2, 3),
                                   "mpix_s": round(world * frames * P / (ms2 / 1e3) / 1e6, 2)},
            "cpu_baseline": None, "e2e": None, "gpu_launches": frames * args.steps, "clocks": clocks.summary(),
        }), flush=True)
    if dist:
        dist.destroy_process_group()


def main():
    args = parse()
    if args.impl == "reference":
        workload = args.workload or DEFAULT_WORKLOAD
        try:
            run_reference(args, workload)
        except Exception as e:  # the reference build is an oracle artefact; say why it is missing
            print(json.dumps({"impl": "reference", "unavailable": f"{type(e).__name__}: {e}"}), flush=True)
        return
    workload = args.workload or DEFAULT_WORKLOAD
    if workload == "rx_ace":
        run_rxace(args)
        return
    if workload == "screen":
        run_screen(args)
        return
    if workload == "batch":
        run_batch(args)
        return
    if workload == "bip":
        run_bip(args)
        return
    run_ours(args, workload)


if __name__ == "__main__":
    main()
