#!/usr/bin/env python
"""Benchmark of the unified-particle step on B200 (one JSON line on stdout).

Workload (one "step" = one frame of 5 substeps x 3 Jacobi iterations):
the reference's GPU default scene — a 20^3 = 8,000-particle body with
93,556 distance constraints and 65,536 fluid particles (deriveOpts(20,
65536, 30), seeded jittered block), with one slice wedge through the body
centre at frame 60 of the timed run.

  value        particle-substeps/s with the state resident in HBM, device
               time (CUDA events per frame, L2 flushed between frames),
               summed over all ranks (each rank steps its own replica)
  e2e          the same metric through the C ABI the way a Solver user
               drives it: per frame the uniform block goes host->device and
               positions + flags come back device->host into pinned memory
  roofline     the dominant kernel's algorithmic bytes per launch over its
               average event-timed duration, against the measured HBM peak;
               `issue` beside it: that kernel's warp instructions per launch
               (committed ncu count) over the same duration, against one
               warp instruction per scheduler per cycle at the sampled clock
  cpu_baseline the CPU solver restated (oracle O1, src/solver.js numerics),
               single thread as JavaScript runs, on a bounded sample
  clocks       nvidia-smi samples taken during the timed region

`--impl reference` times the reference's CPU implementation of the step
(O1, one substep per step) on this host instead and prints its line.
Launch for N GPUs: python -m torch.distributed.run --nproc-per-node N bench.py --gpus N
"""
from __future__ import annotations

import argparse
import json
import math
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "particle-substeps/s plain vs batched; HBM GB/s %peak; p50/p99 served frame ms"
UNIT = "particle-substeps/s"
SERVED_LOAD = 0.8  # the sustainable served stream's offered work, as a fraction of the measured capacity

# Algorithmic bytes per processed element of each kernel: every array a pass
# reads or writes counted once, neighbour re-reads counted as cache hits.
# Units: A = active particles, F = active fluid, S = solids, C = constraints,
# T = hash buckets.
KERNEL_BYTES = {
    "integrate_count": lambda u: 96 * u["A"],
    "scan": lambda u: 8 * u["T"],
    "scatter": lambda u: 20 * u["A"],
    "rankfix": lambda u: 16 * u["A"],
    "grid_build": lambda u: 8 * u["T"] + 36 * u["A"],  # scan + scatter + rankfix, one cooperative launch
    "density": lambda u: 28 * u["F"],
    "disp": lambda u: 40 * u["F"],
    "apply_fluid": lambda u: 48 * u["F"],
    "solid_solve": lambda u: 36 * u["S"] + 24 * u["C"],
    "apply_solid": lambda u: 48 * u["S"],
    "bond_contacts": lambda u: 20 * u["C"] + 40 * u["A"],
    "apply_bounds_vel": lambda u: 84 * u["A"],
    "xsph": lambda u: 52 * u["F"],
    "xsph_apply": lambda u: 32 * u["F"],
}


def log(*a):
    print(*a, file=sys.stderr, flush=True)


def measured_peaks() -> tuple[dict, str]:
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        try:
            return json.loads(p.read_text()), "measured"
        except Exception:
            pass
    return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0}, "fallback"


# Kernels that a captured frame runs on the side stream beside the main chain:
# their time is not the frame's, whatever their share of the eager launches.
SIDE_STREAM = ("solid_solve",)


def dominant_kernel(per_kernel: dict) -> str:
    """The kernel of the frame's main chain with the largest share."""
    return max((k for k in per_kernel if k in KERNEL_BYTES and k not in SIDE_STREAM), key=lambda k: per_kernel[k]["share"])


def ncu_traffic(kernel: str, workload: str):
    """DRAM bytes per launch from a committed ncu summary, if one exists:
    profiles/traffic.txt lines `kernel workload bytes_per_launch`."""
    f = ROOT / "profiles" / "traffic.txt"
    if not f.exists():
        return None
    for line in f.read_text().splitlines():
        parts = line.split()
        if len(parts) >= 3 and parts[0] == kernel and parts[1] == workload:
            try:
                return float(parts[2])
            except ValueError:
                return None
    return None


def ncu_instructions(kernel: str, workload: str):
    """Warp instructions per launch from a committed ncu summary, if one
    exists: profiles/instructions.txt lines `kernel workload count`."""
    f = ROOT / "profiles" / "instructions.txt"
    if not f.exists():
        return None
    for line in f.read_text().splitlines():
        parts = line.split()
        if len(parts) >= 3 and parts[0] == kernel and parts[1] == workload:
            try:
                return float(parts[2])
            except ValueError:
                return None
    return None


class Clocks:
    """nvidia-smi sampling during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.path = None

    def start(self):
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits", "-lms", "200",
                 "-i", str(self.index)], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self) -> dict:
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.25)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in Path(self.path).read_text().splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx.append(float(f[2]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        os.unlink(self.path)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def dist_env():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return ws, rank, local


def reduce_over_ranks(pg, ms: float, units: float, device) -> tuple[float, float]:
    """Replicas: the job's time is the slowest rank's device time, its work
    the sum of the ranks' units (no collective touches the simulation)."""
    if not pg:
        return ms, units
    import torch
    t = torch.tensor([ms], device=device, dtype=torch.float64)
    pg.all_reduce(t, op=pg.ReduceOp.MAX)
    u = torch.tensor([units], device=device, dtype=torch.float64)
    pg.all_reduce(u, op=pg.ReduceOp.SUM)
    return float(t.item()), float(u.item())


def o1_settled(o1, sc) -> str:
    """Loads the CPU solver's own state at frame 300 of the default scene
    (oracle/data, made by oracle/make_settled_o1.py) into an O1 replica of
    it: the settled pool the GPU line is timed on. Returns the start it gave
    the replica, for the JSON line."""
    settled = ROOT / "oracle" / "data" / "gpu_default_o1_frame300.npz"
    if not settled.exists():
        return "its initial state"
    z = np.load(settled)
    o1.set("pos", z["pos"])
    o1.set("prev", z["pos"])  # rewritten from pos at the start of every substep
    o1.set("vel", z["vel"])
    o1.set("active", z["active"])
    o1.set("consRest", z["consRest"])
    o1.set("consAlive", z["consAlive"])
    return f"the CPU solver's own state at frame {int(z['frames'])} (slice at frame {sc.slice_frame})"


def cpu_baseline(seconds: float = 12.0) -> dict:
    """O1 (the CPU solver restated with its JavaScript numerics) on the
    default scene, one thread, a bounded number of substeps from the CPU
    solver's own settled state (o1_settled)."""
    from fluidphysics_b200 import scenes as S
    from oracle.oracle import o1_from_scene
    sc = S.gpu_default(frames=1)
    o1 = o1_from_scene(sc)
    start = o1_settled(o1, sc)
    h = sc.dt / sc.substeps
    n_sub = 0
    parts = 0
    t0 = time.perf_counter()
    while True:
        act = int(o1.get("active").sum())
        o1.step(h, 1)
        n_sub += 1
        parts += act
        el = time.perf_counter() - t0
        if el >= seconds or n_sub >= 500:
            break
    return {"value": parts / el, "unit": UNIT, "cores": 1, "kind": "port",
            "sample": f"{n_sub} substeps of gpu_default (8,000 body + 65,536 fluid) from {start}, "
                      f"O1 restatement of src/solver.js, 1 thread, {el:.1f} s"}


def run_reference(args) -> None:
    """The reference's CPU implementation of the path (O1, the restatement of
    src/solver.js: no JavaScript engine exists on this host) on all the host's
    cores: the CPU solver is sequential (Gauss-Seidel), so every core steps
    its own replica of the default scene and the line reports the replicas'
    total particle-substeps over the wall time. A step is one substep. The
    replicas start from the CPU solver's own state at frame 300 of the
    default scene (oracle/data, made by oracle/make_settled_o1.py), the
    settled pool the GPU arm is timed on."""
    ws, rank, _ = dist_env()
    if rank != 0:
        return
    import threading

    from fluidphysics_b200 import scenes as S
    from oracle.oracle import o1_from_scene
    sc = S.gpu_default(frames=1)
    h = sc.dt / sc.substeps
    cores = max(1, len(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else (os.cpu_count() or 1))
    reps = [o1_from_scene(sc) for _ in range(cores)]
    start = [o1_settled(o, sc) for o in reps][0]
    parts = [0] * cores

    def work(k: int, steps: int, count: bool) -> None:
        o = reps[k]
        for _ in range(steps):
            if count:
                parts[k] += int(o.get("active").sum())
            o.step(h, 1)  # ctypes releases the GIL for the C++ call

    def run_all(steps: int, count: bool) -> float:
        th = [threading.Thread(target=work, args=(k, steps, count)) for k in range(cores)]
        t0 = time.perf_counter()
        for t in th:
            t.start()
        for t in th:
            t.join()
        return time.perf_counter() - t0

    run_all(args.warmup, False)
    el = run_all(args.steps, True)
    v = sum(parts) / el
    sample = (f"{args.steps} substeps of gpu_default from {start} on each of {cores} replicas, one per host "
              "thread, with O1, the restatement of src/solver.js (no JavaScript engine on this host)")
    line = {
        "impl": "reference", "metric": METRIC, "value": v, "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * el / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded jittered fluid block, lattice body)",
        "config": {"workload": "gpu_default: 20^3 body (93,556 constraints) + 65,536 fluid, 1 substep "
                               f"per step (h = 1/300), CPU solver, from {start}", "substeps_per_step": 1,
                   "replicas": cores},
        "cpu_baseline": {"value": v, "unit": UNIT, "cores": cores, "kind": "port", "sample": sample},
        "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def run_batched(args, stream, hbm: float) -> dict:
    """The uneven batch: 256 independent scenes (body dim uniform in 6..20,
    fluid log-uniform in [2k, 65k], one seed each) stepped together, one
    persistent launch per pass; grid shape autotuned first. The state (~4.3 GB)
    is far larger than L2, so no flush is needed between frames. Beside it,
    the plain per-scene path (one single-scene handle per scene, each frame
    its own captured graph) on a sample of the same scenes."""
    import torch
    from fluidphysics_b200 import _lib as L
    from fluidphysics_b200 import batch as B
    from fluidphysics_b200.sim import sim_from_scene
    dt, nsub = 1 / 60, 5
    # tuning: hash-table rule (deriveOpts's, or compact) x grid shape x cell size
    tried = []
    for rule in ("reference", "compact"):
        cand_scs = B.batch_scenes(args.batched_scenes, table=rule)
        cb = B.Batch(max_scenes=max(256, len(cand_scs)))
        cb.set_stream(stream.cuda_stream)
        cids = [cb.add_scene(sc) for sc in cand_scs]
        for _ in range(3):
            cb.step(dt, nsub)
        cb.sync()
        best_r, table_r = B.autotune(cb, dict(zip(cids, cand_scs)), dt, nsub, frames=3,
                                     block_threads=(128, 256), ctas_per_sm=(32, 64, 128, 256), cell_scales=(1.0, 1.1),
                                     warm_frames=1)
        tried.append((best_r.ms_per_frame, rule, best_r, table_r, cb, cids, cand_scs))
    tried.sort(key=lambda x: x[0])
    _, table_rule, best, table, b, ids, scs = tried[0]
    for t in tried[1:]:
        t[4].close()
    for _ in range(3):
        b.step(dt, nsub)
    b.sync()
    K = args.batched_frames
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    l0 = b.launches
    torch.cuda.synchronize()
    e0.record(stream)
    for _ in range(K):
        b.step(dt, nsub)
    e1.record(stream)
    b.sync()
    ms = e0.elapsed_time(e1)
    launches = b.launches - l0
    active, B_sub = 0, 0
    for i in ids:
        si, af = b.scene_info(i), b.active_count(i)
        active += si.solid_n + af
        # the substep's algorithmic bytes (the unit of account of the plain line)
        B_sub += (240 * (si.solid_n + af) + 200 * af + 8 * si.table_size
                  + si.solid_iters * (84 * si.solid_n + 24 * si.num_cons) + 20 * si.num_cons)
    value = active * nsub * K / (ms / 1e3)
    step_gbs = B_sub * nsub * K / (ms / 1e3) / 1e9
    # per-kernel shares of one eager frame
    msk, ln = b.profile_frame(dt, nsub)
    names = [(b.lib.upbd_kernel_name(k) or b"").decode() for k in range(L.KERNEL_KINDS)]
    shares = {names[k]: {"share": round(float(msk[k] / msk.sum()), 4),
                         "avg_us": round(float(msk[k] * 1e3 / ln[k]), 1), "launches_per_frame": int(ln[k])}
              for k in np.argsort(-msk) if ln[k]}
    info = b.info()
    b.close()
    # plain per-scene path on every 8th scene, over the same frames the batch
    # was timed on: 6 untimed frames (the batch's warm-up and tuning frames
    # leave it 6 frames in), then K timed graph frames
    sample = scs[::8]
    pp_units, pp_ms = 0.0, 0.0
    for sc in sample:
        sim = sim_from_scene(sc)
        sim.set_stream(stream.cuda_stream)
        for _ in range(6):
            sim.step(dt, nsub)
        sim.sync()
        a0, a1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a0.record(stream)
        for _ in range(K):
            sim.step(dt, nsub)
        a1.record(stream)
        sim.sync()
        pp_ms += a0.elapsed_time(a1)
        pp_units += (sc.solid_n + sim.active_count()) * nsub * K  # counted as the batched value counts
        sim.close()
    pp = pp_units / (pp_ms / 1e3)
    return {
        "value": value, "unit": UNIT, "frames": K, "scenes": len(scs), "particles": int(info.particles),
        "active_particles": int(active), "ms_per_frame": ms / K, "gpu_launches": int(launches),
        "workload": f"{len(scs)} scenes, body dim U{{6..20}}, fluid floor(2^U(11,16)), deriveOpts at 30 mm, "
                    "seeds 1000+k, 5 substeps x 3 iterations, frames 7.. of each scene",
        "l2": "state ~{:.1f} GB > L2 (no flush)".format(info.bytes_in_use / 1e9),
        "tuning": {"table_rule": table_rule, "block_threads": best.block_threads, "ctas_per_sm": best.ctas_per_sm,
                   "cell_scale": best.cell_scale,
                   "candidates_ms": {r: [[t.block_threads, t.ctas_per_sm, t.cell_scale, round(t.ms_per_frame, 2)]
                                         for t in tab] for _, r, _, tab, *_ in tried}},
        "kernels": shares,
        "step_achieved_gbs": step_gbs, "step_frac": step_gbs / hbm,
        "plain_per_scene": {"value": pp, "unit": UNIT,
                            "sample": f"{len(sample)} of the scenes (every 8th), each its own single-scene "
                                      f"handle, graph frames 7..{6 + K} (the frames the batch was timed on)"},
        "speedup_vs_plain_per_scene": value / pp,
    }


def run_large(args, stream) -> dict:
    """The large scene: 24^3 = 13,824 body + 262,144 fluid at 30 mm, a hose of
    120 particles per frame from a seeded nozzle and 64 grabbed body particles
    moved on y0 + 0.3 sin(pi t), through the single-scene handle; each frame
    timed by CUDA events. The closest scene to the reference's published
    14k body + 253k water figure (README.md:14)."""
    import torch
    from fluidphysics_b200 import scenes as S
    from fluidphysics_b200.sim import sim_from_scene
    K = args.large_frames
    sc = S.large(frames=K + 3)
    sim = sim_from_scene(sc)
    sim.set_stream(stream.cuda_stream)
    idx = S.grab_set(sim.read_state()["pos"], sc.solid_n, sc.desc.solid_dim, sc.grab_count)
    sim.grab_indices(idx)
    hose = S.hose_script(sc, K + 3)
    w = 2 * math.pi * sc.grab_freq_hz
    evs = []
    for k in range(K + 3):
        pos, dr, side, up, speed, phase = hose[k]
        sim.emit(sc.hose_per_frame, pos, dr, side, up, speed, phase)
        sim.grab_move([0.0, sc.grab_amp * (math.sin(w * (k + 1) * sc.dt) - math.sin(w * k * sc.dt)), 0.0])
        timed = k >= 3  # three warm-up frames capture the graphs
        if timed:
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
        sim.step(sc.dt, sc.substeps)
        if timed:
            b.record(stream)
            evs.append((a, b))
    sim.sync()
    ms = sum(a.elapsed_time(b) for a, b in evs)
    active = sc.solid_n + sim.active_count()
    sim.close()
    return {"value": active * sc.substeps * K / (ms / 1e3), "unit": UNIT, "ms_per_frame": ms / K, "frames": K,
            "workload": "24^3 body (13,824) + 262,144 fluid, 30 mm, hose 120/frame, 64-particle grab on "
                        "y0 + 0.3 sin(pi t), 5 substeps x 3 iterations",
            "reference_published": "19 ms per frame for 14k body + 253k water on an RTX PRO 6000 under "
                                   "WebGPU (README.md:14; other hardware, substep count unstated)"}


def _serve(reqs, bt: int, cps: int) -> tuple[dict, list]:
    """Serves one request stream to the end; returns the server's stats and
    each request's (arrival_s, done_s, frames_done, frame_ms_max, state)."""
    from fluidphysics_b200 import server as SV
    with SV.Server(hbm_budget=150 * 10**9, max_scenes=4096, block_threads=bt, ctas_per_sm=cps,
                   builders=8) as srv:
        ids = [srv.submit(r.scene, r.frames, r.arrival_s) for r in reqs]
        srv.run(900)
        st = srv.stats()
        res = []
        for rid in ids:
            q = srv.result(rid)
            res.append((q["arrival_s"], q["done_s"], q["frames_done"], q["frame_ms_max"], q["state"]))
    return st, res


def _served_block(st: dict, res: list, reqs, window: float, rate: float) -> dict:
    """One served line: throughput, frame latencies, and the request latency
    (arrival to last frame, per frame asked) of the window's first and second
    halves by arrival, so a queue that grows over the window shows."""
    offered = sum(r.scene.total * r.frames * 5 for r in reqs) / window

    def half(lo, hi):
        x = [(d - a) * 1e3 / max(f, 1) for a, d, f, m, s in res if lo <= a < hi and s == "done"]
        mx = [m for a, d, f, m, s in res if lo <= a < hi and s == "done"]
        if not x:
            return None
        return {"requests": len(x), "p50_ms_per_frame": float(np.percentile(x, 50)),
                "p99_ms_per_frame": float(np.percentile(x, 99)),
                "p99_slowest_frame_ms": float(np.percentile(mx, 99))}
    value = st["particle_substeps"] / st["wall_s"]
    return {
        "value": value, "unit": UNIT, "arrival_rate_per_s": rate, "window_s": window,
        "offered_particle_substeps_per_s": offered, "load": offered / value,
        "p50_frame_ms": st["frame_ms_p50"], "p99_frame_ms": st["frame_ms_p99"],
        "p90_frame_ms": st["frame_ms_p90"], "mean_frame_ms": st["frame_ms_mean"], "max_frame_ms": st["frame_ms_max"],
        "p50_wait_ms": st["wait_ms_p50"], "p99_wait_ms": st["wait_ms_p99"],
        "p50_batch_frame_ms": st["batch_ms_p50"], "p99_batch_frame_ms": st["batch_ms_p99"],
        "first_half": half(0.0, window / 2), "second_half": half(window / 2, window),
        "requests": st["submitted"], "completed": st["completed"], "rejected": st["rejected"],
        "scene_frames": st["scene_frames"], "batched_frames": st["batch_frames"],
        "mean_live_scenes": st["mean_scenes"], "peak_live_scenes": st["peak_scenes"],
        "peak_bytes": st["peak_bytes"], "wall_s": st["wall_s"], "device_busy_s": st["device_s"],
    }


def run_served(args, batched: dict | None) -> dict:
    """The served stream, twice. Requests: Poisson arrivals; each a scene of
    1k-262k particles (log-uniform, body fraction 0-30 %) asking for 1-60
    frames; admitted by a 150 GB HBM budget, resident between frames, stepped
    in continuous batches.
    1. The configured rate, 200 requests/s, for --served-window seconds: it
       offers more work than one GPU serves, so its throughput is the
       server's capacity and its queue (and latency) grows over the window.
    2. A sustainable rate, SERVED_LOAD of that capacity (requests/s from the
       mean work of a request), over the same window: latencies there are
       stationary, which the two halves of the window show."""
    from fluidphysics_b200 import server as SV
    bt, cps = (256, 8)
    if batched:
        bt, cps = batched["tuning"]["block_threads"], batched["tuning"]["ctas_per_sm"]
    W = args.served_window
    reqs = SV.served_requests(window_s=W, rate=200.0, seed=5)
    st, res = _serve(reqs, bt, cps)
    over = _served_block(st, res, reqs, W, 200.0)
    log(f"served at 200/s: {over['value']:.3e} of {over['offered_particle_substeps_per_s']:.3e} offered, "
        f"p99 {over['p99_frame_ms']:.1f} ms")
    work = np.mean([r.scene.total * r.frames * 5 for r in reqs])
    rate = SERVED_LOAD * over["value"] / work
    reqs2 = SV.served_requests(window_s=W, rate=rate, seed=6)
    st2, res2 = _serve(reqs2, bt, cps)
    sus = _served_block(st2, res2, reqs2, W, rate)
    log(f"served at {rate:.1f}/s: {sus['value']:.3e}, p50 {sus['p50_frame_ms']:.1f} p99 {sus['p99_frame_ms']:.1f} ms")
    out = dict(over)
    out["sustainable"] = sus
    out["workload"] = (f"Poisson arrivals over {W} s: 200/s (seed 5), then {rate:.1f}/s = {SERVED_LOAD:.0%} of the "
                       "measured capacity (seed 6); total particles log-uniform [1k, 262k], body fraction "
                       "U(0, 0.3), frames U{1..60}; HBM budget 150 GB")
    out["latency"] = ("frame latency = completion of the frame minus the time it could first run (arrival for a "
                      "request's first frame, so queueing is included), server wall clock; halves: request "
                      "latency (arrival to last frame) per frame asked, by arrival in the window's first or "
                      "second half")
    return out


def batched_capture(scenes: int, frames: int) -> None:
    """Builds the uneven batch of `scenes` scenes (the batched line's scenes,
    the compact hash-table rule, 256-thread blocks, 16 CTAs per SM), steps it
    `frames` frames, then runs one more frame between cudaProfilerStart and
    cudaProfilerStop: the window of the batched kernel captures."""
    import torch
    from fluidphysics_b200 import batch as B

    scs = B.batch_scenes(scenes, table="compact")
    with B.Batch(max_scenes=max(256, scenes), ctas_per_sm=16) as b:
        for sc in scs:
            b.add_scene(sc)
        for _ in range(frames):
            b.step(1 / 60, 5)
        b.sync()
        torch.cuda.synchronize()
        torch.cuda.cudart().cudaProfilerStart()
        b.step(1 / 60, 5)
        b.sync()
        torch.cuda.synchronize()
        torch.cuda.cudart().cudaProfilerStop()
        print(json.dumps({"batched_capture_scenes": scenes, "bytes": int(b.info().bytes_in_use)}))


def settled_capture(frames: int) -> None:
    """Steps the default scene `frames` frames, then runs 3 more between
    cudaProfilerStart and cudaProfilerStop: the settled-state window that the
    launch lists and kernel captures under profiles/ are taken on."""
    import torch
    from fluidphysics_b200 import scenes as S
    from fluidphysics_b200.sim import sim_from_scene

    sc = S.gpu_default(frames=frames + 3)
    sim = sim_from_scene(sc)
    for k in range(frames):
        if k == sc.slice_frame:
            sim.slice(*sc.wedge)
        sim.step(sc.dt, sc.substeps)
    sim.sync()
    torch.cuda.synchronize()
    torch.cuda.cudart().cudaProfilerStart()
    for _ in range(3):
        sim.step(sc.dt, sc.substeps)
    sim.sync()
    torch.cuda.synchronize()
    torch.cuda.cudart().cudaProfilerStop()
    sim.close()
    print(json.dumps({"settled_capture_frames": frames, "captured_frames": 3}))


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=300)
    ap.add_argument("--settle", type=int, default=300,
                    help="untimed frames from the initial state (slice at frame 60) before the timed "
                         "window: the timed frames are the settled pool, frames settle..settle+steps")
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="upbd", choices=["upbd", "reference"])
    ap.add_argument("--e2e-steps", type=int, default=200)
    ap.add_argument("--profile-frames", type=int, default=20)
    ap.add_argument("--profile-after", type=int, default=10,
                    help="frames stepped from the settled state before the per-kernel profile")
    ap.add_argument("--cpu-seconds", type=float, default=12.0)
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--batched-frames", type=int, default=300,
                    help="timed frames of the 256-scene batch (0 skips the batched line)")
    ap.add_argument("--batched-scenes", type=int, default=256)
    ap.add_argument("--served-window", type=float, default=10.0,
                    help="seconds of Poisson arrivals in each served stream (0 skips the served line)")
    ap.add_argument("--large-frames", type=int, default=120,
                    help="timed frames of the large scene (0 skips the large line)")
    ap.add_argument("--settled-capture", type=int, default=0,
                    help="profiling mode: step the default scene this many frames on its graph (slice "
                         "at frame 60), bracket the next 3 frames with cudaProfilerStart/Stop for "
                         "ncu --profile-from-start off, and exit (no bench line)")
    ap.add_argument("--batched-capture", type=int, default=0,
                    help="profiling mode: build a batch of this many of the batched line's scenes, step "
                         "it 10 frames, bracket the next frame with cudaProfilerStart/Stop, and exit")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)
    if args.batched_capture > 0:
        batched_capture(args.batched_capture, 10)
        return

    if args.impl == "reference":
        run_reference(args)
        return
    if args.settled_capture > 0:
        settled_capture(args.settled_capture)
        return

    import torch
    ws, rank, local = dist_env()
    torch.cuda.set_device(local)
    pg = None
    if ws > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                device_id=torch.device("cuda", local))
        pg = dist

    from fluidphysics_b200 import _lib as L
    from fluidphysics_b200 import scenes as S
    from fluidphysics_b200.sim import sim_from_scene

    sc = S.gpu_default(frames=args.steps)
    sc.desc.device = local
    sim = sim_from_scene(sc)
    stream = torch.cuda.Stream()
    sim.set_stream(stream.cuda_stream)
    init = sim.read_state()
    init_cons = sim.read_constraints()
    info = sim.info
    T = info.table_size

    # L2 flush buffer: twice the 126 MB L2
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device="cuda")

    def do_flush():
        with torch.cuda.stream(stream):
            flush.zero_()

    def reset():
        sim.write_state(**init)
        sim.write_constraints(init_cons)

    # settle: the block falls, splashes and comes to rest as a pool with the
    # body in it (the slice wedge at frame 60); the timed window starts from
    # that state
    for f in range(args.settle):
        if f == sc.slice_frame:
            sim.slice(*sc.wedge)
        sim.step(sc.dt, sc.substeps)
    sim.sync()
    if args.settle <= sc.slice_frame:
        log(f"settle={args.settle} ends before the slice frame {sc.slice_frame}: the timed window has no slice")
    init = sim.read_state()
    init_cons = sim.read_constraints()

    # warm-up (graphs captured here), then back to the settled state
    for _ in range(args.warmup):
        sim.step(sc.dt, sc.substeps)
    sim.sync()
    reset()

    # ---- timed region: K frames, device time per frame, L2 flushed between
    K = args.steps
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(K)]
    cvd = [x for x in os.environ.get("CUDA_VISIBLE_DEVICES", "").split(",") if x.strip()]
    phys = int(cvd[local]) if local < len(cvd) and cvd[local].strip().isdigit() else local
    clocks = Clocks(phys)
    launches0 = sim.launches
    if pg:
        pg.barrier()
    torch.cuda.synchronize()
    clocks.start()
    for k in range(K):
        do_flush()
        ev[k][0].record(stream)
        if args.settle + k == sc.slice_frame:
            sim.slice(*sc.wedge)
        sim.step(sc.dt, sc.substeps)
        ev[k][1].record(stream)
    torch.cuda.synchronize()
    if pg:
        pg.barrier()
    clk = clocks.stop()
    launches = sim.launches - launches0
    ms = sum(a.elapsed_time(b) for a, b in ev)
    sim.sync()
    active = info.solid_n + sim.active_count()
    local_units = active * sc.substeps * K
    t_max, units = reduce_over_ranks(pg, ms, local_units, "cuda")
    value = units / (t_max / 1e3)

    # ---- e2e through the C ABI with pinned host buffers
    reset()
    E = min(args.e2e_steps, K)
    pos_h = torch.empty((info.total, 4), dtype=torch.float32, pin_memory=True)
    flags_h = torch.empty(info.total, dtype=torch.int32, pin_memory=True)
    import ctypes as C
    fp = C.cast(pos_h.data_ptr(), C.POINTER(C.c_float))
    up = C.cast(flags_h.data_ptr(), C.POINTER(C.c_uint32))
    for _ in range(3):  # warm the readback path
        sim.step(sc.dt, sc.substeps)
        L.check(sim.lib, sim.h, sim.lib.upbd_read_state_async(sim.h, fp, up))
    L.check(sim.lib, sim.h, sim.lib.upbd_read_wait(sim.h))
    reset()
    if pg:
        pg.barrier()
    torch.cuda.synchronize()
    # L2 flushed before every frame as in the device-timed loop; the flushes'
    # own event-timed durations (on the same stream) are taken out of the total
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    fev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(E)]
    e0.record(stream)
    for k in range(E):
        fev[k][0].record(stream)
        do_flush()
        fev[k][1].record(stream)
        if args.settle + k == sc.slice_frame:
            sim.slice(*sc.wedge)
        sim.step(sc.dt, sc.substeps)
        # GpuSim._readBuffer: device staging copy, then an asynchronous copy
        # to pinned host memory that overlaps the next frame
        L.check(sim.lib, sim.h, sim.lib.upbd_read_state_async(sim.h, fp, up))
    L.check(sim.lib, sim.h, sim.lib.upbd_read_wait(sim.h))  # every frame's result is on the host
    e1.record(stream)
    torch.cuda.synchronize()
    flush_ms = sum(a.elapsed_time(b) for a, b in fev)
    e2e_ms = e0.elapsed_time(e1) - flush_ms
    if pg:
        t = torch.tensor([e2e_ms], device="cuda", dtype=torch.float64)
        pg.all_reduce(t, op=pg.ReduceOp.MAX)
        e2e_ms = float(t.item())
    e2e_units = active * sc.substeps * E * ws
    e2e_value = e2e_units / (e2e_ms / 1e3)

    # ---- per-kernel device times of eager frames (dominant kernel roofline)
    reset()
    for _ in range(args.profile_after):  # into an interacting state
        sim.step(sc.dt, sc.substeps)
    sim.sync()
    P = args.profile_frames
    tot = np.zeros(L.KERNEL_KINDS)
    cnt = np.zeros(L.KERNEL_KINDS)
    msb = (C.c_double * L.KERNEL_KINDS)()
    lnb = (C.c_uint32 * L.KERNEL_KINDS)()
    for _ in range(P):
        do_flush()
        torch.cuda.synchronize()
        L.check(sim.lib, sim.h, sim.lib.upbd_profile_frame(sim.h, sc.dt, sc.substeps, msb, lnb))
        tot += np.array(msb[:])
        cnt += np.array(lnb[:])
    names = [(sim.lib.upbd_kernel_name(k) or b"").decode() for k in range(L.KERNEL_KINDS)]
    st = sim.read_state()
    n_act = int((st["flags"] & 1).sum())
    n_fl = int((st["flags"][info.solid_n:] & 1).sum())
    units_k = {"A": n_act, "F": n_fl, "S": info.solid_n, "C": info.num_cons, "T": T}
    per_kernel = {}
    for k, nm in enumerate(names):
        if cnt[k] > 0 and nm:
            avg_ms = tot[k] / cnt[k]
            b = KERNEL_BYTES[nm](units_k) if nm in KERNEL_BYTES else None
            per_kernel[nm] = {"share": tot[k] / tot.sum(), "avg_us": avg_ms * 1e3,
                              "launches_per_frame": cnt[k] / P,
                              "gbs": (b / (avg_ms / 1e3) / 1e9) if b else None}
    dom = dominant_kernel(per_kernel)
    peaks, peak_src = measured_peaks()
    hbm = float(peaks.get("hbm_gbs", 6650.0))
    dk = per_kernel[dom]
    achieved = dk["gbs"]
    roofline = {"bound": "hbm", "kernel": dom, "achieved": achieved, "peak": hbm, "unit": "GB/s",
                "frac": achieved / hbm, "peak_source": f"{peak_src} (MEASURED_PEAKS.json hbm_gbs)"
                if peak_src == "measured" else "fallback 6.65 TB/s",
                "bytes_per_launch": KERNEL_BYTES[dom](units_k), "avg_launch_us": dk["avg_us"],
                "traffic": ncu_traffic(dom, "gpu_default"),
                "kernels": {k: {kk: (round(vv, 4) if isinstance(vv, float) else vv) for kk, vv in v.items()}
                            for k, v in sorted(per_kernel.items(), key=lambda x: -x[1]["share"])}}
    # the bound the gathers actually meet on L2-resident data: instruction
    # issue (one warp instruction per scheduler per cycle, 4 schedulers per SM)
    wi = ncu_instructions(dom, "gpu_default")
    if wi:
        sm_count = torch.cuda.get_device_properties(local).multi_processor_count
        roofline["issue"] = {"warp_inst_per_launch": wi, "avg_launch_us": dk["avg_us"],
                             "achieved": wi / (dk["avg_us"] * 1e-6) / 1e9, "unit": "G warp-instructions/s",
                             "sms": sm_count, "source": "profiles/instructions.txt (ncu smsp__inst_executed.sum)"}
        mhz = clk.get("sm_mhz") or clk.get("sm_max_mhz")
        if mhz:  # the SM clock sampled under load in the timed region
            peak_i = sm_count * 4 * float(mhz) * 1e6 / 1e9
            roofline["issue"].update(peak=peak_i, frac=roofline["issue"]["achieved"] / peak_i, sm_mhz=mhz)
    # whole-step roofline: the substep's algorithmic bytes at the measured rate
    B_sub = (240 * n_act + 200 * n_fl + 8 * T + sc.desc.solid_iters * (84 * info.solid_n + 24 * info.num_cons)
             + 20 * info.num_cons)
    step_gbs = B_sub * sc.substeps * K / (ms / 1e3) / 1e9
    roofline["step_achieved_gbs"] = step_gbs
    roofline["step_frac"] = step_gbs / hbm
    # launch floor: the same frame graph with every kernel emptied (same nodes,
    # grids, dependencies and side-stream branches), replayed back to back
    floor_ms, floor_nodes = sim.graph_floor(sc.dt, sc.substeps, 200)
    launch_floor = {"empty_graph_ms": floor_ms, "kernel_nodes": floor_nodes,
                    "share_of_frame": floor_ms / (t_max / K),
                    "how": "the captured frame graph with each kernel node's kernel replaced by an empty one "
                           "of the same grid and block, 200 replays timed by CUDA events"}

    sim.close()
    large = run_large(args, stream) if args.large_frames > 0 else None
    batched = run_batched(args, stream, hbm) if args.batched_frames > 0 else None
    served = run_served(args, batched) if args.served_window > 0 else None
    if pg:
        for key, obj in (("large", large), ("batched", batched), ("served", served)):
            if obj and obj.get("value"):
                t = torch.tensor([obj["value"]], device="cuda", dtype=torch.float64)
                pg.all_reduce(t, op=pg.ReduceOp.SUM)  # replicas: whole-job rate
                obj["value"] = float(t.item())

    cpu = None
    if rank == 0 and ws == 1 and not args.no_cpu:
        try:
            cpu = cpu_baseline(args.cpu_seconds)
        except Exception as e:  # the checker leg must not hide the GPU line
            cpu = {"value": None, "unit": UNIT, "cores": 1, "kind": "port", "sample": f"failed: {e}"}

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": K,
            "warmup": args.warmup, "ms_per_step": t_max / K, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic (seeded jittered fluid block, lattice body; no dataset in the reference)",
            "config": {"workload": "gpu_default: 20^3 body (8,000 particles, 93,556 constraints) + 65,536 "
                                   "fluid, 30 mm radius, T=2^18, 5 substeps x 3 Jacobi iterations per "
                                   f"frame (dt=1/60), slice wedge at frame 60; timed frames {args.settle}.."
                                   f"{args.settle + K - 1} (the settled pool)",
                       "frames": K, "first_frame": args.settle, "particles": active, "substeps": sc.substeps,
                       "solid_iters": sc.desc.solid_iters, "l2": "flushed between frames (256 MB write)",
                       "parallelism": f"replicas x{ws}", "graphs": True},
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": int(info.param_bytes),
                    "d2h_bytes_per_step": int(info.total * 16 + info.total * 4), "frames": E,
                    "l2": "flushed before every frame; the flushes' event-timed durations are not counted",
                    "path": "upbd_step + upbd_read_state_async(pos, flags) into pinned host memory every "
                            "frame (device staging copy, host copy overlapping the next frame), "
                            "upbd_read_wait before the clock stops"},
            "roofline": roofline,
            "launch_floor": launch_floor,
            "cpu_baseline": cpu,
            "gpu_launches": int(launches),
            "clocks": clk,
            "large": large,
            "batched": batched,
            "served": served,
        }
        print(json.dumps(line), flush=True)
    if pg:
        pg.barrier()
        pg.destroy_process_group()


if __name__ == "__main__":
    main()
