#!/usr/bin/env python
"""Particle-steps/s of the GPAT mover on one GB300.

Workload: 2D turbulent shock, 2048 x 2048 grid over [0,1]^2 (tanh shock at
x = 0.5, r = 3.5, w = 0.001; B = x + random-phase Kolmogorov dB/B0 = 0.5 from
Az), kappa_par = 0.01 (p/p0)^(4/3) along the local B, kperp/kpar = 0.05,
1e7 particles injected on the shock at p0, dt_min = dtf / 1000 so each
particle takes 1000 pushes per MHD interval.  One bench step is one pass of
the driver's per-frame hot path: particle_mover over one interval
(interpolation + kappa + push + boundaries + landing, then removal),
split_particle and the global f(p).

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

--impl reference times the CPU restatement of the reference's FP64 mover
(oracle/, OpenMP over all host cores) on a bounded sample of the same
workload.  Under torchrun each rank runs an independent replica (different
seed); the engine itself is single-GPU.
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

REPO = Path(__file__).resolve().parent
for p in (str(REPO / "stochastic-parker_gb300"), str(REPO / "oracle")):
    if p not in sys.path:
        sys.path.insert(0, p)

METRIC = "particle-steps/s on 1 GB300 (mixed/learned vs plain FP64) at f(p) tail err ≤2%"
UNIT = "particle-steps/s"
# Algorithmic bytes of one 2D push: 4 cell corners x 15 FP32 field values
# gathered; per particle and launch the FP64 state is read and written once.
# 3D: 8 corners x 21 values.
# Algorithmic bytes of the push: corners x stored FP32 field arrays x 4 B
# (2D: 4 x 7, 3D: 8 x 8) per push, and the FP64 particle state touched once
# per particle and launch (6 x 8 B read, 5 x 8 B written, the flag).
GATHER_BYTES_PER_STEP = {2: 4 * 7 * 4, 3: 8 * 8 * 4}
STATE_BYTES_PER_PARTICLE = 6 * 8 + 5 * 8 + 2
# What the packed records make the split-precision mover gather per push
# (4 x 15 and 8 x 21 FP32 values, precomputed gradients included).
IMPL_GATHER_BYTES_PER_STEP = {2: 4 * 15 * 4, 3: 8 * 21 * 4}
WORKLOADS = ("turbulent_shock_2d", "turbulence_3d", "batched_shock_2d", "learned_3d")


# The run of the batched workload the CPU baselines sample (its first run).
BATCH_SAMPLE_RUN = 0


def make_workload(args, precision, seed=None, nframes=16, scale=None):
    from gpat import configs
    scale = args.scale if scale is None else scale
    if args.workload == "batched_shock_2d":
        return configs.batched_shock_2d(scale=scale, precision=precision, nframes=nframes,
                                        only=BATCH_SAMPLE_RUN)[0]
    if args.workload in ("turbulence_3d", "learned_3d"):
        grid = args.grid if args.grid != 2048 else 256
        return configs.turbulence_3d(scale=scale, n=grid, precision=precision,
                                     seed=3 if seed is None else seed, nframes=nframes)
    return configs.turbulent_shock_2d(scale=scale, n=args.grid, precision=precision,
                                      seed=2 if seed is None else seed, nframes=nframes)


def parse_args(argv=None):
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=("ours", "reference"), default="ours")
    ap.add_argument("--precision", choices=("mixed", "fp64"), default="mixed")
    ap.add_argument("--scale", type=float, default=1.0, help="particle-count multiplier")
    ap.add_argument("--grid", type=int, default=2048,
                    help="cells per side (the 3D workload uses 256 unless set)")
    ap.add_argument("--workload", choices=WORKLOADS, default="turbulent_shock_2d")
    ap.add_argument("--e2e-steps", type=int, default=2)
    ap.add_argument("--cpu-seconds", type=float, default=12.0)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--bin-interval", type=int, default=0,
                    help="pushes between re-binnings (0: engine default, <0: once per call)")
    ap.add_argument("--no-accuracy", action="store_true",
                    help="skip the FP64 sample and the f(p) tail-error check")
    ap.add_argument("--intervals", type=int, default=0,
                    help="learned_3d: MHD intervals of every arm (0: the first interval count "
                         "at which a pilot plain run has 0.1 %% of its particles above 100 p0)")
    ap.add_argument("--train-trajectories", type=float, default=1e7,
                    help="learned_3d: plain trajectories generating the training records")
    ap.add_argument("--record-every", type=int, default=0,
                    help="learned_3d: intervals between training records of a trajectory "
                         "(0: ten records over the run)")
    ap.add_argument("--fp64-particles", type=float, default=2e5,
                    help="learned_3d: particles of the FP64 reference arms")
    ap.add_argument("--no-extras", action="store_true",
                    help="headline workload only (no 3D and batched keys in its line)")
    ap.add_argument("--tiles-3d", default="off",
                    help="--tiles for the 3D measurement inside the headline line")
    ap.add_argument("--tiles", default="off",
                    help="split-precision mover field bricks: 'off' (global gathers) or "
                         "'bx,by,bz[,hx,hy,hz[,threads[,items]]]': cells per brick and halo "
                         "cells per side staged in shared memory")
    return ap.parse_args(argv)


def parse_tiles(spec: str):
    """(bx, by, bz, hx, hy, hz, threads, items) of --tiles, or None for 'off'."""
    if spec in ("off", "0", ""):
        return None
    v = [int(x) for x in spec.split(",")]
    if len(v) == 2:
        v.append(1)
    return tuple((v + [0] * 8)[:8])


def l2_read_gbs(torch, dev) -> float:
    """Read bandwidth of a 64 MiB L2-resident buffer (torch.sum), an estimate
    of the cache bound the mover's gathers run against."""
    x = torch.ones(16 * 1024 * 1024, dtype=torch.float32, device=dev)
    for _ in range(5):
        x.sum()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record()
    for _ in range(50):
        x.sum()
    e1.record()
    torch.cuda.synchronize()
    return x.numel() * 4 * 50 / (e0.elapsed_time(e1) / 1e3) / 1e9


def fp64_sample(args, seed, device, nptl):
    """Plain FP64 GPU mover on a sample of the same workload: one interval."""
    from gpat import configs
    w = make_workload(args, 0, seed=seed, nframes=2)
    eng = configs.build_engine(w, device=device, nptl_max=nptl)
    configs.inject(eng, w, nptl=nptl)
    eng.particle_mover(nsteps_interval=10, mhd_tframe=1, num_fine_steps=1)
    c = eng.counters()
    eng.close()
    return c.last_mover_steps / (c.last_mover_ms / 1e3), c.last_mover_steps


# ---------------------------------------------------------------------------
class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.path = None

    def start(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.QUERY}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except (FileNotFoundError, OSError):
            self.proc = None

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, smax, reasons, power = [], [], set(), []
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        for line in Path(self.path).read_text().splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                smax.append(float(f[2]))
                power.append(float(f[3]))
            except ValueError:
                continue
            for name, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(name)
        os.unlink(self.path)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "power_w_max": max(power) if power else None,
                "samples": len(sm), "reasons": sorted(reasons)}


def dist_setup():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist
        # NCCL between GPU ranks; GPAT_DIST_BACKEND=gloo runs the same
        # rank logic on CPU processes
        backend = os.environ.get("GPAT_DIST_BACKEND", "nccl")
        dist.init_process_group(backend=backend)
    return world, rank, local


def barrier(world):
    if world > 1:
        import torch.distributed as dist
        dist.barrier()


def max_over_ranks(world, x: float, device) -> float:
    if world == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def sum_over_ranks(world, x: float, device) -> float:
    if world == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.SUM)
    return float(t.item())


def measured_peaks() -> dict:
    p = REPO / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return {"hbm_gbs": d.get("hbm_gbs"), "source": "measured"}
    return {"hbm_gbs": 6800.0, "source": "fallback"}


# Of one whole interval of a workload at its full particle count, per counted push
# (profiles/mover_traffic.md, with the commands): DRAM bytes read and written, and
# wavefronts of up to 128 bytes of the L1TEX data pipe, of which an SM does one per
# clock and which bounds the gather movers.  Both depend on how many particles share
# a cell, so the DRAM figure is given out for that workload and count alone.
NCU_MOVER = {
    2: {"workload": "turbulent_shock_2d_2048x2048", "particles": 10_000_000,
        "dram_bytes_per_push": 0.933, "wavefronts_per_push": 4.18,
        "profile": "profiles/mover_traffic.md"},
    3: {"workload": "turbulence_3d_256^3", "particles": 100_000_000,
        "dram_bytes_per_push": 14.0, "wavefronts_per_push": 15.3,
        "profile": "profiles/mover_traffic.md"},
}
# Bytes per push on that pipe.  Global-gather movers: the wavefronts above; brick
# movers read 16-byte chunks from shared memory (nominal; bank conflicts cost more).
L1_MODEL = {("global", 2): {"bytes_per_push": NCU_MOVER[2]["wavefronts_per_push"] * 128,
                            "bytes_per_clk_sm": 128},
            ("global", 3): {"bytes_per_push": NCU_MOVER[3]["wavefronts_per_push"] * 128,
                            "bytes_per_clk_sm": 128},
            ("tile", 2): {"bytes_per_push": 4 * 64, "bytes_per_clk_sm": 128},
            ("tile", 3): {"bytes_per_push": 8 * (5 * 16 + 4), "bytes_per_clk_sm": 128}}


def roofline_of(kind, ndim, avg_ms, avg_steps, avg_n, sm_count, sm_mhz, peaks, workload=None,
                particles=None) -> dict:
    """Roofline of one mover launch: the L1TEX data path is the bound (ncu),
    HBM is reported beside it on the algorithmic bytes."""
    secs = avg_ms / 1e3
    m = L1_MODEL[(kind, ndim)]
    l1_bytes = avg_steps * m["bytes_per_push"]
    l1_peak = sm_count * m["bytes_per_clk_sm"] * (sm_mhz or 2070.0) * 1e6 / 1e9
    alg = avg_steps * GATHER_BYTES_PER_STEP[ndim] + avg_n * STATE_BYTES_PER_PARTICLE
    ncu = NCU_MOVER[ndim] if kind == "global" else {}
    same = ncu and (workload, particles) == (ncu["workload"], ncu["particles"])
    dram = ncu["dram_bytes_per_push"] if same else None
    what = "L1TEX data pipe" if kind == "global" else "nominal shared-memory rate"
    peak_source = (f"{what}: one wavefront of 128 bytes per clock per SM x {sm_count} SMs x "
                   f"median sampled SM clock {sm_mhz} MHz")
    return {"bound": "l1", "achieved": l1_bytes / secs / 1e9, "peak": l1_peak, "unit": "GB/s",
            "frac": l1_bytes / secs / 1e9 / l1_peak, "peak_source": peak_source,
            "traffic": dram * avg_steps if dram is not None else None,
            "traffic_source": ncu["profile"] if same else None,
            "l1_bytes_per_push": m["bytes_per_push"],
            "l1_measured_at": f"{ncu['workload']}, {ncu['particles']} particles" if ncu else "nominal",
            "kernel_ms_per_launch": avg_ms, "steps_per_launch": avg_steps,
            "kernel_steps_per_s": avg_steps / secs,
            "hbm": {"achieved": alg / secs / 1e9, "peak": peaks["hbm_gbs"],
                    "frac": alg / secs / 1e9 / peaks["hbm_gbs"], "peak_source": peaks["source"],
                    "algorithmic_bytes_per_push": GATHER_BYTES_PER_STEP[ndim],
                    "state_bytes_per_particle": STATE_BYTES_PER_PARTICLE},
            "note": "achieved = L1 data-pipe wavefronts (128 B) per push x pushes / launch "
                    "time, against one per clock and SM, counted where l1_measured_at says; "
                    "hbm = algorithmic bytes (corners x stored field "
                    "arrays x 4 B + FP64 state) over measured HBM"}


# ---------------------------------------------------------------------------
def cpu_sample(w, seconds: float, threads: int | None = None):
    """Oracle (FP64, OpenMP) particle-steps/s on a sample of the workload:
    particles injected on the shock, one MHD interval each."""
    import oracle
    from gpat.engine import make_params
    prm = oracle.params_from(make_params(**w.params))
    cfg = oracle.config_from(w.mhd_config)
    full = oracle.full_fields(w.frame, prm.ndim, w.mhd_config)
    dtf = float(w.tstamps[1] - w.tstamps[0])
    nthreads = threads or os.cpu_count() or 1

    def run(n):
        parts = oracle.Particles(n)
        cnt = oracle.OrcCounters()
        if w.inject["kind"] == "at_x":
            oracle.inject_at_x(prm, cfg, parts, n, w.inject["xpos"], 1e-7, 1, 1.0, 0.0, cnt)
        else:
            c = w.mhd_config
            box = (c.xmin, c.ymin, c.zmin, c.xmin + c.nx * c.dx, c.ymin + c.ny * c.dy,
                   c.zmin + c.nz * c.dz)
            oracle.inject_spatial_uniform(prm, parts, n, 1e-7, w.inject["dist_flag"], 1.0, 0.0,
                                          0.0, box, cnt, power_index=w.inject["power_index"])
        t0 = time.perf_counter()
        oracle.mover(prm, cfg, full, parts, 0.0, dtf, nthreads=nthreads, counters=cnt)
        return cnt.steps, time.perf_counter() - t0

    n = 256 * nthreads
    steps, dt = run(n)
    rate = steps / max(dt, 1e-9)
    n2 = max(n, int(n * seconds / max(dt, 1e-6) * 0.9))
    n2 = min(n2, 4_000_000)
    steps, dt = run(n2)
    return steps / dt, nthreads, n2, steps, dt, rate


def run_reference(args, world, rank):
    from gpat import configs
    if rank != 0:
        return
    w = make_workload(args, 1, nframes=4)
    vals = []
    # the oracle restates the reference's FP64 mover
    per_step = max(2.0, args.cpu_seconds / max(1, args.steps))
    for k in range(args.warmup + args.steps):
        v, cores, n, steps, dt, _ = cpu_sample(w, per_step)
        if k >= args.warmup:
            vals.append((v, n, steps, dt))
    value = statistics.median(v for v, *_ in vals)
    n, steps, dt = vals[-1][1:]
    sample = (f"{n} particles of the {w.name} workload injected on the shock, one MHD "
              f"interval ({steps / n:.0f} pushes each, {steps} particle-steps in {dt:.2f} s) "
              f"per step")
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1e3 * vals[-1][3], "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "impl": "reference",
            "config": {"workload": w.name, "particles_per_rank": w.nptl,
                       "precision": "fp64"},
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": "port",
                             "sample": sample},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def run_ours(args, world, rank, local):
    import numpy as np
    import torch
    from gpat import configs
    from gpat.engine import ParticleSet

    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    prec = 1 if args.precision == "mixed" else 0
    total_frames = args.warmup + args.steps + args.e2e_steps + 2
    w = make_workload(args, prec, seed=(3 if args.workload == "turbulence_3d" else 2) + rank,
                      nframes=total_frames)
    eng = configs.build_engine(w, device=local, nptl_max=int(w.nptl * 1.6),
                               bin_interval=args.bin_interval)
    tiles = parse_tiles(args.tiles) if prec == 1 else None
    if tiles:
        eng.set_mover_tiles(*tiles)
    configs.inject(eng, w)
    stream = torch.cuda.ExternalStream(eng.stream, device=dev)
    frame = [1]
    kernel_ms, kernel_steps, kernel_n, kernel_launches = [], [], [], []

    def step():
        n_before = eng.nptl_current
        eng.particle_mover(nsteps_interval=10, mhd_tframe=frame[0], num_fine_steps=1)
        c = eng.counters()
        kernel_ms.append(c.last_mover_ms)
        kernel_steps.append(c.last_mover_steps)
        kernel_n.append(n_before)
        kernel_launches.append(c.last_mover_launches)
        if w.split:
            eng.split_particle(w.split["ratio"], w.split["pmin"], 10)
        eng.calc_particle_distributions()
        frame[0] += 1

    for _ in range(args.warmup):
        step()
    kernel_ms.clear(); kernel_steps.clear(); kernel_n.clear(); kernel_launches.clear()

    clocks = ClockSampler(local)
    steps0 = eng.counters().steps
    barrier(world)
    torch.cuda.synchronize()
    clocks.start()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ev0.record(stream)
    for _ in range(args.steps):
        step()
    ev1.record(stream)
    torch.cuda.synchronize()
    clk = clocks.stop()
    barrier(world)
    elapsed = ev0.elapsed_time(ev1) / 1e3
    psteps = eng.counters().steps - steps0
    t_max = max_over_ranks(world, elapsed, dev)
    total_steps = sum_over_ranks(world, float(psteps), dev)
    value = total_steps / t_max

    # End to end through the public API with host buffers: the particle set
    # goes host -> device, the frame's hot path runs, f(p) and the particle
    # set come back.
    n_cap = int(w.nptl * 1.6)
    pinned = {}
    from gpat import _abi
    for name, t in (_abi.PARTICLE_FIELDS if args.e2e_steps > 0 else []):
        tt = torch.empty(n_cap, dtype=getattr(torch, {"f8": "float64", "i1": "int8", "i4": "int32",
                                                        "u4": "uint32"}[t]), pin_memory=True)
        pinned[name] = tt.numpy()
    host = ParticleSet(pinned) if pinned else None
    cur = eng.get_particles(out=host) if host is not None else None
    e2e_steps, e2e_h2d, e2e_d2h = 0, 0, 0
    bytes_per_ptl = sum(np.dtype(t).itemsize for _, t in _abi.PARTICLE_FIELDS)
    barrier(world)
    torch.cuda.synchronize()
    t_start = time.perf_counter()
    for _ in range(args.e2e_steps):
        s0 = eng.counters().steps
        eng.put_particles(cur)
        e2e_h2d += len(cur) * bytes_per_ptl
        eng.particle_mover(nsteps_interval=10, mhd_tframe=frame[0], num_fine_steps=1)
        if w.split:
            eng.split_particle(w.split["ratio"], w.split["pmin"], 10)
        f, counts = eng.calc_particle_distributions()
        cur = eng.get_particles(out=host)
        e2e_d2h += len(cur) * bytes_per_ptl + f.nbytes + counts.nbytes
        e2e_steps += eng.counters().steps - s0
        frame[0] += 1
    torch.cuda.synchronize()
    e2e_elapsed = max_over_ranks(world, time.perf_counter() - t_start, dev)
    e2e_total = sum_over_ranks(world, float(e2e_steps), dev)
    e2e_value = e2e_total / e2e_elapsed if e2e_elapsed > 0 else None

    if rank != 0:
        eng.close()
        return None
    peaks = measured_peaks()
    launches = statistics.mean(kernel_launches)
    avg_ms = statistics.mean(kernel_ms) / launches          # per mover launch
    avg_steps = statistics.mean(kernel_steps) / launches
    avg_n = statistics.mean(kernel_n)
    ndim = 3 if args.workload == "turbulence_3d" else 2
    ncells = (w.mhd_config.nx + 4) * (w.mhd_config.ny + 4) * ((w.mhd_config.nz + 4) if ndim == 3 else 1)
    rec_mb = ncells * (64 if ndim == 2 else 96) / 1e6
    state_mb = avg_n * 98 / 1e6
    kind = "tile" if tiles else "global"
    sm_count = torch.cuda.get_device_properties(dev).multi_processor_count
    roofline = roofline_of(kind, ndim, avg_ms, avg_steps, avg_n, sm_count, clk.get("sm_mhz"),
                           peaks, w.name if prec else None, w.nptl)
    roofline["kernel"] = (f"mover_tile_kernel<{ndim}> + mover_overflow_kernel<{ndim}>" if tiles
                          else f"mover_{args.precision}_kernel<{ndim}>")
    roofline["mover_launches_per_interval"] = launches
    if tiles:
        roofline["tiles"] = eng.mover_tiles()
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * elapsed / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32" if prec else "f64", "data": "synthetic",
            "config": {"workload": w.name, "particles_per_rank": w.nptl,
                       "pushes_per_particle_per_interval":
                           round(statistics.mean(kernel_steps) / max(1.0, avg_n), 1),
                       "precision": args.precision + (" (FP32 fields, kappa, drift and dt; "
                                                      "Kahan-compensated FP32 momentum and clock; "
                                                      "integer cell + FP32 offset positions)"
                                                      if prec else ""),
                       "step": "particle_mover" + (" + split_particle" if w.split else "") +
                               " + f(p) over one MHD interval",
                       "l2": f"inputs exceed L2 (packed field records {rec_mb:.0f} MB, "
                             f"particle state {state_mb:.0f} MB)",
                       "parallelism": f"replicas x{world}"},
            "clocks": clk,
            # per step: mover launches, a binning of 5 kernels (6 from 600 000 particles
            # on) after each, split (3), f(p) (1)
            "gpu_launches": int(round(sum((7 if w.nptl >= 600_000 else 6) * l + 4
                                          for l in kernel_launches))) if prec
            else 8 * args.steps,
            "e2e": {"value": e2e_value, "unit": UNIT,
                    "h2d_bytes_per_step": e2e_h2d // max(1, args.e2e_steps),
                    "d2h_bytes_per_step": e2e_d2h // max(1, args.e2e_steps)},
            "roofline": roofline}
    eng.close()
    if not args.no_accuracy and prec == 1:
        from gpat import accuracy
        n64 = max(1000, int(1e6 * args.scale))
        v64, s64 = fp64_sample(args, (3 if args.workload == "turbulence_3d" else 2) + rank, local,
                               n64)
        line["fp64_gpu"] = {"value": v64, "unit": UNIT, "sample": f"{n64} particles, one interval, "
                                                                  f"{s64} particle-steps",
                            "mixed_over_fp64": value / v64}
        if args.workload == "turbulent_shock_2d":
            line["accuracy"] = accuracy.turbulent_shock_check(scale=0.1, intervals=25,
                                                              device=local, tiles=tiles)
        else:
            line["accuracy"] = accuracy.planar_shock_check(scale=1.0, device=local)
    if world == 1 and not args.no_cpu_baseline:
        v, cores, n, steps, dt, _ = cpu_sample(w, args.cpu_seconds)
        line["cpu_baseline"] = {"value": v, "unit": UNIT, "cores": cores, "kind": "port",
                                "sample": f"{n} particles of {w.name} injected as the workload "
                                          f"does, one MHD interval of FP64 pushes ({steps} "
                                          f"particle-steps in {dt:.2f} s)"}
    return line


def run_batch(args, world, rank, local):
    """64 independent 2D turbulent-shock runs of uneven sizes and parameters
    moved by the batched mover: one persistent launch per chunk for all runs,
    replayed as a CUDA graph, launch shape from the autotuner."""
    import numpy as np
    import torch
    from gpat import _abi, accuracy, configs
    from gpat.engine import Batch, ParticleSet

    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    total_frames = args.warmup + args.steps + args.e2e_steps + 2
    runs = configs.batched_shock_2d(scale=args.scale, nframes=total_frames, seed=11 + rank)
    engines = [configs.build_engine(w, device=local, nptl_max=int(w.nptl * 1.6) + 16,
                                    bin_interval=args.bin_interval) for w in runs]
    for e, w in zip(engines, runs):
        configs.inject(e, w)
    batch = Batch(engines)
    tuning = batch.autotune(mhd_tframe=1)
    stream = torch.cuda.ExternalStream(engines[0].stream, device=dev)
    frame = [1]
    graph_ms, graph_launches, chunk_pushes = [], [], []

    def step():
        batch.particle_mover(mhd_tframe=frame[0])
        st = batch.stats()
        graph_ms.append(st["ms"])
        graph_launches.append(st["graph_launches"])
        chunk_pushes.append(st["pushes"])
        for e, w in zip(engines, runs):
            e.split_particle(w.split["ratio"], w.split["pmin"], 10)
            e.calc_particle_distributions()
        frame[0] += 1

    for _ in range(args.warmup):
        step()
    graph_ms.clear(); graph_launches.clear(); chunk_pushes.clear()
    steps0 = sum(e.counters().steps for e in engines)
    n_timed = sum(e.nptl_current for e in engines)
    clocks = ClockSampler(local)
    barrier(world)
    torch.cuda.synchronize()
    clocks.start()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ev0.record(stream)
    for _ in range(args.steps):
        step()
    ev1.record(stream)
    torch.cuda.synchronize()
    clk = clocks.stop()
    barrier(world)
    elapsed = ev0.elapsed_time(ev1) / 1e3
    psteps = sum(e.counters().steps for e in engines) - steps0
    t_max = max_over_ranks(world, elapsed, dev)
    value = sum_over_ranks(world, float(psteps), dev) / t_max
    intervals_done = frame[0] - 1

    # f(p) of every run's first injected particles against an FP64 run of the
    # same particles
    acc = []
    if not args.no_accuracy:
        acc = accuracy.batched_runs_check(runs, engines, intervals_done, sample=20000,
                                          device=local)

    # end to end: every run's particles host -> device, the batched frame,
    # f(p) and particles back
    bytes_per_ptl = sum(np.dtype(t).itemsize for _, t in _abi.PARTICLE_FIELDS)
    hosts = []
    for e in (engines if args.e2e_steps > 0 else []):
        cap = e.params.nptl_max
        arrs = {name: torch.empty(cap, dtype=getattr(torch, {"f8": "float64", "i1": "int8",
                                                             "i4": "int32", "u4": "uint32"}[t]),
                                  pin_memory=True).numpy()
                for name, t in _abi.PARTICLE_FIELDS}
        hosts.append(ParticleSet(arrs))
    curs = [e.get_particles(out=h) for e, h in zip(engines, hosts)]
    e2e_steps, e2e_h2d, e2e_d2h = 0, 0, 0
    barrier(world)
    torch.cuda.synchronize()
    t_start = time.perf_counter()
    for _ in range(args.e2e_steps):
        s0 = sum(e.counters().steps for e in engines)
        for e, c in zip(engines, curs):
            e.put_particles(c)
            e2e_h2d += len(c) * bytes_per_ptl
        batch.particle_mover(mhd_tframe=frame[0])
        for i, (e, w) in enumerate(zip(engines, runs)):
            e.split_particle(w.split["ratio"], w.split["pmin"], 10)
            f, counts = e.calc_particle_distributions()
            curs[i] = e.get_particles(out=hosts[i])
            e2e_d2h += len(curs[i]) * bytes_per_ptl + f.nbytes + counts.nbytes
        e2e_steps += sum(e.counters().steps for e in engines) - s0
        frame[0] += 1
    torch.cuda.synchronize()
    e2e_elapsed = max_over_ranks(world, time.perf_counter() - t_start, dev)
    e2e_value = sum_over_ranks(world, float(e2e_steps), dev) / e2e_elapsed if e2e_elapsed else None

    if rank != 0:
        batch.close()
        for e in engines:
            e.close()
        return None
    peaks = measured_peaks()
    chunks = statistics.mean(graph_launches)
    ms_chunk = statistics.mean(graph_ms) / chunks
    pushes_chunk = statistics.mean(chunk_pushes) / chunks
    sm_count = torch.cuda.get_device_properties(dev).multi_processor_count
    batch_roofline = roofline_of("global", 2, ms_chunk, pushes_chunk, n_timed, sm_count,
                                 clk.get("sm_mhz"), peaks)
    batch_roofline.update({"kernel": "mover_mixed_batch_kernel<2> chunk graph (mover + binning)",
                           "ms_per_chunk": ms_chunk, "pushes_per_chunk": pushes_chunk,
                           "chunks_per_interval": chunks,
                           "timing": "whole chunk graph (the binning kernels included)"})
    nruns = len(runs)
    sizes = sorted({w.mhd_config.nx for w in runs})
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * elapsed / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32", "data": "synthetic",
            "config": {"workload": f"batched_shock_2d_{nruns}_runs",
                       "runs": nruns,
                       "particles_total": int(sum(w.nptl for w in runs)),
                       "particles_per_run_min_max": [int(min(w.nptl for w in runs)),
                                                     int(max(w.nptl for w in runs))],
                       "grids": [f"{n}x{n}" for n in sizes],
                       "pushes_per_particle_per_interval": round(psteps / args.steps /
                                                                 max(1, n_timed), 1),
                       "step": "batched particle_mover (graph-replayed chunks) + per-run "
                               "split_particle + f(p) over one MHD interval",
                       "autotuned": tuning,
                       "l2": "inputs exceed L2 (fields of 64 runs and their particles)",
                       "parallelism": f"replicas x{world}"},
            "clocks": clk,
            # per chunk: prefix + batched mover + 5 binning kernels per run; per step and run:
            # split (3) + f(p) (1)
            "gpu_launches": int(round(sum(l * (2 + 5 * nruns) for l in graph_launches) +
                                      args.steps * 4 * nruns)),
            "e2e": {"value": e2e_value, "unit": UNIT,
                    "h2d_bytes_per_step": e2e_h2d // max(1, args.e2e_steps),
                    "d2h_bytes_per_step": e2e_d2h // max(1, args.e2e_steps)},
            "roofline": batch_roofline,
            "per_run_fp_error": acc}
    batch.close()
    for e in engines:
        e.close()
    if world == 1 and not args.no_cpu_baseline:
        w = runs[BATCH_SAMPLE_RUN]
        v, cores, n, steps, dt, _ = cpu_sample(w, args.cpu_seconds)
        line["cpu_baseline"] = {"value": v, "unit": UNIT, "cores": cores, "kind": "port",
                                "sample": f"{n} particles of {w.name} injected on the shock, one "
                                          f"MHD interval of FP64 pushes ({steps} particle-steps "
                                          f"in {dt:.2f} s)"}
    return line


# Fraction of the weighted mean importance added to every particle's in the
# learned arm (defensive importance sampling, Hesterberg 1995).
DEFENSIVE = 0.1


def run_learned(args, world, rank, local):
    """Learned splitting on the 256^3 compressible-turbulence field (the 3D
    workload's field and transport, f(p) up to 1e4 p0).  A plain run of
    n_train trajectories over the whole run length generates the training
    records (every record_every intervals) and labels them by whether the
    trajectory ends above p_label (the 99.9th percentile of its final
    momenta, or 100 p0 if lower); the network is trained on the GPU.  Then,
    on fresh particles, five arms run the same intervals:
      plain        split-precision, no splitting (2x the particles);
      fixed        split-precision with split_particle's fixed thresholds;
      learned      split-precision with the network applied inside the mover
                   as particles finish each interval (weight window 4, the
                   particle cap of 4e8, importance exp(z) floored at
                   DEFENSIVE times its weighted mean);
      fp64         the FP64 mover, no splitting: the independent reference;
      fp64_learned the FP64 mover with the same network applied by the
                   separate split kernel after each interval: the FP64
                   reference with samples in the tail.
    Each reports, above 100 p0 and above p_label, the weighted fraction, its
    Monte Carlo error and the effective samples per second, with one sample
    per injected particle (the tail weight of all its descendants)."""
    import numpy as np
    import torch
    from gpat import configs
    from gpat.engine import (FusedWindow, GPATCapacityError, Mlp, mover_learned_stats,
                             set_mover_learned, tail_by_ancestor, tail_weights, weighted_split,
                             window_params)

    torch.cuda.set_device(local)
    n_train = max(1000, int(args.train_trajectories * args.scale))
    n_cmp = max(1000, int(1e6 * args.scale))
    n_fp64 = max(1000, int(args.fp64_particles * args.scale))
    max_intervals = args.intervals if args.intervals > 0 else 100
    w = make_workload(args, 1, seed=3 + rank, nframes=max_intervals, scale=n_train / 1e8)
    p0 = w.params["p0"]
    pyield = 100.0 * p0

    def fresh(n, seed, cap, precision=1):
        """An engine holding n particles injected as the workload does
        (log-uniform in [p0, 10 p0]: the injection draws up to the workload's
        pmax) in an engine whose pmax is 1e4 p0, so split_particle's p <= pmax
        rule does not stop the splitting of the tail."""
        inj = configs.build_engine(w, device=local, nptl_max=n, seed=seed)
        configs.inject(inj, w, nptl=n)
        ps = inj.get_particles()
        inj.close()
        eng = configs.build_engine(w, device=local, nptl_max=cap, seed=seed,
                                   precision=precision, pmax=1.0e4 * p0)
        eng.put_particles(ps)
        return eng

    if args.intervals > 0:
        nint, pilot = args.intervals, None
    else:
        # run length: the first interval count at which 0.1 % of a plain
        # run's particles are above 100 p0 (100 p0 is then a tail)
        n_pilot = max(20000, int(2e5 * args.scale))
        eng = fresh(n_pilot, 50 + rank, n_pilot)
        nint, frac = max_intervals, 0.0
        for k in range(max_intervals):
            eng.particle_mover(mhd_tframe=k + 1)
            frac = tail_weights(eng, pyield)[1] / n_pilot
            if frac >= 1e-3:
                nint = k + 1
                break
        eng.close()
        pilot = {"particles": n_pilot, "intervals": nint, "fraction_above_100p0": frac}
        print(f"learned_3d: run length {nint} intervals ({frac:.2e} of {n_pilot} pilot "
              f"particles above 100 p0)", file=sys.stderr, flush=True)
    fixed_ratio, fixed_pmin = 1.5, 6.0
    every = args.record_every if args.record_every > 0 else max(1, nint // 10)

    def arm(kind, n, seed, recorder=None, net=None, target=None, cap=None, precision=1):
        eng = fresh(n, seed, cap or 2 * n, precision)
        pushes, capped, judged, pop = 0, False, 0, []
        win = FusedWindow(target, DEFENSIVE) if kind == "learned" else None
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        if kind == "learned":
            win.start(*net.score(eng, 0.0)[1:])
        for k in range(nint):
            if recorder is not None and k % every == 0:
                recorder.record(eng, k / nint)
            if kind == "learned":
                z_ref, z_floor = win.params()
                set_mover_learned(eng, net, (k + 1) / nint, 1.0, z_ref, 4.0, 3, z_floor=z_floor)
            eng.particle_mover(mhd_tframe=k + 1)
            pushes += eng.counters().last_mover_steps
            if kind == "learned":
                st = mover_learned_stats(eng)
                judged += st["judged"]
                win.update(st)
            if kind == "fp64_learned":
                _, lse, lsw = net.score(eng, (k + 1) / nint)
                z_ref, z_floor = window_params(lse, lsw, target, DEFENSIVE)
                weighted_split(eng, net, (k + 1) / nint, 1.0, z_ref, 4.0, 3, z_floor=z_floor)
            if kind == "fixed" and not capped:
                try:
                    eng.split_particle(fixed_ratio, fixed_pmin, 10)
                except GPATCapacityError:
                    capped = True
            pop.append(eng.nptl_current)
        torch.cuda.synchronize()
        secs = time.perf_counter() - t0
        if kind == "learned":
            set_mover_learned(eng, None)
        return eng, pushes, secs, capped, pop

    # 1. plain run generating the training records; labels from its final momenta
    net = Mlp(device=local, seed=7 + rank,
              record_capacity=n_train * ((nint + every - 1) // every))
    eng, train_pushes, train_s, _, _ = arm("plain", n_train, 100 + rank, recorder=net)
    print(f"learned_3d: training run {n_train} trajectories, {train_pushes} pushes in "
          f"{train_s:.1f} s", file=sys.stderr, flush=True)
    p_end = eng.get_particles()["p"]
    p_label = float(min(pyield, np.quantile(p_end, 0.999)))
    reached = int(np.sum(p_end > pyield))
    npos, nrec = net.label(eng, p_label)
    eng.close()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    loss = net.train(epochs=3, batch=8192, lr=3e-3, neg_keep=0.25, seed=5)
    torch.cuda.synchronize()
    fit_s = time.perf_counter() - t0

    print(f"learned_3d: labels {npos} positive of {nrec} records at p > {p_label / p0:.1f} p0, "
          f"fit {fit_s:.1f} s", file=sys.stderr, flush=True)

    # 2. the arms on fresh particles (another injection seed)
    out = {}
    clocks = ClockSampler(local)
    clocks.start()
    for kind, n, kw in (("plain", 2 * n_cmp, {}),
                        ("fixed", n_cmp, dict(cap=4 * n_cmp)),
                        ("learned", n_cmp, dict(net=net, target=2 * n_cmp, cap=int(4e8))),
                        ("fp64", n_fp64, dict(precision=0)),
                        ("fp64_learned", n_fp64, dict(net=net, target=2 * n_fp64,
                                                      cap=16 * n_fp64, precision=0))):
        e, pushes, secs, capped, pop = arm(kind, n, 200 + rank, **kw)
        d = {"particles": n, "pushes": pushes, "seconds": secs,
             "particle_steps_per_s": pushes / secs, "capped": capped,
             "final_particles": e.nptl_current,
             "population_min_max": [min(pop), max(pop)],
             "max_split_level": int(e.get_particles()["split_times"].max())}
        _, wall, _ = tail_weights(e, 0.0)
        d["total_weight_over_injected"] = wall / n
        for name, thr in (("above_100p0", pyield), ("above_p_label", p_label)):
            # one sample per injected particle: split copies share their
            # parent's history (the per-particle (sum w)^2 / sum w^2 is kept
            # as ess_particles, which overstates the samples of split runs)
            a = tail_by_ancestor(e, thr, n)
            _, ws, w2 = tail_weights(e, thr)
            d[name] = {"particles": a["particles"], "ancestors": a["ancestors"],
                       "fraction": a["fraction"], "sigma": a["sigma"], "ess": a["ess"],
                       "ess_per_s": a["ess"] / secs,
                       "ess_particles": ws * ws / w2 if w2 > 0 else 0.0}
        out[kind] = d
        print(f"learned_3d: {kind} " + json.dumps(d), file=sys.stderr, flush=True)
        e.close()
    clk = clocks.stop()
    net.close()
    for name in ("above_100p0", "above_p_label"):
        for ref in ("fp64", "fp64_learned"):
            j = out[ref][name]
            for kind in ("plain", "fixed", "learned", "fp64_learned"):
                if kind == ref or j["fraction"] <= 0:
                    continue
                d = out[kind][name]
                d[f"err_vs_{ref}"] = d["fraction"] / j["fraction"] - 1.0
                d[f"err_sigma_vs_{ref}"] = math.hypot(d["sigma"], j["sigma"]) / j["fraction"]
    if rank != 0:
        return
    learned = out["learned"]
    line = {"metric": METRIC, "value": learned["particle_steps_per_s"], "unit": UNIT,
            "n_gpus": world, "steps": 1, "warmup": 0,
            "ms_per_step": 1e3 * learned["seconds"] / nint,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32", "data": "synthetic",
            "config": {"workload": f"learned_splitting_{w.name}", "particles": n_cmp,
                       "intervals": nint, "run_length_pilot": pilot,
                       "yield_threshold_p_over_p0": pyield / p0,
                       "label_threshold_p_over_p0": p_label / p0,
                       "label_rule": "trajectory ends above min(100 p0, 99.9th percentile of "
                                     "the plain run's final momenta)",
                       "training_particles_above_100p0": reached,
                       "step": "one MHD interval of the learned arm (mover with the network "
                               "applied to particles finishing the interval)",
                       "l2": "inputs exceed L2 (256^3 field records 1.7 GB)",
                       "parallelism": f"replicas x{world}"},
            "clocks": clk, "gpu_launches": None, "e2e": None,
            "learned_splitting": {
                "network": "8-64-64-64-1 SiLU, BF16 weights and activations, FP32 accumulation "
                           "(mma.sync m16n8k16)",
                "importance": f"exp(z) + {DEFENSIVE} x weighted mean of exp(z) (defensive mixture)",
                "weight_window_ratio": 4.0, "max_split_level": 3,
                "training": {"trajectories": n_train, "records": nrec, "positives": npos,
                             "record_every_intervals": every, "plain_run_seconds": train_s,
                             "fit_seconds": fit_s, "final_loss": loss, "epochs": 3},
                "fixed_threshold": {"split_ratio": fixed_ratio, "pmin_split": fixed_pmin},
                "fp64_references": {
                    "fp64": "FP64 mover, no splitting (independent of the method)",
                    "fp64_learned": "FP64 mover with the network applied by the separate "
                                    "split kernel (tail samples)"},
                "arms": out,
                "ess_per_s_learned_over_fixed": {
                    name: learned[name]["ess_per_s"] / max(out["fixed"][name]["ess_per_s"], 1e-30)
                    for name in ("above_100p0", "above_p_label")},
                "ess_per_s_learned_over_plain": {
                    name: learned[name]["ess_per_s"] / max(out["plain"][name]["ess_per_s"], 1e-30)
                    for name in ("above_100p0", "above_p_label")}}}
    return line


# Keys of a workload's own line kept when it is reported inside the headline.
EXTRA_KEYS = ("value", "unit", "ms_per_step", "steps", "warmup", "config", "clocks",
              "roofline", "per_run_fp_error", "accuracy")


def other_configs(args, local) -> dict:
    """The 3D compressible turbulence (256^3, 1e8 particles) and the batch of
    64 turbulent-shock runs, each measured for one timed MHD interval after
    one warm-up interval with the same mover options, and the learned
    splitting comparison at a tenth of its size, for the headline line."""
    out = {}
    common = dict(steps=1, warmup=1, e2e_steps=0, no_cpu_baseline=True, scale=1.0, grid=2048)

    def extra(key, fn):
        # a failing extra is recorded in the line, which the headline keeps
        try:
            out[key] = fn()
        except Exception as e:  # noqa: BLE001 - reported, not hidden
            out[key] = {"error": f"{type(e).__name__}: {e}"}
            print(f"bench: {key} failed: {e}", file=sys.stderr, flush=True)

    def turbulence_3d():
        a3 = argparse.Namespace(**{**vars(args), **common, "workload": "turbulence_3d",
                                   "no_accuracy": True, "tiles": args.tiles_3d})
        l3 = run_ours(a3, 1, 0, local)
        return {k: l3[k] for k in EXTRA_KEYS if k in l3}

    def batched():
        ab = argparse.Namespace(**{**vars(args), **common, "workload": "batched_shock_2d",
                                   "no_accuracy": False})
        lb = run_batch(ab, 1, 0, local)
        return {k: lb[k] for k in EXTRA_KEYS if k in lb}

    def learned():
        # learned vs fixed-threshold splitting on the 3D field at a tenth of
        # the full comparison's particles (1e6 training trajectories, 1e5
        # particles per split-precision arm, 2e4 per FP64 reference arm,
        # 100 intervals)
        al = argparse.Namespace(**{**vars(args), "workload": "learned_3d", "scale": 0.1,
                                   "grid": 2048, "tiles": "off"})
        ll = run_learned(al, 1, 0, local)
        return {k: ll[k] for k in ("value", "unit", "ms_per_step", "config", "clocks",
                                   "learned_splitting")}

    extra("turbulence_3d_256", turbulence_3d)
    extra("batched_shock_2d_64", batched)
    extra("learned_3d_scale_0.1", learned)
    return out


# What the line on standard output may take; readers that keep the end of a log then
# have all of it.
LINE_BYTES = 3000
CONTRACT_KEYS = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
                 "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "impl", "config",
                 "clocks", "gpu_launches", "e2e")


def rounded(x):
    """Figures to six digits, long texts and lists cut."""
    if isinstance(x, float):
        return float(f"{x:.6g}")
    if isinstance(x, dict):
        return {k: rounded(v) for k, v in x.items()}
    if isinstance(x, (list, tuple)):
        return [rounded(v) for v in x[:8]]
    return x[:100] if isinstance(x, str) else x


def summary(line) -> dict:
    """The figures of a workload's own line that its summary keeps."""
    out = {k: line[k] for k in ("error", "value", "unit", "ms_per_step") if k in line}
    roof = line.get("roofline") or {}
    out.update({k: roof[k] for k in ("bound", "frac") if k in roof})
    errs = [abs(r["tail_err"]) for r in line.get("per_run_fp_error") or []
            if isinstance(r.get("tail_err"), (int, float))]
    if errs:
        out["runs_compared"], out["max_abs_tail_err"] = len(errs), max(errs)
    learned = line.get("learned_splitting") or {}
    for k in ("ess_per_s_learned_over_fixed", "ess_per_s_learned_over_plain"):
        if k in learned:   # no particle of the other arm up there: no ratio
            out[k] = {name: v if v < 1e12 else None for name, v in learned[k].items()}
    return out


def short_line(line) -> dict:
    """The line of standard output: the contract's keys whole, of the rest the figures,
    and of the other configurations their summaries."""
    out = {k: line[k] for k in CONTRACT_KEYS if k in line}
    rest = {k: v for k, v in line.items() if k not in out}
    roof = rest.pop("roofline", None)
    if roof:
        hbm = roof.get("hbm") or {}
        out["roofline"] = rounded({**{k: roof[k] for k in ("bound", "achieved", "peak", "unit", "frac",
                                                           "traffic", "kernel_steps_per_s", "kernel")
                                      if k in roof}, "hbm_frac": hbm.get("frac")})
    acc = rest.pop("accuracy", None)
    if acc:
        out["accuracy"] = rounded({k: v for k, v in acc.items() if not isinstance(v, (list, str))})
    for key in ("cpu_baseline", "fp64_gpu"):
        if rest.get(key):
            out[key] = rounded(rest.pop(key))
    out.update(rounded({k: v for k, v in summary(rest).items() if k not in out}))
    configs = rest.pop("configs", None)
    if configs:
        out["configs"] = {k: rounded(summary(v)) for k, v in configs.items()}
    for key in ("configs", "fp64_gpu", "cpu_baseline", "accuracy", "roofline"):
        if len(json.dumps(out)) <= LINE_BYTES:
            break
        out.pop(key, None)
    return out


def emit(line):
    """The whole line, with every figure, on standard error; the short one on standard
    output."""
    print("bench: details " + json.dumps(line), file=sys.stderr, flush=True)
    print(json.dumps(short_line(line)), flush=True)


def main():
    args = parse_args()
    world, rank, local = dist_setup()
    if args.impl == "reference":
        run_reference(args, world, rank)
    elif args.workload == "batched_shock_2d":
        line = run_batch(args, world, rank, local)
        if line is not None:
            emit(line)
    elif args.workload == "learned_3d":
        line = run_learned(args, world, rank, local)
        if line is not None:
            emit(line)
    else:
        line = run_ours(args, world, rank, local)
        if line is not None and args.workload == "turbulent_shock_2d" and not args.no_extras \
                and world == 1:
            line["configs"] = other_configs(args, local)
        if line is not None:
            emit(line)
    if world > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
