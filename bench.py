#!/usr/bin/env python
"""bench.py -- particle-steps/s of the Stokes-limit midpoint step on B200.

Workload (default): the single large instance of the benchmark set, 128^3
periodic cells (dx = 1), 65,536 particles as 4,096 bead-spring chains of 16
beads (k = 10, r0 = 1), soft repulsion eps = 1, rc = 1.5, eta = 1, kT = 0.01,
dt = 0.005, 4-point kernel; noise drawn on the device.  Inputs are seeded
synthetic data (there is no dataset).

One step = one full midpoint step (noise, 2 x (cell list, forces, spread,
FFT Stokes solve), RFD drift spreads, predictor and corrector).  `value` is
device time (CUDA events on the library's stream), L2 flushed between timed
steps with a 256 MiB write.  `e2e` is the same metric through the C ABI with
the step's input positions copied from pinned host memory and the new
positions read back every step.

Multi-GPU: one process per GPU, each an independent replica (the path has no
exchange step); value = all particle-steps / max-over-ranks time.
`--impl reference`: the FP64 CPU implementation of the same step on the
host's cores (the reference's CUDA build does not compile with CUDA 12).
"""
import argparse
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

WORKLOAD = "plain_128"


def parse_args():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=200)
    p.add_argument("--warmup", type=int, default=10)
    p.add_argument("--impl", default="ours", choices=["ours", "reference"])
    p.add_argument("--workload", default=WORKLOAD)
    p.add_argument("--cpu-seconds", type=float, default=20.0)
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--no-batched", action="store_true", help="skip the batched and served lines")
    return p.parse_args()


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


# ------------------------------------------------------------------ clocks --
class ClockSampler:
    FIELDS = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.rows = []
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            parts = [x.strip() for x in line.split(",")]
            if len(parts) >= 8:
                self.rows.append(parts)

    def stop(self):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"], "samples": 0}
        sm = [float(r[0]) for r in self.rows if r[0].replace(".", "").isdigit()]
        mx = [float(r[1]) for r in self.rows if r[1].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in self.rows for i in range(4)
                          if r[4 + i].lower().startswith("active")})
        return {"sm_mhz": float(np.median(sm)) if sm else None,
                "sm_max_mhz": max(mx) if mx else None, "reasons": reasons,
                "samples": len(self.rows)}


# ---------------------------------------------------------- algorithmic bytes
MULTI_KERNEL_STAGES = ("noise",)
# stages that are launches of one kernel
KERNEL_OF_STAGE = {"spread": "k_spread", "spread_rfd": "k_spread"}

def stage_bytes(name, P):
    """Algorithmic DRAM bytes of one interval of a stage as the per-stage
    timer marks it: one kernel, except "noise" (k_noise and both k_div).
    FP32 fields, FP64 particle state, FP32 stress samples and their
    divergence, int64 fixed-point spread grid.  P["fused"]: the Verlet-list
    forces are computed inside the spread that follows them (the default)."""
    nc, npart, k = P["nc"], P["np"], P["kernel"]
    spec = 3 * 8 * (P["mx"] // 2 + 1) * P["my"] * P["mz"]
    touched = 3 * 8 * min(P["nc"], k ** 3 * npart)
    # positions read + F written and the pair lists read, when fused;
    # positions and F read otherwise
    part = 52 * npart if P.get("fused", True) else 48 * npart
    return {
        # the whole interval (three kernels): the raw samples and particle
        # noise written (48 nc + 36 np), the divergence of sample 1
        # (6 nc read, 3 nc written) and of sample 2 added to it (9 nc read,
        # 3 nc written)
        "noise": 48 * nc + 36 * npart + 36 * nc + 48 * nc,
        "cells": 40 * npart + 12 * P["mN"],
        "forces": 52 * npart + 4 * P["mN"],
        "grid_zero": 24 * nc,
        "spread": part + 2 * touched,
        # force spread + the drift test (reference mode: the drift spreads
        # cancel and are skipped except at stencil changes)
        "spread_rfd": part + 2 * touched + 36 * npart,
        # (five-pass schedule) int64 field read, divergence of the noise read,
        # W written
        "wbuild": 24 * nc + 12 * nc + 12 * nc,
        "field_clear": 24 * nc,
        # W built on the way in: int64 field read, divergence of the noise
        # read, half spectrum written (the pass also clears the field for the
        # next spread, which is this design's own traffic)
        "plane_fwd": 24 * nc + 12 * nc + spec,
        "plane_inv": spec + 12 * nc,
        "fft_x": 12 * nc + spec,                   # line schedule: x forward or inverse
        "fft_y": 2 * spec,
        "xfwd": 12 * nc + spec,                    # general sizes: x forward of W
        "yfft": 2 * spec,
        "zsolve": 2 * spec,
        "xinv": spec + 12 * nc,
        "interp_update": 72 * npart + min(12 * nc, 12 * k ** 3 * npart),
        "counter": 8,
    }.get(name, 0)


# --------------------------------------------------------------- cpu side ---
def cpu_run(workload, seconds, real="f64", native=True):
    """Time the CPU implementation of the step (the oracle, built for this
    host with -march=native, OpenMP over all host threads) on a bounded
    sample of the workload; real="f32" times the FP32 build of the same
    source."""
    from oracle import oracle_py as O
    from fluam_b200 import workloads as W
    w = W.WORKLOADS[workload]
    m, L = w["cells"], w["box"]
    if w["chains"]:
        q, bi, bj = W.chains(w["chains"], w["beads"], L, 1, w["r0"])
    else:
        q, bi, bj = W.uniform(w["n"], L, 1), None, None
    try:
        o = O.Oracle(m, m, m, L, L, L, q, eta=w["eta"], kT=w["kT"], dt=w["dt"], cutoff=w["rc"],
                     kernel=w["kernel"], pair=O.PAIR_SOFT, soft_epsilon=w["eps"], seed=1,
                     real=real, native=native)
        build = "-march=native" if native else "-march=x86-64-v3"
    except Exception:  # no compiler on this host: the portable build
        o = O.Oracle(m, m, m, L, L, L, q, eta=w["eta"], kT=w["kT"], dt=w["dt"], cutoff=w["rc"],
                     kernel=w["kernel"], pair=O.PAIR_SOFT, soft_epsilon=w["eps"], seed=1,
                     real=real, native=False)
        build = "-march=x86-64-v3"
    if bi is not None:
        o.set_bonds(bi, bj, np.full(len(bi), w["k"]), np.full(len(bi), w["r0"]))
    o.step(1)  # warm-up (page faults, thread pool)
    n = 0
    t0 = time.perf_counter()
    while True:
        o.step(1)
        n += 1
        el = time.perf_counter() - t0
        if el >= seconds or (n >= 2 and el * (n + 1) / n > 3 * seconds):
            break
    npart = q.shape[1]
    prec = "FP64" if real == "f64" else "FP32"
    return {"value": npart * n / el, "unit": "particle-steps/s", "cores": O.num_threads(),
            "kind": "port", "steps": n, "seconds": el, "precision": prec,
            "sample": f"{n} steps of {workload} ({m}^3, {npart} particles), {prec} CPU "
                      f"restatement ({build}), {el:.1f} s, OpenMP {O.num_threads()} threads"}


def run_reference(args, rank, world):
    if rank != 0:
        return 0
    per = max(args.cpu_seconds / max(args.steps, 1), 1.0)
    per = min(per, args.cpu_seconds)
    r = cpu_run(args.workload, per * max(1, min(args.steps, 3)))
    r32 = cpu_run(args.workload, min(per, 10.0), real="f32")
    line = {
        "metric": "particle-steps/s", "value": r["value"], "unit": "particle-steps/s",
        "impl": "reference", "n_gpus": world, "steps": r["steps"], "warmup": 1,
        "requested_steps": args.steps, "requested_warmup": args.warmup,
        "higher_is_better": True, "dtype": "f64", "data": "synthetic",
        "config": workload_config(args.workload),
        "precision": {"fields": "fp64", "positions": "fp64", "spread": "fp64 sums"},
        "cpu_baseline": {"value": r["value"], "unit": r["unit"], "cores": r["cores"],
                         "kind": r["kind"], "sample": r["sample"]},
        "cpu_fp32": {"value": r32["value"], "unit": r32["unit"], "cores": r32["cores"],
                     "kind": r32["kind"], "sample": r32["sample"]},
        "e2e": {"value": r["value"], "unit": r["unit"], "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
        "note": "the reference's CUDA build does not compile with CUDA 12 (legacy texture "
                "references); this arm times the CPU restatement of its step (FP64, and its "
                "FP32 build in cpu_fp32) on the host's cores",
    }
    print(json.dumps(line), flush=True)
    return 0


def aggregate(local_times, dist=None, device=None):
    """Max over ranks of each local time (ms or s), as floats; the replicas
    do not exchange data, so this is the only collective of a run."""
    if dist is None or not dist.is_initialized() or dist.get_world_size() == 1:
        return [float(x) for x in local_times]
    import torch
    t = torch.tensor([float(x) for x in local_times], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return [float(x) for x in t.cpu()]


def replica_seed(rank, base=1):
    """Each rank runs its own replica of the workload: same sizes, own seed."""
    return base + rank


def workload_config(name):
    from fluam_b200 import workloads as W
    w = W.WORKLOADS[name]
    return {"workload": f"{name}: {w['cells']}^3 periodic cells dx=1, {w['n']} particles"
                        + (f" ({w['chains']} chains x {w['beads']} beads, k={w['k']}, r0={w['r0']})"
                           if w["chains"] else " uniform")
                        + f", soft repulsion eps={w['eps']} rc={w['rc']}, {w['kernel']}-pt kernel,"
                          f" eta={w['eta']} kT={w['kT']} dt={w['dt']}",
            "cells": w["cells"], "np": w["n"], "kernel": w["kernel"],
            "l2": "flushed between timed steps (256 MiB write)"}


# -------------------------------------------------------------- GPU side ---
def step_bytes(nc, npart):
    """Algorithmic HBM bytes of one midpoint step: 144 nc + 384 np (FP32
    fields written and read once per pass, FP64 particle state, noise kept
    in registers)."""
    return 144 * nc + 384 * npart


def run_fp64_form(torch, workload, steps=20, warmup=3):
    """The all-FP64 precision form (noise, spreading, fields, FFTs and
    interpolation in FP64) on the same workload, device time per step."""
    from fluam_b200 import StokesLimit, workloads
    cfg, q, bonds = workloads.build(workload, seed=1)
    cfg.precision = 2  # FSL_PRECISION_FP64
    g = StokesLimit(cfg, q)
    if bonds is not None:
        g.load_bonds(*bonds)
    s = torch.cuda.ExternalStream(g.L.fsl_stream(g.h))
    g.step(warmup)
    g.sync()
    a, z = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record(s)
    g.step(steps)
    z.record(s)
    g.sync()
    ms = a.elapsed_time(z) / steps
    g.close()
    return {"value": q.shape[1] / (ms * 1e-3), "unit": "particle-steps/s", "ms_per_step": ms,
            "steps": steps,
            "precision": "fp64 noise, spreading (FP64 atomics), fields, FFTs, interpolation",
            "l2": "not flushed (the step's FP64 state exceeds the L2)"}


def compact_tuning(t):
    """The picks of one size class's tuner (made at its first step), for the
    JSON line."""
    return {"cells": t["mx"], "instances": t["n"], "fft_schedule": t["fft_schedule"],
            "schedule_us": [round(u, 2) for u in t["schedule_us"]],
            "z_tile": [t["z_tile_kx"], t["z_tile_ky"]], "z_us": [round(u, 2) for u in t["z_us"]],
            "planes_per_block": t["plane_pb"], "plane_us": [round(u, 2) for u in t["plane_us"]],
            "list_build": t["list_build"], "list_us": [round(u, 2) for u in t["list_us"]]}


def run_batched(torch, steps=20, warmup=3, plain_sample=128):
    """The mixed 1,024-replica workload as one batch (one launch per stage and
    size class, one graph per step), next to the same replicas stepped one at
    a time on the plain single-instance path (a seeded sample of them)."""
    import ctypes
    from fluam_b200 import Batch, StokesLimit, workloads
    inst = workloads.mixed(1024)
    b = Batch([c for c, _ in inst], [q for _, q in inst])
    info = b.info()
    stream = torch.cuda.ExternalStream(b.stream())
    b.step(warmup)
    b.sync()
    tuning = [compact_tuning(t) for t in b.class_tuning()]
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    b.step(steps)
    e1.record(stream)
    b.sync()
    ms = e0.elapsed_time(e1) / steps
    npt, nct = info["np_total"], info["nc_total"]
    # end to end: every step's positions in from and out to pinned host memory
    # (fsl_batch_step_io: the copies, scatter and gather inside the step's
    # graph, the copy in beside the noise); one untimed call captures it
    hq = torch.empty(int(b.offsets[-1]), dtype=torch.float64).pin_memory()
    b.positions_packed(hq.numpy())
    b.step_io(hq.data_ptr(), hq.data_ptr())
    ke = max(5, steps // 2)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(ke):
        b.step_io(hq.data_ptr(), hq.data_ptr())
    b.sync()
    e2e_s = time.perf_counter() - t0
    launches = b.info()["launches_per_step"]
    b.close()
    # plain path, one replica at a time: device time of its own steps
    tot_p, tot_ms = 0, 0.0
    for c, q in inst[:plain_sample]:
        g = StokesLimit(c, q)
        s = torch.cuda.ExternalStream(g.L.fsl_stream(g.h))
        g.step(3)
        g.sync()
        a, z = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(s)
        g.step(5)
        z.record(s)
        g.sync()
        tot_ms += a.elapsed_time(z)
        tot_p += 5 * q.shape[1]
        g.close()
    plain = tot_p / (tot_ms * 1e-3)
    value = npt / (ms * 1e-3)
    return {
        "workload": "mixed_1024: 1,024 cubic replicas, edge U{16,24,32,48,64}, np log-U[8,2048], "
                    "eta U[0.5,2], kT 0.01, dt 0.01, 3-pt kernel, soft repulsion eps 1 rc 1.5",
        "replicas": info["n"], "classes": info["classes"], "np_total": npt, "nc_total": nct,
        "value": value, "unit": "particle-steps/s", "ms_per_step": ms, "steps": steps,
        "grid_cell_updates_per_s": nct / (ms * 1e-3),
        "step_bytes": step_bytes(nct, npt),
        "achieved_GBs": step_bytes(nct, npt) / (ms * 1e-3) / 1e9,
        "e2e": {"value": npt * ke / e2e_s, "unit": "particle-steps/s",
                "h2d_bytes_per_step": 24 * npt, "d2h_bytes_per_step": 24 * npt},
        "plain_one_at_a_time": {"value": plain, "unit": "particle-steps/s",
                                "sample": f"first {plain_sample} replicas, 5 graph-replayed steps "
                                          "each, device time"},
        "speedup_vs_plain": value / plain,
        "gpu_launches_per_step": launches,
        "autotune": tuning,
        "l2": "inputs (device state of all replicas) far larger than L2",
    }


def serve_requests(n_per_s, duration, seed, steps_range):
    """A seeded open-loop Poisson request stream: (arrival s, config, q, steps)."""
    from fluam_b200 import PAIR_SOFT, make_config, workloads
    rng = np.random.default_rng(seed)
    t, out = 0.0, []
    while True:
        t += rng.exponential(1.0 / n_per_s)
        if t > duration:
            return out
        m = int(rng.choice(np.arange(16, 97, 8)))
        npart = int(round(np.exp(rng.uniform(np.log(16), np.log(16384)))))
        nst = int(round(np.exp(rng.uniform(np.log(steps_range[0]), np.log(steps_range[1])))))
        cfg = make_config((m, m, m), (float(m),) * 3, eta=float(rng.uniform(0.5, 2.0)), kT=0.01,
                          dt=0.01, cutoff=1.5, kernel=int(rng.choice((3, 4))), pair=PAIR_SOFT,
                          seed=int(rng.integers(1, 1 << 40)))
        out.append((t, cfg, workloads.uniform(npart, m, int(rng.integers(1 << 30))), nst))


# Arrival rates of the serving sweep (requests/s) and how long each stream
# keeps arriving (s): about 200 requests per rate.
SERVE_SWEEP = ((10.0, 20.0), (100.0, 2.0), (1000.0, 0.2))


def serve_stream(srv, reqs):
    """Submits reqs at their arrival times; returns (infos, span s)."""
    ids = []
    t0 = time.perf_counter()
    for t, c, q, n in reqs:
        d = t0 + t - time.perf_counter()
        if d > 0:
            time.sleep(d)
        ids.append(srv.submit(c, q, n))
    infos = [srv.wait(i) for i in ids]
    for i in ids:
        srv.result(i)
    span = max(x["done_s"] for x in infos) - min(x["submit_s"] for x in infos)
    return infos, span


def run_served(sweep=SERVE_SWEEP, steps_range=(100, 5000), seed=11, plain_sample=12):
    """The serving loop under open-loop Poisson streams at each rate of the
    sweep: completion latency and aggregate throughput, next to a sample of
    the same requests run one at a time on the plain path (wall time of
    create + steps + read-back)."""
    from fluam_b200 import Server, StokesLimit
    streams = [serve_requests(rate, dur, seed + k, steps_range) for k, (rate, dur) in enumerate(sweep)]
    srv = Server(hbm_budget=150 * 10 ** 9)
    # warm-up: one short request per size class builds the FFT plans
    warm = {}
    for reqs in streams:
        for _, c, q, _ in reqs:
            warm.setdefault((c.mx, c.kernel), (c, q[:, :16]))
    for rid in [srv.submit(c, q, 2) for c, q in warm.values()]:
        srv.wait(rid)
        srv.result(rid)
    rows = []
    for (rate, dur), reqs in zip(sweep, streams):
        infos, span = serve_stream(srv, reqs)
        lat = np.array([x["done_s"] - x["submit_s"] for x in infos])
        work = sum(q.shape[1] * n for _, _, q, n in reqs)
        rows.append({"rate_per_s": rate, "arrivals_s": dur, "requests": len(reqs),
                     "completed": int(sum(x["state"] == 2 for x in infos)),
                     "value": work / span, "unit": "particle-steps/s", "span_s": span,
                     "latency_p50_s": float(np.percentile(lat, 50)),
                     "latency_p99_s": float(np.percentile(lat, 99))})
    st = srv.stats()
    srv.close()
    # plain path, one request at a time (a seeded sample across the sweep)
    pool = [r for reqs in streams for r in reqs]
    pick = np.random.default_rng(seed).choice(len(pool), size=min(plain_sample, len(pool)), replace=False)
    p_work, p_s = 0, 0.0
    for k in pick:
        _, c, q, n = pool[int(k)]
        a = time.perf_counter()
        g = StokesLimit(c, q)
        g.step(n)
        g.positions()
        g.close()
        p_s += time.perf_counter() - a
        p_work += q.shape[1] * n
    plain = p_work / p_s
    top = rows[-1]
    return {
        "workload": f"Poisson streams at {', '.join('%g' % r for r, _ in sweep)} req/s: edge "
                    f"U{{16,24,...,96}}, np log-U[16,16384], steps log-U[{steps_range[0]},{steps_range[1]}], "
                    "eta U[0.5,2], 3/4-pt kernel 50/50, soft repulsion, 150 GB budget",
        "sweep": rows, "value": top["value"], "unit": "particle-steps/s",
        "latency_p50_s": top["latency_p50_s"], "latency_p99_s": top["latency_p99_s"],
        "rounds": st["rounds"], "captures": st["captures"], "slots": st["slots"],
        "plain_one_at_a_time": {"value": plain, "unit": "particle-steps/s",
                                "sample": f"{len(pick)} requests of the sweep, wall time"},
        "speedup_vs_plain": top["value"] / plain,
    }


def main():
    args = parse_args()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", str(args.gpus)))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        return run_reference(args, rank, world)

    import torch
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                device_id=torch.device("cuda", local))

    from fluam_b200 import StokesLimit, workloads
    cfg, q, bonds = workloads.build(args.workload, seed=replica_seed(rank))
    cfg.device = local
    sim = StokesLimit(cfg, q)
    if bonds is not None:
        sim.load_bonds(*bonds)
    npart = q.shape[1]
    stream = torch.cuda.ExternalStream(sim.L.fsl_stream(sim.h))
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device="cuda")

    sim.step(max(args.warmup, 3))
    sim.sync()
    tuning = compact_tuning(sim.tuning())
    if dist:
        dist.barrier()
    torch.cuda.synchronize()

    def timed_pass(k):
        e0 = [torch.cuda.Event(enable_timing=True) for _ in range(k)]
        e1 = [torch.cuda.Event(enable_timing=True) for _ in range(k)]
        for i in range(k):
            flush.fill_(float(i))
            torch.cuda.synchronize()
            e0[i].record(stream)
            sim.step(1)
            e1[i].record(stream)
        torch.cuda.synchronize()
        return sum(a.elapsed_time(b) for a, b in zip(e0, e1))

    clocks = ClockSampler(local)
    clocks.start()
    time.sleep(0.3)
    total_ms = timed_pass(args.steps)            # pass A: the headline number
    launches_a = sim.status()["launches_per_step"]  # kernels per step of pass A
    sim.profile(True)                            # pass B: per-stage events
    sim.step(1)
    sim.sync()
    sim.profile(True)
    prof_ms = timed_pass(args.steps)
    stages = sim.profile_read()
    sim.profile(False)
    clk = clocks.stop()
    sim.sync()
    st = sim.status()

    # e2e through the C ABI with pinned host buffers: every step's positions
    # in from and out to host memory (fsl_step_io: the copies are nodes of
    # the step's graph, the copy in beside the noise); one untimed call
    # captures that graph
    hq = torch.empty((3, npart), dtype=torch.float64).pin_memory()
    hq.copy_(torch.from_numpy(sim.positions()))
    import ctypes
    qp = ctypes.c_void_p(hq.data_ptr())
    check_rc = sim.L.fsl_step_io(sim.h, qp, qp)
    if check_rc != 0:
        raise RuntimeError(f"fsl_step_io failed ({check_rc})")
    ke = max(10, args.steps // 4)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(ke):
        sim.L.fsl_step_io(sim.h, qp, qp)
    e2e_s = time.perf_counter() - t0
    sim.sync()

    t_max, e2e_max = aggregate([total_ms, e2e_s], dist, device="cuda")
    if dist:
        dist.barrier()

    if rank == 0:
        hbm, peak_kind = peaks()
        P = {"nc": cfg.mx * cfg.my * cfg.mz, "np": npart, "kernel": cfg.kernel, "mx": cfg.mx,
             "my": cfg.my, "mz": cfg.mz,
             "mN": int(np.prod(sim.neighbor_grid())), "fused": "forces" not in stages}
        # the dominant kernel: the one with the most time over its stages, of
        # those whose timed intervals hold one kernel ("noise" holds three)
        kernels = {}
        for k, v in stages.items():
            if k not in MULTI_KERNEL_STAGES:
                kernels.setdefault(KERNEL_OF_STAGE.get(k, k), []).append(k)
        dname, dom = max(kernels.items(), key=lambda kv: sum(stages[k]["total_ms"] for k in kv[1]))
        launches = max(sum(stages[k]["launches"] for k in dom), 1)
        avg_ms = sum(stages[k]["total_ms"] for k in dom) / launches
        abytes = sum(stage_bytes(k, P) * stages[k]["launches"] for k in dom) / launches
        achieved = abytes / (avg_ms * 1e-3) / 1e9
        traffic = None  # DRAM bytes of a launch (mean) from the committed ncu capture
        try:
            with open(os.path.join(ROOT, "profiles", "traffic_%s.json" % args.workload.replace("plain_", "plain"))) as f:
                tr = json.load(f)["stages"]
            traffic = sum(tr[k]["dram_bytes"] * stages[k]["launches"] for k in dom) / launches
        except (OSError, KeyError, ValueError):
            traffic = None
        cpu = cpu32 = None
        if not args.no_cpu_baseline:
            try:
                cpu = cpu_run(args.workload, args.cpu_seconds)
                cpu32 = cpu_run(args.workload, min(args.cpu_seconds, 10.0), real="f32")
            except Exception as e:  # reported, not fatal
                cpu = {"value": None, "unit": "particle-steps/s", "cores": 0, "kind": "port",
                       "sample": f"failed: {e}"}
        value = world * npart * args.steps / (t_max * 1e-3)
        line = {
            "metric": "particle-steps/s", "value": value, "unit": "particle-steps/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": t_max / args.steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": workload_config(args.workload),
            "parallelism": f"replicas{world}" if world > 1 else "single",
            "precision": {"fields": "fp32", "positions": "fp64", "spread": "int64 fixed point 2^-40"},
            "grid_cell_updates_per_s": world * P["nc"] * args.steps / (t_max * 1e-3),
            "e2e": {"value": world * npart * ke / e2e_max, "unit": "particle-steps/s",
                    "h2d_bytes_per_step": 24 * npart, "d2h_bytes_per_step": 24 * npart},
            "roofline": {"bound": "hbm", "kernel": dname, "achieved": achieved, "peak": hbm,
                         "peak_kind": peak_kind, "unit": "GB/s", "frac": achieved / hbm,
                         "traffic": traffic, "algorithmic_bytes_per_launch": abytes,
                         "avg_launch_ms": avg_ms},
            "stages_ms_per_step": {k: v["total_ms"] / args.steps for k, v in sorted(stages.items())},
            "profiled_ms_per_step": prof_ms / args.steps,
            "cpu_baseline": cpu,
            "cpu_fp32": cpu32,
            "clocks": clk,
            "gpu_launches": launches_a * args.steps,
            "autotune": tuning,
            "step_roofline": {"bytes_per_step": step_bytes(P["nc"], npart),
                              "achieved": step_bytes(P["nc"], npart) / (t_max / args.steps * 1e-3) / 1e9,
                              "peak": hbm, "unit": "GB/s",
                              "frac": step_bytes(P["nc"], npart) / (t_max / args.steps * 1e-3) / 1e9 / hbm},
        }
        if world == 1:
            try:
                line["fp64_form"] = run_fp64_form(torch, args.workload)
            except Exception as e:  # reported, not fatal
                line["fp64_form"] = {"error": repr(e)}
        if world == 1 and not args.no_batched:
            sim.close()
            for key, fn in (("batched", run_batched), ("served", run_served)):
                try:
                    line[key] = fn(torch) if key == "batched" else fn()
                except Exception as e:  # reported, not fatal
                    line[key] = {"error": repr(e)}
        print(json.dumps(line), flush=True)
    sim.close()
    if dist:
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
