#!/usr/bin/env python
"""Spin-flip attempts/s of the B200 annealer on the muon-tomography pyramid.

Workload (one step): the 306,328-bit, 75,594-ray pyramid QUBO (11.2 M bit-ray
entries, kappa = ln 999, lambda = 2), 16 branches annealed T 50 -> 1 over 200
sweeps then held 50 sweeps at T = 1 (the reference's default posterior
schedule, ising_recon.hpp:81-86), fp64 residual refresh every 50 sweeps; the
branches' fp64 energies and per-bit void fractions are computed on the device.
attempts per step = 16 * 250 * 306,328.

  value   -- device-resident problem, CUDA events on the solve's stream, L2
             flushed (256 MB write) before every timed step, outside the events;
  e2e     -- the public C ABI from pinned host buffers every step: upload and
             plan the problem, solve, read the void fractions back (after up
             to 3 untimed warm-up steps, as for the timed region);
  --impl reference -- the reference's own CPU branch_fractions
             (oracle/_ref, compiled from the reference sources) on this host.

The default run (one GPU) also records, beside the pyramid line, the batched
4,096-instance Max-Cut stream ("batch": packed solve against one qb_solve per
instance) and the weighted 200,000-bit lattice QUBO ("qubo"), each measured by
its own ``--workload`` run in a child process with 3 warm-up steps and 1 timed
step (``--no-side-workloads`` skips them).

Multi-GPU: one process per GPU (torchrun); every rank solves its own copy of
the workload (branches are independent: weak scaling, no collective on the
data path); the timed region is bracketed by barriers and the slowest rank's
time is reported.
"""
import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

WORKLOAD = "muon-tomography pyramid: 306,328 bits, 75,594 rays, 16 branches, T 50->1 (200 sweeps) + 50 at T=1"
METRIC = "spin-flip attempts/s"
BRANCHES = 16
# DRAM bytes (read + write) per sweep of resid_lockstep_kernel from the
# committed ncu capture of a 10-sweep launch on the same pyramid and 16
# branches (profiles/resid_lockstep_pyramid.md): 1040.9 MB + 4.6 MB over 10
# sweeps. The bit->ray structure (8-byte entries, 87 MB) streams from DRAM
# once per sweep, so the traffic of a full launch is this figure times its
# sweeps.
NCU_TRAFFIC_PER_SWEEP = (1040.907e6 + 4.588288e6) / 10


def log(*a):
    print(*a, file=sys.stderr, flush=True)


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks and throttle reasons, sampled every 200 ms."""

    FIELDS = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
              "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
              "clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_id):
        self.gpu_id = gpu_id
        self.proc = None
        self.lines = []
        self.t = None

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu_id), f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.t.join(timeout=2)
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 7:
                continue
            try:
                sm.append(float(f[0]))
                smax.append(float(f[1]))
            except ValueError:
                continue
            for nm, v in zip(names, f[3:7]):
                if v.lower() == "active":
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def algorithmic_bytes(a, R, sweeps, refresh, accepted):
    """Bytes one launch of the lockstep residual sweep must move: the residual
    form's per-sweep figure with a replica tile of 16 branches (one stream
    of the bit->ray CSR -- ray id + a', 8 B per entry -- serves 16 branches),
    each branch's compensated residuals (hi + lo, s_r = 8 B) read and written
    once per sweep (rays x 2 x 8 B), its bits read and written (2 x 1/8 B
    each), the prior's neighbour lists once per tile (4 B per entry), plus
    every accepted flip's residual read-modify-write (entries of the bit x 2
    x 8 B, from the device's accept count, at the mean entries per bit) and
    the fp64 refreshes (ray-major CSR, 8 B per entry, once per tile)."""
    nnz = int(a["ray"].size)
    n = int(a["row_ptr"].size - 1)
    rays = int(a["d"].size)
    nbr = int(a["nbr"].size)
    tiles = (R + 15) // 16
    per_sweep = nnz * 8 * tiles + R * (rays * 2 * 8 + n * 2 / 8) + nbr * 4 * tiles
    refreshes = (sweeps - 1) // refresh if refresh > 0 else 0
    return per_sweep * sweeps + refreshes * tiles * nnz * 8 + accepted * (nnz / n) * 2 * 8


def cpu_baseline(a, sched, threads, branches):
    """The reference's branch_fractions (oracle/_ref) on a bounded sample."""
    from oracle import oracle as O
    n = int(a["row_ptr"].size - 1)
    if O.ref_available():
        rp = O.RefProblem(a)
        _, _, wall = rp.branch_fractions(sched.t_hot, sched.t_cold, sched.anneal_sweeps, sched.hold_sweeps,
                                         branches, threads, 0, keep=False)
        kind = "reference"
    else:
        from concurrent.futures import ThreadPoolExecutor
        t0 = time.perf_counter()
        with ThreadPoolExecutor(threads) as ex:
            list(ex.map(lambda b: O.anneal_branch(a, sched.t_hot, sched.t_cold, sched.anneal_sweeps,
                                                  sched.hold_sweeps, b + 1), range(branches)))
        wall = time.perf_counter() - t0
        kind = "port"
    attempts = branches * (sched.anneal_sweeps + sched.hold_sweeps) * n
    return attempts / wall, wall, kind


class _Sched:
    """A schedule's four numbers (the reference arm imports nothing of the solver)."""

    def __init__(self, t_hot, t_cold, anneal_sweeps, hold_sweeps, refresh_sweeps=50):
        self.t_hot, self.t_cold = t_hot, t_cold
        self.anneal_sweeps, self.hold_sweeps, self.refresh_sweeps = anneal_sweeps, hold_sweeps, refresh_sweeps

    @property
    def sweeps(self):
        return self.anneal_sweeps + self.hold_sweeps


POSTERIOR = _Sched(50.0, 1.0, 200, 50, 50)   # ising_recon.hpp:81-86


def workload_config(a, sweeps, gpus):
    """The workload's identity, the same in both arms' lines."""
    return {"workload": WORKLOAD, "bits": int(a["row_ptr"].size - 1), "rays": int(a["d"].size),
            "entries": int(a["ray"].size), "branches": BRANCHES, "sweeps": sweeps,
            "schedule": "T 50 -> 1 geometric over 200 sweeps, then 50 sweeps at T = 1",
            "parallelism": f"{gpus} independent replica{'' if gpus == 1 else 's'} (one per GPU)",
            "l2": "GPU arm: flushed (256 MB write) before every timed step"}


def run_reference(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return 0
    from oracle import oracle as O
    a = O.tomography()   # the pyramid from oracle/libqb_inputs.so: the solver library is not loaded
    threads = os.cpu_count() or 1
    # each step: the reference's branch_fractions on the full 306,328-bit
    # problem with the full posterior schedule; min(16, cores) branches
    branches = min(BRANCHES, threads)
    rates, walls = [], []
    kind = None
    for k in range(args.warmup + args.steps):
        rate, wall, kind = cpu_baseline(a, POSTERIOR, threads, branches)
        if k >= args.warmup:
            rates.append(rate)
            walls.append(wall)
    value = statistics.mean(rates)
    n = int(a["row_ptr"].size - 1)
    ms = BRANCHES * POSTERIOR.sweeps * n / value * 1e3
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "attempts/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": workload_config(a, POSTERIOR.sweeps, args.gpus),
            "cpu_baseline": {"value": value, "unit": "attempts/s", "cores": threads, "kind": kind,
                             "sample": f"{branches} of the 16 branches per step (branch_fractions), the full "
                                       f"250-sweep schedule on the full problem, {threads} threads, "
                                       f"{statistics.mean(walls):.1f} s per step"},
            "e2e": {"value": value, "unit": "attempts/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


# ---- batch: many Max-Cut instances in one persistent launch ----------------------------------

BATCH_WORKLOAD = ("4096 Max-Cut instances, N log-uniform 200..20,000, alternately 2D +-1 tori and random "
                  "d-regular graphs (d 3..50, +-1), 32 replicas each, 2000 sweeps (scaled schedule sigma -> "
                  "0.1 w_min), one persistent launch")


def _spawn_map(fn, items, procs=None):
    """Builds inputs in spawned processes (before any CUDA call of this one)."""
    import multiprocessing as mp
    procs = procs or min(32, os.cpu_count() or 1)
    with mp.get_context("spawn").Pool(procs) as pool:
        return pool.map(fn, items, chunksize=max(1, len(items) // (4 * procs)))


def _create_all(make, items, threads=16):
    from concurrent.futures import ThreadPoolExecutor
    with ThreadPoolExecutor(threads) as ex:   # planning runs in the library, outside the GIL
        return list(ex.map(make, items))


def batch_algorithmic_bytes(probs, R, sweeps, G):
    """Bytes per launch by the Ising formula: the CSR (4 B column + weight
    bytes per directed entry) streamed once per replica group of G per sweep,
    every replica's state (int32 field + int8 spin) read and written once per
    sweep. Accepted flips' field updates are not counted (a lower bound)."""
    b = 0.0
    for P in probs:
        i = P.info()
        b += sweeps * (i.nnz * (4 + i.weight_bytes) * ((R + G - 1) // G) + R * i.n * (2 * 4 + 2 * 1))
    return b


def run_batch(args):
    from qublar_b200 import synth
    specs = synth.mixed_batch_specs(args.instances)
    t0 = time.perf_counter()
    graphs = _spawn_map(synth.build_spec, specs)
    log(f"[batch] built {len(graphs)} instances in {time.perf_counter() - t0:.1f} s")
    import torch

    from qublar_b200 import IsingProblem, autotune_batch, solve_batch
    torch.cuda.set_device(int(os.environ.get("LOCAL_RANK", "0")))
    stream = torch.cuda.current_stream()
    R, S = 32, args.batch_sweeps
    t0 = time.perf_counter()
    probs = _create_all(lambda g: IsingProblem(*g), graphs)
    log(f"[batch] planned and uploaded in {time.perf_counter() - t0:.1f} s")
    items = [(P, P.scaled_schedule(S, 0), R, 0) for P in probs]
    attempts = sum(R * S * P.n for P in probs)
    if args.shape:
        from qublar_b200._abi import BatchConfig
        t_, s_, g_ = (int(v) for v in args.shape.split(","))
        cfg = BatchConfig(t_, s_, g_, 0)
    else:
        cfg = autotune_batch(items, 8)
    log(f"[batch] shape: {cfg.threads} threads, {cfg.smem_bytes} B, groups of {cfg.max_group}")
    for _ in range(args.warmup):
        B = solve_batch(items, cfg, stream=stream)
        B.info()
        B.close()
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    sampler = ClockSampler(int(os.environ.get("LOCAL_RANK", "0")))
    torch.cuda.synchronize()
    sampler.start()
    infos = []
    for _ in range(args.steps):
        flush.zero_()
        B = solve_batch(items, cfg, stream=stream)
        infos.append(B.info())
        B.close()
    clocks = sampler.stop()
    total_ms = statistics.mean(i.total_ms for i in infos)
    anneal_ms = statistics.mean(i.anneal_ms for i in infos)
    value = attempts / (total_ms / 1e3)
    if args.kernel_only:
        print(json.dumps({"metric": METRIC, "value": value, "unit": "attempts/s", "kernel_ms": anneal_ms,
                          "config": {"instances": len(probs), "sweeps": S, "work_items": infos[0].work_items}}))
        return 0
    # plain form: one qb_solve per instance, on a size-stratified sample
    order = sorted(range(len(probs)), key=lambda k: probs[k].n)
    sample = [order[int(j)] for j in np.linspace(0, len(order) - 1, min(64, len(order)))]
    p_att, p_ms = 0, 0.0
    for k in sample:
        P, sch, _, _ = items[k]
        r = P.solve(sch, R, stream=stream)
        inf = r.info()
        p_att += inf.attempts
        p_ms += inf.total_ms
        r.close()
    plain = p_att / (p_ms / 1e3)
    # end to end: host graphs -> plan + upload -> packed solve -> every instance's fractions on the host
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    probs2 = _create_all(lambda g: IsingProblem(*g), graphs)
    items2 = [(P, P.scaled_schedule(S, 0), R, 0) for P in probs2]
    B = solve_batch(items2, cfg, stream=stream)
    d2h = 0
    for k in range(len(items2)):
        d2h += B.marginals(k).nbytes
    e2e_s = time.perf_counter() - t0
    B.close()
    h2d = sum(g[1].nbytes * 3 for g in graphs)
    hbm, peak_kind = peaks()
    alg = batch_algorithmic_bytes(probs, R, S, cfg.max_group)
    achieved = alg / (anneal_ms / 1e3) / 1e9
    line = {
        "metric": METRIC, "value": value, "unit": "attempts/s", "n_gpus": 1, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": total_ms, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "int32", "data": "synthetic",
        "config": {"workload": BATCH_WORKLOAD, "instances": len(probs), "bits": int(sum(P.n for P in probs)),
                   "replicas": R, "sweeps": S, "shape": {"threads": cfg.threads, "smem_bytes": cfg.smem_bytes,
                                                         "max_group": cfg.max_group},
                   "work_items": infos[0].work_items, "global_items": infos[0].global_items,
                   "l2": "flushed (256 MB write) before every timed step", "parallelism": "1 GPU"},
        "plain": {"value": plain, "unit": "attempts/s", "form": "one qb_solve per instance",
                  "sample": f"{len(sample)} instances stratified by size"},
        "vs_plain": value / plain,
        "e2e": {"value": attempts / e2e_s, "unit": "attempts/s", "h2d_bytes_per_step": int(h2d),
                "d2h_bytes_per_step": int(d2h), "s_per_step": e2e_s},
        "gpu_launches": sum(i.launches for i in infos),
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": hbm, "unit": "GB/s", "frac": achieved / hbm,
                     "peak_kind": peak_kind, "traffic": None, "kernel": "ising_word_kernel",
                     "kernel_ms": anneal_ms, "algorithmic_bytes": alg,
                     "note": "CSR and state stay in L2 and shared memory; the sweep is issue-bound (Philox, "
                             "neighbour counts), not DRAM-bound"},
        "clocks": clocks,
    }
    if not args.no_cpu_baseline:
        line["cpu_baseline"] = batch_cpu_baseline(graphs, items, R, S)
    print(json.dumps(line), flush=True)
    return 0


def batch_cpu_baseline(graphs, items, R, S):
    """The reference's wising::anneal (oracle/_ref) on the host's cores: the
    instances nearest the mean size, all R replicas, the full schedule, until
    about 1e9 attempts."""
    from oracle import oracle as O
    threads = os.cpu_count() or 1
    mean_n = statistics.mean(g[0] for g in graphs)
    order = sorted(range(len(graphs)), key=lambda k: abs(graphs[k][0] - mean_n))
    att, wall, used = 0, 0.0, 0
    for k in order:
        n, eu, ev, ew = graphs[k]
        sch = items[k][1]
        if O.ref_available():
            g = O.RefGraph(O.Graph(n, eu, ev, ew).rudy())
            _, _, w = g.anneal_many(sch.t_hot, sch.t_cold, sch.anneal_sweeps, sch.hold_sweeps, 1, R, threads)
            kind = "reference"
        else:
            g = O.Graph(n, eu, ev, ew)
            t0 = time.perf_counter()
            for r in range(R):
                g.wising_anneal(sch.t_hot, sch.t_cold, sch.anneal_sweeps, sch.hold_sweeps, r + 1)
            w = time.perf_counter() - t0
            kind = "port"
        att += R * S * n
        wall += w
        used += 1
        if att >= 1e9:
            break
    return {"value": att / wall, "unit": "attempts/s", "cores": threads, "kind": kind,
            "sample": f"{used} instances near the mean size (N ~ {mean_n:.0f}), {R} replicas, {S} sweeps, "
                      f"{threads} threads, {wall:.1f} s"}


# ---- serve: a Poisson request stream through the serving loop -----------------------------------

SERVE_LOCKSTEP_BITS = int(os.environ.get("QB_SERVE_LOCKSTEP_BITS", "10000"))
SERVE_QUBO_MAXCUT_BITS = 50000
SERVE_WORKLOAD = ("Poisson request stream: N log-uniform 1,000..300,000, half tomography-style pyramids, half "
                  "sparse +-1 Max-Cut (d-regular, d 3..12), sweeps 500..5000, branches 8..32")


def _serve_schedule(spec, P, data):
    from qublar_b200 import Budget, Schedule
    S = spec["sweeps"]
    if spec["kind"] == "tomography":
        hold = S // 5
        return Schedule(50.0, 1.0, S - hold, hold, 50)
    if hasattr(P, "scaled_schedule"):
        return P.scaled_schedule(S, 0)
    # a Max-Cut graph served as the equal QUBO: the integer form's scaled
    # schedule (T_hot = sqrt(2 sum w^2 / n), T_cold = w_min / 10)
    n, _, _, ew = data
    a = np.abs(np.asarray(ew, np.float64))
    nz = a[a > 0]
    return Budget(float(np.sqrt(2.0 * np.sum(a * a) / n)), 0.1 * float(nz.min() if nz.size else 0.0), S, 0, 0)


def _serve_path(P, spec):
    if spec["kind"] != "tomography":
        return "maxcut partitioned qubo" if spec["n"] >= SERVE_QUBO_MAXCUT_BITS else "maxcut ticks"
    return "pyramid partitioned lockstep" if P.info().variant == 1 else "pyramid cluster"


def _serve_run(probs, specs, scheds, rate, seed):
    """Submits the stream (all at once when rate is None, else Poisson at
    `rate` requests/s) to a fresh server; returns per-request latencies,
    the makespan and the server's stats."""
    from qublar_b200 import Server
    S = Server()
    rng = np.random.default_rng(seed)
    gaps = np.zeros(len(probs)) if rate is None else rng.exponential(1.0 / rate, len(probs))
    t0 = time.perf_counter()
    due = t0
    ids = []
    for k, P in enumerate(probs):
        due += gaps[k]
        dt = due - time.perf_counter()
        if dt > 0:
            time.sleep(dt)
        ids.append(S.submit(P, scheds[k], specs[k]["branches"], k))
    for i in ids:
        S.wait(i, -1)
    infos = [S.info(i) for i in ids]
    first = min(i.t_submit for i in infos)
    last = max(i.t_done for i in infos)
    lat = np.array([i.t_done - i.t_submit for i in infos])
    stats = S.stats()
    # where the time went: service (admission to done) and queueing, by path
    paths = {}
    for P, sp, inf in zip(probs, specs, infos):
        d = paths.setdefault(_serve_path(P, sp), {"requests": 0, "attempts": 0.0, "service_s": 0.0, "queue_s": 0.0})
        d["requests"] += 1
        d["attempts"] += float(inf.attempts)
        d["service_s"] += inf.t_done - inf.t_admit
        d["queue_s"] += inf.t_admit - inf.t_submit
    out = {"ids": ids, "server": S, "lat": lat, "makespan": last - first, "ticks": stats.ticks,
           "peak_bytes": stats.peak_bytes, "paths": paths}
    return out


def serve_measure(n_requests, rates=(0.5, 0.8), plain_sample=24, warm=3):
    """The serving stream of n_requests through a fresh server, saturated
    (everything submitted at once) and at Poisson rates that are fractions of
    the measured capacity; the plain form (each request alone through
    qb_solve) on a sample of plain_sample requests (all of them when 0 or more
    than the stream); the served results against the plain ones."""
    from qublar_b200 import synth
    specs = synth.serve_specs(n_requests)
    t0 = time.perf_counter()
    data = _spawn_map(synth.build_request, specs)
    log(f"[serve] built {len(data)} requests in {time.perf_counter() - t0:.1f} s")
    import torch

    from qublar_b200 import (OPT_DEFER_UPLOAD, OPT_RESID_CLUSTER, IsingProblem, QuboProblem, ResidualProblem)
    torch.cuda.set_device(int(os.environ.get("LOCAL_RANK", "0")))

    def make(k, served=True):
        # pyramids of SERVE_LOCKSTEP_BITS and more take the lockstep sweep on
        # one partition of the device (several side by side); smaller ones one
        # cluster per branch beside the rest. Max-Cut graphs of 50,000 bits and
        # more run as the equal weighted QUBO on a partition (identical
        # branches); smaller ones in ticks. The plain form (served=False) is
        # the same problem solved alone; its pyramids always take the lockstep
        # sweep, qb_solve's default plan.
        sp = specs[k]
        fl = OPT_DEFER_UPLOAD if served else 0
        if sp["kind"] == "tomography":
            if served and sp["n"] < SERVE_LOCKSTEP_BITS:
                fl |= OPT_RESID_CLUSTER
            return ResidualProblem.from_arrays(data[k], flags=fl)
        if sp["n"] >= SERVE_QUBO_MAXCUT_BITS:
            return QuboProblem.from_dict(synth.maxcut_qubo(*data[k]), flags=fl)
        return IsingProblem(*data[k], flags=fl)

    t0 = time.perf_counter()
    probs = _create_all(make, range(len(specs)))
    log(f"[serve] planned in {time.perf_counter() - t0:.1f} s")
    scheds = [_serve_schedule(sp, P, data[k]) for k, (sp, P) in enumerate(zip(specs, probs))]
    attempts = [sp["branches"] * sch.sweeps * P.n for sp, sch, P in zip(specs, scheds, probs)]
    total = float(sum(attempts))
    # warm-up: a few small requests through a server
    small = sorted(range(len(probs)), key=lambda k: attempts[k])[:max(3, warm)]
    w = _serve_run([probs[k] for k in small], [specs[k] for k in small], [scheds[k] for k in small], None, 0)
    w["server"].close()
    sampler = ClockSampler(int(os.environ.get("LOCAL_RANK", "0")))
    sampler.start()
    sat = _serve_run(probs, specs, scheds, None, 1)
    clocks = sampler.stop()
    value = total / sat["makespan"]
    # served results against the plain solve of the same problem (sampled)
    mu = len(probs) / sat["makespan"]
    S = sat["server"]
    n_plain = len(probs) if plain_sample <= 0 else min(plain_sample, len(probs))
    sample = [int(j) for j in np.linspace(0, len(probs) - 1, n_plain)]
    same = 0
    e_rel = []
    p_att, p_s = 0.0, 0.0
    for k in sample:
        x_served = S.branches(sat["ids"][k])
        e_served = S.energies(sat["ids"][k])
        Q = make(k, served=False)
        r = Q.solve(scheds[k], specs[k]["branches"], k)
        inf = r.info()
        p_att += inf.attempts
        p_s += inf.total_ms / 1e3
        x_plain = r.branches()
        e_plain = r.energies()
        if specs[k]["kind"] != "tomography" or probs[k].info().variant == 1:
            same += int((x_plain == x_served).all())   # the same sweep: identical branches
        else:
            same += 1 if abs(e_plain.mean() - e_served.mean()) <= 0.05 * abs(e_plain.mean()) + 1e-9 else 0
        e_rel.append(float((e_served.mean() - e_plain.mean()) / max(1e-12, abs(e_plain.mean()))))
        r.close()
        Q.close()
    plain = p_att / p_s
    S.close()
    lat_sat = sat["lat"]
    at_rates = {}
    for frac in rates:
        run = _serve_run(probs, specs, scheds, frac * mu, 2)
        at_rates[f"{frac:.1f}x capacity"] = {"rate_per_s": frac * mu, "p50_s": float(np.percentile(run["lat"], 50)),
                                             "p99_s": float(np.percentile(run["lat"], 99)),
                                             "throughput": total / run["makespan"]}
        run["server"].close()
    return {"requests": len(probs), "total_attempts": total, "value": value, "makespan_s": sat["makespan"],
            "warm": len(small), "plain": plain, "plain_sample": len(sample), "vs_plain": value / plain,
            "latency": {"saturated": {"p50_s": float(np.percentile(lat_sat, 50)),
                                      "p99_s": float(np.percentile(lat_sat, 99))}, **at_rates},
            "equal_energy": {"checked": len(sample), "agree": same,
                             "mean_rel_energy_diff": float(np.mean(e_rel)) if e_rel else None,
                             "rule": "Max-Cut and lockstep pyramids: identical branches; cluster pyramids: mean "
                                     "energy within 5% (cluster vs lockstep summation order)"},
            "ticks": sat["ticks"], "peak_bytes": sat["peak_bytes"], "paths_saturated": sat["paths"],
            "clocks": clocks}


SERVE_POLICY = (f"pyramids >= {SERVE_LOCKSTEP_BITS} bits: lockstep sweep on one of 4 SM partitions, side by side; "
                "smaller pyramids: one CTA or cluster per branch; Max-Cut >= "
                f"{SERVE_QUBO_MAXCUT_BITS} bits: the equal weighted QUBO on a partition; smaller Max-Cut: ticks of "
                "word units")


def run_serve(args):
    m = serve_measure(args.requests)
    hbm, peak_kind = peaks()
    line = {
        "metric": "spin-flip attempts/s; p50/p99 solve latency at equal energy, served vs plain", "value": m["value"],
        "unit": "attempts/s", "n_gpus": 1, "steps": 1, "warmup": m["warm"], "ms_per_step": m["makespan_s"] * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "mixed (int32 / f32)",
        "data": "synthetic",
        "config": {"workload": SERVE_WORKLOAD, "requests": m["requests"], "total_attempts": m["total_attempts"],
                   "policy": SERVE_POLICY, "budget": "150 GB (capped at 90% of free memory)", "parallelism": "1 GPU"},
        "latency": m["latency"],
        "plain": {"value": m["plain"], "unit": "attempts/s",
                  "form": "each request alone through qb_solve (lockstep sweep for pyramids, the whole-device "
                          f"QUBO sweep for Max-Cut >= {SERVE_QUBO_MAXCUT_BITS} bits, its own sweep below)",
                  "sample": f"{m['plain_sample']} requests"},
        "vs_plain": m["vs_plain"],
        "equal_energy": m["equal_energy"],
        "e2e": {"value": m["value"], "unit": "attempts/s", "h2d_bytes_per_step": None, "d2h_bytes_per_step": None,
                "note": "requests enter as host problems (deferred upload) and the server uploads them at "
                        "admission inside the timed makespan"},
        "server": {"ticks": m["ticks"], "peak_bytes": m["peak_bytes"], "paths_saturated": m["paths_saturated"]},
        "peak_hbm_gbs": hbm, "peak_kind": peak_kind,
        "clocks": m["clocks"],
    }
    print(json.dumps(line), flush=True)
    return 0


# ---- qubo: the weighted fp32 lattice QUBO --------------------------------------------------------

# DRAM bytes (read + write) per sweep of qubo_lockstep_kernel from the
# committed ncu capture of a 100-sweep launch on the same 200,000-bit QUBO with
# 64 replicas (profiles/qubo_lockstep_lattice.md): the replicas' compensated
# fields stream once per sweep, so a full launch moves this times its sweeps.
QUBO_NCU_TRAFFIC_PER_SWEEP = (13.313979e9 + 10.124942e9) / 100
QUBO_WORKLOAD = ("weighted QUBO on a 58^3 periodic lattice + 4,888 extra sites with random long-range edges "
                 "(N = 200,000, average degree 20), J and h ~ N(0,1) fp32, 64 replicas, 5000 sweeps T 3 -> 0.05, "
                 "compensated fp32 fields with an fp64 refresh every 64 sweeps")


def qubo_algorithmic_bytes(info, n, m, R, sweeps, refresh, accepted):
    """Bytes per launch by the weighted formula: the CSR (4 B column + 4 B
    coupling per directed entry) once per sweep for all 64 replicas, every
    replica's compensated field (8 B) read and written and its bit words once
    per sweep, each accepted flip's delta applied to its neighbours' fields
    (d x 2 x 8 B), and the fp64 refreshes' extra CSR pass."""
    nnz = 2 * m
    d = nnz / n
    tiles = (R + 63) // 64
    per_sweep = nnz * 8 * tiles + R * n * (2 * 8 + 2 / 8)
    refreshes = (sweeps - 1) // refresh if refresh > 0 else 0
    return per_sweep * sweeps + accepted * d * 2 * 8 + refreshes * nnz * 8 * tiles


def run_qubo(args):
    from qublar_b200 import synth
    t0 = time.perf_counter()
    q = synth.lattice_qubo()
    log(f"[qubo] built in {time.perf_counter() - t0:.1f} s")
    import torch

    from qublar_b200 import QuboProblem, Schedule
    torch.cuda.set_device(int(os.environ.get("LOCAL_RANK", "0")))
    stream = torch.cuda.current_stream()
    R, S = 64, args.qubo_sweeps
    sched = Schedule(3.0, 0.05, S - S // 10, S // 10, 64)
    P = QuboProblem.from_dict(q, stream=stream)
    n, m = int(q["n"]), int(q["eu"].size)
    attempts = R * S * n
    for _ in range(args.warmup):
        r = P.solve(sched, R, stream=stream)
        r.info()
        r.close()
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    sampler = ClockSampler(int(os.environ.get("LOCAL_RANK", "0")))
    torch.cuda.synchronize()
    sampler.start()
    infos, energies = [], []
    for _ in range(args.steps):
        flush.zero_()
        r = P.solve(sched, R, stream=stream)
        infos.append(r.info())
        energies.append(r.energies())
        r.close()
    clocks = sampler.stop()
    total_ms = statistics.mean(i.total_ms for i in infos)
    anneal_ms = statistics.mean(i.anneal_ms for i in infos)
    value = attempts / (total_ms / 1e3)
    if args.kernel_only:
        print(json.dumps({"metric": METRIC, "value": value, "unit": "attempts/s", "kernel_ms": anneal_ms,
                          "config": {"bits": n, "replicas": R, "sweeps": S}}))
        return 0
    # end to end: host arrays -> plan + upload -> solve -> fractions back
    torch.cuda.synchronize()
    e2e = []
    e2e_warm = min(args.warmup, 3)   # untimed, like the timed region's warm-up (first-use mappings, module loads)
    for k in range(e2e_warm + max(1, args.e2e_steps)):
        t0 = time.perf_counter()
        Q = QuboProblem.from_dict(q, stream=stream)
        r = Q.solve(sched, R, stream=stream)
        p = r.marginals()
        if k >= e2e_warm:
            e2e.append(time.perf_counter() - t0)
        r.close()
        Q.close()
    h2d = int(q["eu"].nbytes + q["ev"].nbytes + q["ew"].nbytes + q["h"].nbytes)
    hbm, peak_kind = peaks()
    acc = statistics.mean(i.accepted for i in infos)
    alg = qubo_algorithmic_bytes(infos[0], n, m, R, S, sched.refresh_sweeps, acc)
    achieved = alg / (anneal_ms / 1e3) / 1e9
    line = {
        "metric": METRIC, "value": value, "unit": "attempts/s", "n_gpus": 1, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": total_ms, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32 (compensated) + f64 refresh", "data": "synthetic",
        "config": {"workload": QUBO_WORKLOAD, "bits": n, "edges": m, "replicas": R, "sweeps": S,
                   "colours": int(P.info().n_colours), "refresh_sweeps": sched.refresh_sweeps,
                   "l2": "flushed (256 MB write) before every timed step; state 106 MB", "parallelism": "1 GPU"},
        "precision": {"max_field_drift": max(i.max_drift for i in infos),
                      "max_energy_error": max(i.max_energy_error for i in infos),
                      "mean_final_energy": float(np.mean(energies[-1])),
                      "note": "drift: |compensated fp32 field - fp64 field| at refreshes; energy error: |offset + "
                              "sum of accepted fp32 dE - fp64 energy from scratch|"},
        "e2e": {"value": attempts / statistics.mean(e2e), "unit": "attempts/s", "h2d_bytes_per_step": h2d,
                "d2h_bytes_per_step": n * 4, "s_per_step": statistics.mean(e2e), "warmup_steps": e2e_warm},
        "gpu_launches": sum(i.launches for i in infos),
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": hbm, "unit": "GB/s", "frac": achieved / hbm,
                     "peak_kind": peak_kind, "traffic": QUBO_NCU_TRAFFIC_PER_SWEEP * S, "kernel": "qubo_lockstep_kernel",
                     "kernel_ms": anneal_ms, "algorithmic_bytes": alg, "accepted_flips": acc},
        "clocks": clocks,
    }
    if not args.no_cpu_baseline:
        line["cpu_baseline"] = qubo_cpu_baseline(q, sched)
    print(json.dumps(line), flush=True)
    return 0


def qubo_cpu_baseline(q, sched):
    """The reference's anneal_branch on the pair-ray encoding of the same
    QUBO (check_ree_qubo.cu:172-192, oracle/_ref) on the host's cores: 16
    branches of a 40-sweep sample of the schedule (one ray per coupling)."""
    from concurrent.futures import ThreadPoolExecutor

    from oracle import oracle as O
    from qublar_b200 import synth
    threads = os.cpu_count() or 1
    arr = synth.qubo_pair_ray(q)
    n = int(q["n"])
    hold = 4
    branches = min(16, threads)
    if O.ref_available():
        rp = O.RefProblem(arr)
        _, _, wall = rp.branch_fractions(sched.t_hot, sched.t_cold, 40 - hold, hold, branches, threads, 0, keep=False)
        kind = "reference"
    else:
        t0 = time.perf_counter()
        with ThreadPoolExecutor(threads) as ex:
            list(ex.map(lambda b: O.anneal_branch(arr, sched.t_hot, sched.t_cold, 40 - hold, hold, b + 1),
                        range(branches)))
        wall = time.perf_counter() - t0
        kind = "port"
    return {"value": branches * 40 * n / wall, "unit": "attempts/s", "cores": threads, "kind": kind,
            "sample": f"{branches} branches x 40 sweeps of the pair-ray encoding (one ray per coupling), "
                      f"{threads} threads, {wall:.1f} s"}


# ---- maxcut: the 800-node Erdos-Renyi graph ------------------------------------------------------

def run_maxcut(args):
    import torch

    from qublar_b200 import Budget, IsingProblem, synth
    torch.cuda.set_device(int(os.environ.get("LOCAL_RANK", "0")))
    stream = torch.cuda.current_stream()
    n, eu, ev, ew = synth.erdos_renyi(800, 0.06, 1)
    R, S = 16, 1000
    sched = Budget(3.0, 0.05, S, 0, 0)
    P = IsingProblem(n, eu, ev, ew, stream=stream)
    for _ in range(args.warmup):
        P.solve(sched, R, stream=stream).info()
    infos, cuts = [], []
    for _ in range(args.steps):
        r = P.solve(sched, R, stream=stream)
        infos.append(r.info())
        cuts.append(-r.energies_tracked())
        r.close()
    total_ms = statistics.mean(i.total_ms for i in infos)
    value = R * S * n / (total_ms / 1e3)
    line = {"metric": METRIC, "value": value, "unit": "attempts/s", "n_gpus": 1, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": total_ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "int32", "data": "synthetic",
            "config": {"workload": "Max-Cut on ER(800, 0.06), w = +1, 16 replicas, 1000 sweeps T 3 -> 0.05",
                       "edges": int(eu.size), "parallelism": "1 GPU"},
            "best_cut": int(max(c.max() for c in cuts)), "mean_cut": float(np.mean(cuts[-1])),
            "gpu_launches": sum(i.launches for i in infos)}
    if not args.no_cpu_baseline:
        from oracle import oracle as O
        threads = os.cpu_count() or 1
        if O.ref_available():
            g = O.RefGraph(O.Graph(n, eu, ev, ew).rudy())
            _, _, wall = g.anneal_many(3.0, 0.05, S, 0, 1, R, threads)
            line["cpu_baseline"] = {"value": R * S * n / wall, "unit": "attempts/s", "cores": threads,
                                    "kind": "reference", "sample": f"all {R} replicas, {threads} threads"}
    print(json.dumps(line), flush=True)
    return 0


SIDE_KEYS = ("value", "unit", "steps", "warmup", "ms_per_step", "dtype", "plain", "vs_plain", "e2e", "gpu_launches",
             "roofline", "precision", "clocks")


def side_workload(argv, timeout_s=900):
    """One of the other benchmark workloads (its own ``--workload`` line), run
    as a child process after the pyramid line is measured, so that the default
    run records it too: a failure there is reported in its block and touches
    nothing else. Returns the child's figures, or {"error": ...}."""
    env = {k: v for k, v in os.environ.items()
           if k not in ("RANK", "WORLD_SIZE", "MASTER_ADDR", "MASTER_PORT", "GROUP_RANK", "ROLE_RANK",
                        "LOCAL_WORLD_SIZE") and not k.startswith("TORCHELASTIC")}
    cmd = [sys.executable, os.path.abspath(__file__)] + list(argv)
    t0 = time.perf_counter()
    try:
        r = subprocess.run(cmd, env=env, stdout=subprocess.PIPE, stderr=subprocess.PIPE, timeout=timeout_s,
                           text=True)
    except subprocess.TimeoutExpired:
        return {"command": "bench.py " + " ".join(argv), "error": f"no line within {timeout_s} s"}
    wall = time.perf_counter() - t0
    got = None
    for ln in reversed(r.stdout.splitlines()):
        if ln.startswith("{"):
            try:
                got = json.loads(ln)
                break
            except ValueError:
                pass
    if r.returncode != 0 or got is None:
        tail = (r.stderr.strip().splitlines() or ["(no output)"])[-1]
        return {"command": "bench.py " + " ".join(argv), "error": f"exit {r.returncode}: {tail[:300]}"}
    out = {"command": "bench.py " + " ".join(argv), "wall_s": round(wall, 1)}
    out.update({k: got[k] for k in SIDE_KEYS if k in got})
    cfg = got.get("config", {})
    out["config"] = {k: cfg[k] for k in ("workload", "shape", "l2") if k in cfg}
    return out


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--e2e-steps", type=int, default=3)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--sweeps", type=int, default=250,
                    help="schedule length (default 250 = 200 + 50, the benchmark); shorter runs are for profiling only")
    ap.add_argument("--workload", default="tomography", choices=["tomography", "batch", "serve", "qubo", "maxcut"],
                    help="tomography: the pyramid (default); batch: many Max-Cut instances in one persistent "
                         "launch; serve: a Poisson request stream through the serving loop; qubo: the weighted "
                         "fp32 lattice QUBO; maxcut: the 800-node ER graph")
    ap.add_argument("--instances", type=int, default=4096, help="batch: instances")
    ap.add_argument("--batch-sweeps", type=int, default=2000, help="batch: sweeps per instance")
    ap.add_argument("--requests", type=int, default=160, help="serve: requests in the stream")
    ap.add_argument("--serve-requests", type=int, default=24,
                    help="tomography: also measure served vs plain on a stream of this many requests (0 = skip)")
    ap.add_argument("--shape", default=None,
                    help="batch: fixed packed-kernel shape 'threads,smem_bytes,max_group' instead of autotuning")
    ap.add_argument("--qubo-sweeps", type=int, default=5000, help="qubo: sweeps (shorter runs are for profiling)")
    ap.add_argument("--kernel-only", action="store_true",
                    help="batch/qubo: time the kernel only (no plain-form, end-to-end or CPU legs; for profiling)")
    ap.add_argument("--no-side-workloads", action="store_true",
                    help="tomography: skip the batched (C3) and weighted-QUBO (C4) lines recorded beside the pyramid")
    args = ap.parse_args()
    if args.workload == "batch":
        return run_batch(args)
    if args.workload == "serve":
        return run_serve(args)
    if args.workload == "qubo":
        return run_qubo(args)
    if args.workload == "maxcut":
        return run_maxcut(args)
    if args.impl == "reference":
        return run_reference(args)

    import torch
    import torch.distributed as dist

    from qublar_b200 import ResidualProblem, Schedule, synth

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    if world > 1:
        import datetime
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300), device_id=torch.device("cuda", local))

    def barrier():
        if world > 1:
            dist.barrier()

    def max_over_ranks(v):
        if world == 1:
            return v
        t = torch.tensor([v], dtype=torch.float64, device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item())

    stream = torch.cuda.current_stream()
    a = synth.tomography()
    n = int(a["row_ptr"].size - 1)
    sched = Schedule()   # 50 -> 1, 200 + 50, refresh 50 (POSTERIOR)
    if args.sweeps != 250:
        hold = args.sweeps // 5
        sched = Schedule(50.0, 1.0, args.sweeps - hold, hold, 50)
    P = ResidualProblem.from_arrays(a, device=local, stream=stream)
    pinfo = P.info()
    attempts_step = BRANCHES * sched.sweeps * n
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")

    energy_err = None   # the last warm-up solve is traced: E(0) + accepted fp32 dE against the fp64 energy
    for k in range(args.warmup):
        r = P.solve(sched, BRANCHES, stream=stream, trace=k == args.warmup - 1)
        energy_err = r.info().max_energy_error
        r.close()

    sampler = ClockSampler(local) if rank == 0 else None
    barrier()
    torch.cuda.synchronize()
    if sampler:
        sampler.start()
    starts = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    ends = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    results = []
    for k in range(args.steps):
        flush.zero_()
        starts[k].record(stream)
        results.append(P.solve(sched, BRANCHES, stream=stream))
        ends[k].record(stream)
    torch.cuda.synchronize()
    barrier()
    clocks = sampler.stop() if sampler else None
    total_ms = sum(s.elapsed_time(e) for s, e in zip(starts, ends))
    infos = [r.info() for r in results]
    anneal_ms = statistics.mean(i.anneal_ms for i in infos)
    accepted = statistics.mean(i.accepted for i in infos)
    launches = sum(i.launches for i in infos)
    drift = max(i.max_drift for i in infos)
    for r in results:
        r.close()
    total_ms = max_over_ranks(total_ms)
    value = world * attempts_step * args.steps / (total_ms / 1e3)

    # e2e through the C ABI from pinned host memory
    pinned = {}
    for k, v in a.items():
        if isinstance(v, np.ndarray):
            t = torch.empty(v.shape, dtype=getattr(torch, str(v.dtype)), pin_memory=True)
            t.numpy()[...] = v
            pinned[k] = t.numpy()
        else:
            pinned[k] = v
    h2d = sum(v.nbytes for v in pinned.values() if isinstance(v, np.ndarray))
    d2h = n * 4
    e2e_s = [float("nan")]
    if args.e2e_steps > 0:
        e2e_s = []
    barrier()
    # untimed warm-up steps first, as for the timed region: a process's first
    # creates pay one-time costs (module loads, fresh device-memory mappings)
    e2e_warm = min(args.warmup, 3) if args.e2e_steps > 0 else 0
    for k in range(e2e_warm + args.e2e_steps):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        Q = ResidualProblem.from_arrays(pinned, device=local, stream=stream)
        r = Q.solve(sched, BRANCHES, stream=stream)
        p = r.marginals()
        if k >= e2e_warm:
            e2e_s.append(time.perf_counter() - t0)
        r.close()
        Q.close()
        assert p.shape == (n,)
    barrier()
    e2e_mean = max_over_ranks(statistics.mean(e2e_s))
    e2e_value = world * attempts_step / e2e_mean

    hbm, peak_kind = peaks()
    alg = algorithmic_bytes(a, BRANCHES, sched.sweeps, sched.refresh_sweeps, accepted)
    achieved = alg / (anneal_ms / 1e3) / 1e9
    traffic = None
    if NCU_TRAFFIC_PER_SWEEP is not None:
        traffic = NCU_TRAFFIC_PER_SWEEP * sched.sweeps
    line = {
        "metric": METRIC, "value": value, "unit": "attempts/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32 dE; residuals compensated f32 (hi + lo), f64 refresh every 50 sweeps",
        "data": "synthetic",
        "config": workload_config(a, sched.sweeps, world),
        "plan": {"colours": int(pinfo.n_colours), "footprint_mib": round(pinfo.device_bytes / 2**20)},
        "e2e": {"value": e2e_value, "unit": "attempts/s", "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": d2h,
                "s_per_step": e2e_mean, "warmup_steps": e2e_warm},
        "gpu_launches": launches,
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": hbm, "unit": "GB/s", "frac": achieved / hbm,
                     "peak_kind": peak_kind, "traffic": traffic, "kernel": "resid_lockstep_kernel",
                     "kernel_ms": anneal_ms, "algorithmic_bytes": alg, "accepted_flips": accepted},
        "max_residual_drift": drift,
        "max_energy_error": energy_err,
        "clocks": clocks,
    }
    if rank == 0 and world == 1 and args.serve_requests > 0:
        # the serving target on a stated stream of the mixed workload, recorded
        # beside the pyramid line: served throughput against each request
        # solved alone, latencies, identical results
        m = serve_measure(args.serve_requests, rates=(0.5,), plain_sample=0)
        line["serve"] = {"stream": f"{m['requests']} requests of the serving workload ({SERVE_WORKLOAD})",
                         "policy": SERVE_POLICY, "total_attempts": m["total_attempts"],
                         "served_attempts_per_s": m["value"], "plain_attempts_per_s": m["plain"],
                         "served_vs_plain": m["vs_plain"], "makespan_s": m["makespan_s"], "latency": m["latency"],
                         "equal_energy": m["equal_energy"], "clocks": m["clocks"]}
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        threads = os.cpu_count() or 1
        branches = min(BRANCHES, threads)
        rate, wall, kind = cpu_baseline(a, sched, threads, branches)
        line["cpu_baseline"] = {"value": rate, "unit": "attempts/s", "cores": threads, "kind": kind,
                                "sample": f"{branches} of 16 branches, the full 250-sweep schedule, "
                                          f"{threads} threads, {wall:.1f} s"}
    if rank == 0 and world == 1 and not args.no_side_workloads:
        # the batched stream and the weighted lattice QUBO, each in its own
        # process after this line's measurements (W = 3 warm-up steps, 1 timed)
        line["batch"] = side_workload(["--workload", "batch", "--steps", "1", "--warmup", "3", "--no-cpu-baseline"])
        line["qubo"] = side_workload(["--workload", "qubo", "--steps", "1", "--warmup", "3", "--no-cpu-baseline"])
    if rank == 0:
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
