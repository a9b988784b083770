#!/usr/bin/env python
"""Benchmark: overlap-search reads/s and suffix-sort Msuffix/s of PASQUAL's hot path, the learned
index with the batched (queued, graph-replayed) search against the plain GPU backward search.

Workload (default): 250 Mbp synthetic genome, GC 42 %, 15 % repeat copies of 1-5 kbp segments at
0.5-2 % divergence; 100 bp reads at 20x from both strands (50 M reads) with 0.5 % substitution
errors; t = 55; 64-bit index, 4.8 G suffixes per index after de-duplication (equal or
reverse-complement reads dropped).  Data is seeded synthetic.

A step is one overlap search (find_intervals + transitive reduction + edge CSR) over every read,
with both indexes resident in HBM, in the library's default seed mode (1: depth-t interval scan
with sorted-continuation reduction).  ``value`` = reads searched / step time, whole job.

Beside it, on the same index: ``plain`` = the reference's method on the GPU (seed mode 0: walk
and FM-index DFS), ``learned`` = seed mode 2 (learned-index windows), ``learned_batched`` = seed
mode 2 through the queued persistent search replayed from a CUDA graph with the autotuned plan,
``learned_batched_vs_plain`` = the ratio of the last two.  Every mode's edges are compared with
the plain search's.  ``roofline`` is the dominant kernel's algorithmic traffic as the library
counts it inside the kernels (32-byte sectors of index data loaded + result bytes written) over
its CUDA-event time, against the measured HBM copy bandwidth; ``reference_probes_per_read`` is the
reference method's work, which the GPU method avoids.

``e2e`` runs the public API end to end each step: pinned host reads -> GPU suffix sorts and
FM-indexes -> overlap search -> edges back to host arrays.

``--impl reference`` times the reference's CPU algorithm for the same metric and workload: the C
restatement of the reference (oracle/), OpenMP over all host cores, each step a bounded sample.
"""
from __future__ import annotations

import argparse
import json
import os
import re
import signal
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

import numpy as np  # noqa: E402

METRIC = "overlap-search reads/s + sort Msuffix/s, learned vs plain GPU, bit-exact"
WORKLOAD = "250Mbp_L100_20x_t55"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default=WORKLOAD)
    ap.add_argument("--scale", type=float, default=1.0, help="genome-size scale (1.0 = full)")
    ap.add_argument("--cpu-scale", type=float, default=0.05,
                    help="genome-size scale of the CPU-baseline sample's index")
    ap.add_argument("--cpu-seconds", type=float, default=20.0,
                    help="CPU work of the cpu_baseline sample (reference arm: of all steps together)")
    ap.add_argument("--e2e-steps", type=int, default=3)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-modes", action="store_true", help="skip the plain/learned comparison")
    ap.add_argument("--batched-scale", type=float, default=0.1,
                    help="genome scale of the mixed read-set queued workload (0 = skip)")
    ap.add_argument("--detail", default="", help="also write every figure to this JSON file")
    ap.add_argument("--seed-mode", type=int, default=1, choices=[0, 1, 2],
                    help="seed mode of the timed search (0: the reference's walk and DFS, k_search_fast)")
    return ap.parse_args()


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def _group_size() -> int:
    import torch.distributed as dist
    return dist.get_world_size() if dist.is_available() and dist.is_initialized() else 1


def rank_barrier() -> None:
    """Barrier over the replicas (the default process group); nothing with one rank."""
    if _group_size() > 1:
        import torch.distributed as dist
        dist.barrier()


def rank_max(x: float, device="cpu") -> float:
    """Maximum of x over the replicas (x itself with one rank).  `device` is where the reduction
    tensor lives: the rank's GPU under NCCL, the CPU under gloo."""
    if _group_size() == 1:
        return x
    import torch
    import torch.distributed as dist
    tt = torch.tensor([x], device=device, dtype=torch.float64)
    dist.all_reduce(tt, op=dist.ReduceOp.MAX)
    return float(tt.item())


def replica_throughput(reads_per_rank: int, world: int, slowest_ms: float) -> float:
    """Whole-job reads/s of `world` replicas that each searched reads_per_rank reads, the slowest
    in slowest_ms per step (weak scaling: every rank searches its own full read set)."""
    return reads_per_rank * world / (slowest_ms * 1e-3)


def workload_reads(name: str, scale: float):
    from pasqual_gb300 import synth
    _, rd, L, t = synth.make_workload(name, scale=scale)
    return synth.dedup(rd), L, t


def workload_config(name: str) -> dict:
    """The workload as both arms report it (its definition, not quantities measured on it)."""
    from pasqual_gb300 import synth
    w = synth.WORKLOADS[name]
    return {"workload": name, "genome_bp": w["genome"], "read_len": w["L"], "coverage": w["cov"],
            "t": w["t"], "index": "U%d" % w.get("index", 32),
            "l2": "inputs larger than L2 (both FM-indexes, suffix arrays and packed texts), no flush"}


def measured_peak_hbm():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(p) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


def profile_figure(name: str, key: str):
    """A figure recorded in a committed ncu summary under profiles/ ("key = value")."""
    p = os.path.join(ROOT, "profiles", name)
    try:
        txt = open(p).read()
    except OSError:
        return None
    m = re.search(re.escape(key) + r"\s*=\s*([0-9.]+)", txt)
    return float(m.group(1)) if m else None


def r4(x):
    """Four significant digits (keeps the JSON line short)."""
    if x is None or isinstance(x, (bool, int)):
        return x
    return float("%.4g" % x)


class Clocks:
    """nvidia-smi sampling during the timed region."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.path = None

    def start(self):
        """Start sampling and wait (up to 10 s) for the first sample, so that the sampler's own
        start-up stays out of the timed region."""
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.device), "--query-gpu=" + self.Q,
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None
            return
        t0 = time.time()
        while time.time() - t0 < 10.0 and self.proc.poll() is None:
            if os.path.getsize(self.path) > 0:
                break
            time.sleep(0.05)

    def stop(self):
        if not self.proc:
            return None
        self.proc.send_signal(signal.SIGTERM)
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx.append(float(f[2]))
            except ValueError:
                continue
            for nm, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        os.unlink(self.path)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx),
                "reasons": sorted(reasons), "samples": len(sm)}


class CpuSample:
    """The C restatement of the reference's overlap search on the host cores (OpenMP): the index
    of the workload's genome scaled by `scale` (same read length, coverage, t and error rate),
    built once, then searched read range by read range."""

    def __init__(self, workload: str, scale: float, threads: int | None = None):
        from oracle import port
        port.build()
        self.rd, self.L, self.t = workload_reads(workload, scale)
        self.workload, self.scale = workload, scale
        self.threads = threads or os.cpu_count() or 1
        from pasqual_gb300 import synth
        width = synth.WORKLOADS[workload].get("index", 32)
        self.P = port.Port(width)
        self.ix = self.P.build_index(self.rd, self.t, threads=self.threads, seed_k=min(12, self.t))
        self.seeds = (self.ix["seed0"], self.ix["seed1"])
        self.next = 0

    def search(self, seconds: float):
        """Search about `seconds` of reads, continuing where the last call stopped and wrapping
        around the sample's reads as often as needed; returns (reads, seconds, probes)."""
        nr = self.rd.shape[0]
        probe = min(nr, 4000)
        t0 = time.perf_counter()
        self._run(probe)
        dt = time.perf_counter() - t0
        count = int(max(probe, probe * seconds / max(dt, 1e-6)))
        t0 = time.perf_counter()
        probes = self._run(count)
        return count, time.perf_counter() - t0, probes

    def _run(self, count: int) -> int:
        nr = self.rd.shape[0]
        probes = 0
        while count > 0:
            take = min(count, nr - self.next)
            g = self.P.overlaps(self.ix, self.next, take, threads=self.threads, seeds=self.seeds)
            probes += g.probes
            self.next = (self.next + take) % nr
            count -= take
        return probes

    def describe(self, count: int, secs: float) -> str:
        return ("%d reads of the %s workload's reads at genome scale %g (%d reads kept, %d bp, "
                "t=%d), searched in %.1f s against their own index (seeds at depth 12)"
                % (count, self.workload, self.scale, self.rd.shape[0], self.L, self.t, secs))


def cpu_baseline(workload: str, scale: float, seconds: float):
    cs = CpuSample(workload, scale)
    n, secs, probes = cs.search(seconds)
    return {"value": n / secs, "unit": "reads/s", "cores": cs.threads, "kind": "port",
            "sample": cs.describe(n, secs), "probes_per_read": probes / max(n, 1)}


def run_reference(args):
    rank, world, _ = dist_env()
    if rank != 0:
        return
    cs = CpuSample(args.workload, args.cpu_scale)
    per_step = max(0.5, args.cpu_seconds / max(1, args.steps))
    for _ in range(args.warmup):
        cs.search(per_step / 4)
    vals, total_n, total_s = [], 0, 0.0
    for _ in range(args.steps):
        n, secs, _ = cs.search(per_step)
        vals.append(n / secs)
        total_n += n
        total_s += secs
    v = statistics.median(vals)
    out = {"impl": "reference", "metric": METRIC, "value": r4(v), "unit": "reads/s", "n_gpus": world,
           "steps": args.steps, "warmup": args.warmup, "higher_is_better": True,
           "scaling": "weak", "vs_baseline": None,
           "dtype": "int%s-index" % workload_config(args.workload)["index"][1:],
           "data": "synthetic", "config": workload_config(args.workload),
           "cpu_baseline": {"value": r4(v), "unit": "reads/s", "cores": cs.threads, "kind": "port",
                            "sample": "per step: " + cs.describe(total_n // max(1, args.steps),
                                                                 total_s / max(1, args.steps))},
           "e2e": {"value": r4(v), "unit": "reads/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(out), flush=True)


def timed_mode(P, nr: int, steps: int, run, stream, device):
    """Warm-up, then `steps` timed runs of one search configuration: search ms (CUDA events
    around the whole call), kernel ms, probes and algorithmic bytes per read, the graph."""
    import torch
    run()
    ms, kern = [], []
    for _ in range(steps):
        torch.cuda.synchronize(device)
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        run()
        e1.record(stream)
        torch.cuda.synchronize(device)
        ms.append(e0.elapsed_time(e1))
        kern.append(P.kernel_stats()[0])
    g = P.graph()
    sec, outb = P.search_traffic()
    return {"ms": statistics.median(ms), "kernel_ms": statistics.median(kern), "graph": g,
            "probes_per_read": g.probes / max(nr, 1), "bytes": 32.0 * sec + outb}


def modes_block(P, nr: int, steps: int, stream, device, peak: float, plain_ref):
    """The reference's method (mode 0), learned windows (mode 2) and learned windows through the
    queued search with graph replay, each on the same index, each with its edges compared with
    the default mode's (which the caller has checked against its own search)."""
    import pasqual_gb300 as pq
    out = {}
    ref_dest, ref_off = plain_ref
    P.learned_build(0, 400)
    P.learned_build(1, 400)
    for name, mode, batched in (("plain", 0, False), ("learned", 2, False), ("learned_batched", 2, True)):
        P.set_seed_mode(mode)
        if batched:
            pq.autotune_batched([P], graph=True)
            r = timed_mode(P, nr, steps, lambda: pq.overlaps_batched([P], graph=True), stream, device)
        else:
            r = timed_mode(P, nr, steps, P.overlaps, stream, device)
        g = r["graph"]
        same = bool(np.array_equal(g.dest, ref_dest) and np.array_equal(g.edge_off, ref_off))
        tiers = P.tier_stats()
        out[name] = {"reads_per_s": r4(nr / (r["ms"] * 1e-3)), "ms": r4(r["ms"]),
                     "handed_over": [tiers[k] for k in ("deferred", "block", "heavy", "wide")],
                     "kernel_ms": r4(r["kernel_ms"]), "probes_per_read": r4(r["probes_per_read"]),
                     "bytes_per_read": r4(r["bytes"] / max(nr, 1)),
                     "frac": r4(r["bytes"] / (r["kernel_ms"] * 1e-3) / 1e9 / peak),
                     "edges_equal": same}
    lx = [P.learned_info(d) for d in (0, 1)]
    out["learned_model"] = {
        "train_ms": r4(sum(x["train_ms"] for x in lx)),
        "build_ms": r4(sum(x["keys_ms"] + x["train_ms"] + x["eval_ms"] for x in lx)),
        "window_rows": r4(statistics.mean(x["mean_window"] for x in lx)),
        "window_rows_root": r4(statistics.mean(x["mean_window_root"] for x in lx)),
        "misses": lx[0]["misses"]}
    st = P.batch_stats()
    out["learned_batched"]["plan"] = [st["ctas_per_sm"], st["groups_per_item"], st["edge_slots"]]
    P.set_seed_mode(1)
    return out


def mixed_sets(scale: float, steps: int, device, stream):
    """Several read sets of uneven read length and mixed t (100 Mbp genome scaled): one search
    launch per set against the queued persistent search from a CUDA graph with the autotuned
    plan, in seed mode 2; the edges must be each set's own."""
    import torch
    import pasqual_gb300 as pq
    from pasqual_gb300 import synth
    name = "100Mbp_L75-250_25x_batched"
    sets = synth.make_batches(name, scale=scale)
    ctxs = []
    try:
        for rd, L, t in sets:
            P = pq.Pasqual(32, device=device, stream=stream.cuda_stream)
            P.set_reads(rd, t)
            P.set_seed_mode(2)
            P.build_index()
            ctxs.append(P)
        total = sum(rd.shape[0] for rd, _, _ in sets)

        def timed(fn):
            fn()
            torch.cuda.synchronize(device)
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            for _ in range(steps):
                fn()
            e1.record(stream)
            torch.cuda.synchronize(device)
            return e0.elapsed_time(e1) / steps

        seq_ms = timed(lambda: [P.overlaps() for P in ctxs])
        ref = [P.graph().dest.copy() for P in ctxs]
        pq.autotune_batched(ctxs, graph=True)
        q_ms = timed(lambda: pq.overlaps_batched(ctxs, graph=True))
        same = all(np.array_equal(P.graph().dest, r) for P, r in zip(ctxs, ref))
        return {"scale": scale, "sets": len(sets),
                "L": [L for _, L, _ in sets], "t": [t for _, _, t in sets], "reads": int(total),
                "seq_reads_per_s": r4(total / (seq_ms * 1e-3)),
                "queued_reads_per_s": r4(total / (q_ms * 1e-3)), "queued_vs_seq": r4(seq_ms / q_ms),
                "edges_equal": bool(same)}
    finally:
        for P in ctxs:
            P.close()


def run_ours(args):
    import torch
    import pasqual_gb300 as pq
    from pasqual_gb300 import synth

    rank, world, local = dist_env()
    detail = {}
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)

    t_start = time.time()
    # the end-to-end steps' input buffer: page-locked (pq_host_alloc), which pq_set_reads copies
    # with a kernel that keeps the link's rate after the sorts and the search
    w = synth.WORKLOADS[args.workload]
    raw_reads = int(max(int(w["genome"] * args.scale), 4 * w["L"]) * w["cov"] // w["L"])
    pinned_all = torch.from_numpy(pq.host_empty((raw_reads, w["L"]), np.uint8))
    rd, L, t = workload_reads(args.workload, args.scale)
    nr = rd.shape[0]
    n = nr * L
    detail["workload_s"] = r4(time.time() - t_start)
    width = 32 if n < (1 << 32) else 64          # the reference's U32/U64 split by index size
    width = max(width, synth.WORKLOADS[args.workload].get("index", 32))
    stream = torch.cuda.Stream(device=dev)
    P = pq.Pasqual(width, device=local, stream=stream.cuda_stream)
    P.set_seed_mode(args.seed_mode)
    peak, peak_kind = measured_peak_hbm()

    # ---- index build (setup) and suffix-sort throughput (suffix arrays only, both directions)
    P.set_reads(rd, t)
    P.build_index()                       # warm-up build
    sort_ms = []
    for _ in range(max(1, min(args.steps, 3))):
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize(dev)
        e0.record(stream)
        P.sort(0)
        P.sort(1)
        e1.record(stream)
        torch.cuda.synchronize(dev)
        sort_ms.append(e0.elapsed_time(e1))
    P.build_index()                       # index for the search; sort scratch given back
    sort_ms_med = statistics.median(sort_ms)

    # ---- overlap search in the default mode: warm-up, then K timed steps (clocks sampled)
    clocks = Clocks(local)
    clocks.start()
    for _ in range(args.warmup):
        P.overlaps()
    _, l0 = P.kernel_stats()
    kern_ms = []
    rank_barrier()
    torch.cuda.synchronize(dev)
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(args.steps):
        P.overlaps()
        kern_ms.append(P.kernel_stats()[0])
    e1.record(stream)
    torch.cuda.synchronize(dev)
    rank_barrier()
    ck = clocks.stop()
    _, l1 = P.kernel_stats()
    step_ms = rank_max(e0.elapsed_time(e1) / args.steps, dev)
    g = P.graph()
    sec, outb = P.search_traffic()
    detail["tiers"] = {k: r4(v) for k, v in P.tier_stats().items()}
    ref_graph = (g.dest.copy(), g.edge_off.copy())
    kms = statistics.median(kern_ms)
    alg_bytes = 32.0 * sec + outb
    achieved = alg_bytes / (kms * 1e-3) / 1e9
    dram_per_read = profile_figure("search_kernels.md", "dram_bytes_per_read")
    # the committed capture describes this launch only if its kernel did the same work per read
    # (same algorithmic bytes, within 5 %): otherwise no traffic figure is claimed
    cap_alg = profile_figure("search_kernels.md", "algorithmic_bytes_per_read")
    traffic_applies = bool(dram_per_read and cap_alg and args.seed_mode == 1 and
                           abs(alg_bytes / nr - cap_alg) <= 0.05 * cap_alg)

    # ---- end to end through the public API with host buffers
    pinned = pinned_all[:nr]
    pinned.numpy()[:] = rd
    del rd
    # the page-locked buffer's plain copy rate (torch), for the record
    probe = torch.empty((nr, L), dtype=torch.uint8, device=dev)
    torch.cuda.synchronize(dev)
    c0 = torch.cuda.Event(enable_timing=True)
    c1 = torch.cuda.Event(enable_timing=True)
    c0.record(stream)
    with torch.cuda.stream(stream):
        probe.copy_(pinned, non_blocking=True)
    c1.record(stream)
    torch.cuda.synchronize(dev)
    detail["h2d_copy_gbs"] = r4(nr * L / (c0.elapsed_time(c1) * 1e-3) / 1e9)
    del probe
    e2e_ms, parts = [], []
    h2d = nr * L
    d2h = 0
    # the graph's host arrays: page-locked, of the sizes of the search's graph, reused every step
    gg = pq.Graph(**{f: pq.host_empty((getattr(g, f).size,), getattr(g, f).dtype)
                     for f in ("num_B", "num_F", "olp_B", "olp_F", "edge_off", "dest", "length", "etype", "trans")})
    for s in range(args.e2e_steps + 1 if args.e2e_steps > 0 else 0):
        torch.cuda.synchronize(dev)
        g0 = torch.cuda.Event(enable_timing=True)
        g1 = torch.cuda.Event(enable_timing=True)
        t0 = time.perf_counter()
        g0.record(stream)
        P.set_reads(pinned.numpy(), t)
        g1.record(stream)
        t1 = time.perf_counter()
        P.build_index()
        t2 = time.perf_counter()
        P.overlaps()
        t3 = time.perf_counter()
        gg = P.graph(out=gg)
        d2h = sum(a.nbytes for a in (gg.num_B, gg.num_F, gg.olp_B, gg.olp_F, gg.edge_off, gg.dest,
                                      gg.length, gg.etype, gg.trans))
        torch.cuda.synchronize(dev)
        t4 = time.perf_counter()
        if s > 0:                          # first pass is a warm-up
            e2e_ms.append((t4 - t0) * 1e3)
            sm, fm, _ = P.stage_ms()
            g1.synchronize()
            parts.append({"set_reads": r4((t1 - t0) * 1e3), "set_reads_gpu": r4(g0.elapsed_time(g1)), "build_index": r4((t2 - t1) * 1e3),
                          "sort": r4(sm), "fm": r4(fm), "search": r4((t3 - t2) * 1e3),
                          "d2h": r4((t4 - t3) * 1e3)})
    e2e_ms_med = rank_max(statistics.median(e2e_ms), dev) if e2e_ms else None
    detail["e2e_steps"] = [dict(p, step_ms=r4(ms)) for p, ms in zip(parts, e2e_ms)]
    del pinned, pinned_all

    if rank != 0:
        P.close()
        return
    cb = None
    if world == 1 and not args.no_cpu_baseline:
        cb = cpu_baseline(args.workload, args.cpu_scale, args.cpu_seconds)
    ref_ppr = cb["probes_per_read"] if cb else profile_figure("search_kernels.md", "reference_probes_per_read")
    out = {
        "metric": METRIC, "value": r4(replica_throughput(nr, world, step_ms)), "unit": "reads/s",
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": r4(step_ms),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "int%d-index" % width, "data": "synthetic",
        "config": workload_config(args.workload),
        "gpu_launches": int(l1 - l0),
        "roofline": {"bound": "hbm", "achieved": r4(achieved), "peak": peak, "unit": "GB/s",
                     "frac": r4(achieved / peak), "peak_kind": peak_kind,
                     "kernel": "k_search_fast" if args.seed_mode == 0 else "k_search_lean", "kernel_ms": r4(kms),
                     "bytes_per_read": r4(alg_bytes / nr),
                     "traffic": r4(dram_per_read * nr) if traffic_applies else None,
                     "reference_probes_per_read": r4(ref_ppr), "probes_per_read": r4(g.probes / nr)},
        "e2e": ({"value": r4(replica_throughput(nr, world, e2e_ms_med)), "unit": "reads/s",
                 "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h, "ms_per_step": r4(e2e_ms_med),
                 "parts_ms": parts[-1]} if e2e_ms_med else None),
    }
    if ck:
        out["clocks"] = ck
    if cb:
        out["cpu_baseline"] = {k: (r4(cb[k]) if k == "value" else cb[k])
                               for k in ("value", "unit", "cores", "kind", "sample")}
    detail["reads"] = nr
    detail["wall_s"] = r4(time.time() - t_start)
    detail["suffixes_per_index"] = n
    detail["edges"] = len(g.dest)
    detail["wide_tier_reads"] = g.wide_reads
    if not args.no_modes:
        m = modes_block(P, nr, max(1, min(args.steps, 3)), stream, dev, peak, ref_graph)
        detail["modes"] = m
    P.close()
    if args.batched_scale > 0:
        detail["mixed_sets"] = mixed_sets(args.batched_scale, max(1, min(args.steps, 3)), local, stream)
    if args.detail:
        with open(args.detail, "w") as f:
            json.dump({"line": out, "detail": detail}, f, indent=1)
    # the figures read most often go last: a reader that keeps only the end of the line sees them
    out["reads"] = nr
    out["modes"] = detail.get("modes")
    out["mixed_sets"] = detail.get("mixed_sets")
    out["sort_msuffix_per_s"] = r4(2 * n / (sort_ms_med * 1e-3) / 1e6)
    # the sort against its algorithmic bytes: per suffix, the 2-bit text of the prefix that tells
    # it apart from its neighbours plus one suffix-array entry (measured on the oracle's suffix
    # arrays of a sample of this workload, recorded with its counters)
    sbytes = (profile_figure("sort_and_block_kernels.md", "sort_bytes_per_suffix")
              if args.workload == "250Mbp_L100_20x_t55" else None)
    if sbytes:
        sach = sbytes * 2 * n / (sort_ms_med * 1e-3) / 1e9
        out["sort_roofline"] = {"bound": "hbm", "achieved": r4(sach), "peak": peak, "unit": "GB/s",
                                "frac": r4(sach / peak), "bytes_per_suffix": sbytes}
    if "modes" in detail:
        mo = detail["modes"]
        out["plain_reads_per_s"] = mo["plain"]["reads_per_s"]
        out["learned_batched_reads_per_s"] = mo["learned_batched"]["reads_per_s"]
        out["learned_batched_vs_plain"] = r4(mo["learned_batched"]["reads_per_s"] / mo["plain"]["reads_per_s"])
        out["edges_equal_all_modes"] = all(mo[k]["edges_equal"] for k in ("plain", "learned", "learned_batched"))
    print(json.dumps(out, separators=(",", ":")), flush=True)


def main():
    args = parse()
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
