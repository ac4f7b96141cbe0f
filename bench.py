#!/usr/bin/env python
"""Headline benchmark: pull-direction Jacobi PageRank (PageRankPull) on the
Kronecker scale-25 graph (edge factor 16, RMAT 0.57/0.19/0.19, symmetrized,
2^25 vertices, ~1.05e9 directed edges), float scores, damping 0.85,
epsilon 1e-4, at most 20 sweeps -- the configuration the reference's
pr_spmv -g 25 runs.

One step = one complete solve (init, sweeps until the L1 change < epsilon,
scores written in the caller's vertex order).  Prints ONE JSON line on rank 0:
  value        GTEPS (directed edges x sweeps / second), whole job, inputs
               resident in HBM, CUDA events on the launching stream
  e2e          the same metric through the C-ABI host call (pr_gpu_run):
               scores copied back to a pinned host buffer every step
  roofline     the fused sweep kernel: algorithmic bytes per sweep
               (4M + 20N + 4) / average sweep time vs measured HBM copy peak
  cpu_baseline the reference's own PageRankPull (compiled from its sources)
               on this host's cores, bounded sample
  ppr          batched personalized PageRank (64 teleport vectors, Kronecker
               scale 22) vs 64 sequential single-vector solves
  noalloc      pr_gpu_run_noalloc (no device allocation) at its size limit,
               beside the regular entry point on the same graph
  verify       the reference's PRVerifier on the device (pr_gpu_verify) on
               the timed solve's scores, beside the reference's serial one
               on the same scores (whose error must be the same double)

--gpus N under torchrun: N independent replicas (the path does not shard),
timed as the max over ranks.  --impl reference: the reference arm (rank 0).
"""
from __future__ import annotations

import argparse
import hashlib
import json
import os
import statistics
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

HBM_FALLBACK_GBS = 6650.0
METRIC = "PR GTEPS & HBM GB/s vs peak; batched PPR vs plain GPU at L1<=1e-4"


def parse_args():
    p = argparse.ArgumentParser(description=__doc__.split("\n\n")[0])
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=10)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", choices=["ours", "reference"], default="ours")
    p.add_argument("--graph", default="-g 25", help="pr_spmv graph options of the workload")
    p.add_argument("--max-iters", type=int, default=20)
    p.add_argument("--epsilon", type=float, default=1e-4)
    p.add_argument("--ppr-graph", default="-g 22")
    p.add_argument("--ppr-cols", type=int, default=64)
    p.add_argument("--no-ppr", action="store_true")
    p.add_argument("--adjoint-graph", default="-g 20")
    p.add_argument("--no-adjoint", action="store_true")
    p.add_argument("--no-cc", action="store_true")
    p.add_argument("--no-bfs", action="store_true")
    p.add_argument("--bfs-sources", type=int, default=8)
    p.add_argument("--e2e-upload-steps", type=int, default=5,
                   help="steps of the end-to-end variant that uploads the graph every step")
    p.add_argument("--no-verify", action="store_true")
    p.add_argument("--noalloc-graph", default="-g 20",
                   help="graph of the no-allocation entry point's leg (at most 2^20 vertices)")
    p.add_argument("--no-noalloc", action="store_true")
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--cpu-trials", type=int, default=2)
    return p.parse_args()


# ---------------------------------------------------------------------------
# distributed plumbing (replicas only: one barrier and one max per timing)

class Dist:
    def __init__(self, init: bool = True):
        self.world = int(os.environ.get("WORLD_SIZE", "1"))
        self.rank = int(os.environ.get("RANK", "0"))
        self.local_rank = int(os.environ.get("LOCAL_RANK", "0"))
        self.pg = None
        if self.world > 1 and init:
            import datetime
            import torch.distributed as dist
            backend = "nccl" if _cuda_ok() else "gloo"
            if backend == "nccl":
                import torch
                torch.cuda.set_device(self.local_rank)
            dist.init_process_group(backend=backend, timeout=datetime.timedelta(seconds=300))
            self.pg = dist

    def barrier(self):
        if self.pg:
            self.pg.barrier()

    def max(self, x: float) -> float:
        if not self.pg:
            return x
        import torch
        dev = f"cuda:{self.local_rank}" if _cuda_ok() else "cpu"
        t = torch.tensor([x], dtype=torch.float64, device=dev)
        self.pg.all_reduce(t, op=self.pg.ReduceOp.MAX)
        return float(t.item())

    def sum(self, x: float) -> float:
        if not self.pg:
            return x
        import torch
        dev = f"cuda:{self.local_rank}" if _cuda_ok() else "cpu"
        t = torch.tensor([x], dtype=torch.float64, device=dev)
        self.pg.all_reduce(t, op=self.pg.ReduceOp.SUM)
        return float(t.item())

    def close(self):
        if self.pg:
            self.pg.destroy_process_group()


def _cuda_ok() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


# ---------------------------------------------------------------------------
# clocks during the timed region

class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.rows = []
        self._t = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-i", str(self.gpu), "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None
            return
        self._t = threading.Thread(target=self._read, daemon=True)
        self._t.start()

    def _read(self):
        for line in self.proc.stdout:
            parts = [x.strip() for x in line.split(",")]
            if len(parts) >= 9:
                self.rows.append(parts)

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        if self._t:
            self._t.join(timeout=5)
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in self.rows:
            try:
                sm.append(float(r[1]))
                smax.append(float(r[2]))
            except ValueError:
                continue
            for name, val in zip(names, r[5:9]):
                if val.strip().lower() == "active":
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm)}


# ---------------------------------------------------------------------------

def measured_peak():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as fh:
            d = json.load(fh)
        if d.get("hbm_gbs"):
            return float(d["hbm_gbs"]), "measured (MEASURED_PEAKS.json hbm_gbs)"
    return HBM_FALLBACK_GBS, "fallback"


def profiled_traffic(graph_args: str):
    """DRAM bytes per slice-blocked sweep (its three kernels) from the committed
    ncu summary."""
    p = os.path.join(ROOT, "profiles", "blocked_sweep_traffic.json")
    if not os.path.exists(p):
        return None
    with open(p) as fh:
        d = json.load(fh)
    e = d.get(graph_args.strip())
    return None if e is None else float(e["dram_bytes_per_sweep"])


def sweep_bytes(n: int, m: int, directed: bool) -> int:
    """Algorithmic bytes of one plain sweep: neighbour ids 4M, offsets 4(N+1),
    contrib read 4N, old score 4N, new score 4N, next contrib 4N (+4(N+1)
    out-offsets for a directed graph)."""
    b = 4 * m + 20 * n + 4
    if directed:
        b += 4 * (n + 1)
    return b


def synthetic(args_str: str) -> bool:
    """-g / -u graphs are generated on the GPU (pr_gpu_generate)."""
    toks = args_str.split()
    return bool(toks) and toks[0] in ("-g", "-u") and all(t in ("-g", "-u", "-k") or t.isdigit()
                                                          for t in toks)


def shm_graph_path(args_str: str) -> str:
    h = hashlib.sha1(args_str.encode()).hexdigest()[:12]
    base = "/dev/shm" if os.path.isdir("/dev/shm") else tempfile.gettempdir()
    return os.path.join(base, f"gapbs_bench_{h}.sg")


def load_graph(args_str: str, dist: Dist):
    from gapbs_b200.graph import make_graph
    if dist.world == 1:
        return make_graph(args_str)
    path = shm_graph_path(args_str)
    if dist.rank == 0:
        g = make_graph(args_str)
        g.write_sg(path + ".tmp")
        os.replace(path + ".tmp", path)
    dist.barrier()
    if dist.rank != 0:
        g = make_graph(f"-f {path}")
    dist.barrier()
    if dist.rank == 0:
        os.remove(path)
    return g


def ppr_teleports(g, k: int, seed: int):
    """k teleport vectors, seed sets of log-uniform size in [1, 4096] drawn
    from the non-isolated vertices; uniform 1/|S| on each set."""
    rng = np.random.default_rng(seed)
    cand = np.nonzero(np.diff(g.out_offsets) > 0)[0]
    T = np.zeros((g.num_nodes, k), np.float32)
    sizes = []
    for c in range(k):
        size = int(round(np.exp(rng.uniform(0.0, np.log(4096.0)))))
        size = max(1, min(size, cand.size))
        seeds = rng.choice(cand, size=size, replace=False)
        T[seeds, c] = np.float32(1.0 / size)
        sizes.append(size)
    return T, sizes


# ---------------------------------------------------------------------------
# our arm

def run_ours(a, dist: Dist):
    import torch
    from gapbs_b200 import PageRankEngine
    dev = dist.local_rank
    torch.cuda.set_device(dev)
    eng = PageRankEngine(dev)
    g = None
    on_gpu = synthetic(a.graph)  # (g may be downloaded later for other legs)
    if on_gpu:
        # the reference's -g / -u graph, built on this GPU (identical CSR)
        t0 = time.perf_counter()
        n, m = eng.generate(a.graph)
        build_s = time.perf_counter() - t0
        upload_s, upload_bytes, directed = 0.0, 0, False
    else:
        t0 = time.perf_counter()
        g = load_graph(a.graph, dist)
        build_s = time.perf_counter() - t0
        n, m, directed = g.num_nodes, g.num_edges_directed, g.directed
        t0 = time.perf_counter()
        eng.upload(g)
        upload_s = time.perf_counter() - t0
        upload_bytes = 4 * (n + 1) + 4 * m
    # a stream of its own for the bench and the engine: a handle given the
    # default stream issues on its own one, beside the buffer write that evicts
    # L2, and the events around a step would not be on the launching stream
    stream = torch.cuda.Stream(dev)
    torch.cuda.set_stream(stream)
    eng.set_stream(stream.cuda_stream)
    out = torch.empty(n, dtype=torch.float32, device=f"cuda:{dev}")
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device=f"cuda:{dev}")  # 256 MB > L2

    # ---- device-resident solves (value)
    for _ in range(a.warmup):
        eng.run_device(a.max_iters, a.epsilon, 0.85, 1, None, out.data_ptr())
    torch.cuda.synchronize()
    dist.barrier()
    clocks = ClockSampler(dev)
    clocks.start()
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
          for _ in range(a.steps)]
    sweeps_total, sweep_ms_total, launches = 0, 0.0, 0
    torch.cuda.synchronize()
    for i in range(a.steps):
        flush.fill_(float(i))                      # evict L2 between steps
        ev[i][0].record(stream)
        sw, _ = eng.run_device(a.max_iters, a.epsilon, 0.85, 1, None, out.data_ptr())
        ev[i][1].record(stream)
        sweep_ms, _total_ms, nl = eng.last_timing()
        sweeps_total += int(sw[0])
        sweep_ms_total += sweep_ms
        launches += nl
    torch.cuda.synchronize()
    step_ms = [s.elapsed_time(e) for s, e in ev]
    clk = clocks.stop()
    local_ms = float(sum(step_ms))
    dist.barrier()
    max_ms = dist.max(local_ms)
    sweeps_per_step = sweeps_total / a.steps
    edges_all = dist.sum(float(m) * sweeps_total)
    value = edges_all / (max_ms / 1e3) / 1e9
    # the sweep layout the timed solves ran with
    layout = eng.sweep_layout_info()
    blocked = layout["last_run_blocked"]
    one_launch = launches == a.steps  # gather solves, each a launch

    # ---- end to end through the C-ABI host call (pinned host result buffer)
    eng.set_stream(None)
    host_out = torch.empty(n, dtype=torch.float32, pin_memory=True).numpy()
    for _ in range(max(1, a.warmup)):
        eng.run(a.max_iters, a.epsilon, out=host_out)
    dist.barrier()
    e2e_s, e2e_sweeps = 0.0, 0
    for i in range(a.steps):
        flush.fill_(float(i))
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        res = eng.run(a.max_iters, a.epsilon, out=host_out)
        e2e_s += time.perf_counter() - t0
        e2e_sweeps += int(res.sweeps[0])
        launches_e2e = eng.last_timing()[2]
    e2e_s = dist.max(e2e_s)
    e2e_edges = dist.sum(float(m) * e2e_sweeps)
    e2e_value = e2e_edges / e2e_s / 1e9

    # ---- the reference's PRVerifier on the device (pr_gpu_verify: the host
    # scores of the last solve in, the error out) on the same graph
    verify = None
    if not a.no_verify:
        scores_v = np.array(host_out, copy=True)
        eng.verify(scores_v)  # warm-up
        vt = []
        for _ in range(3):
            t0 = time.perf_counter()
            err_v = eng.verify(scores_v)
            vt.append(time.perf_counter() - t0)
        verify = {"workload": f"PRVerifier of the timed solve's scores on {a.graph.strip()}",
                  "ms": round(dist.max(float(np.median(vt))) * 1e3, 3),
                  "unit": "ms per call (C ABI: host scores in, error out; copies included)",
                  "statistic": "median of 3 calls", "error": err_v,
                  "passes": bool(err_v < a.epsilon)}

    # ---- connected components (the reference's Afforest) on the same graph
    cc = None
    if not a.no_cc:
        comp = torch.empty(n, dtype=torch.int32, device=f"cuda:{dev}")
        eng.set_stream(stream.cuda_stream)
        for _ in range(max(1, a.warmup)):
            eng.connected_components_device(comp.data_ptr())
        torch.cuda.synchronize()
        c0, c1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        c0.record(stream)
        for _ in range(a.steps):
            eng.connected_components_device(comp.data_ptr())
        c1.record(stream)
        torch.cuda.synchronize()
        cc_ms = dist.max(c0.elapsed_time(c1) / a.steps)
        cc = {"workload": f"Afforest connected components of {a.graph.strip()}",
              "ms": round(cc_ms, 3), "unit": "ms per run (device-resident graph)",
              "edges_per_s": round(m / (cc_ms / 1e3) / 1e9, 2),
              "components": int(torch.unique(comp).numel())}
        eng.set_stream(None)

    # ---- direction-optimizing BFS from fixed sources on the same graph
    bfs = None
    if not a.no_bfs:
        parent = torch.empty(n, dtype=torch.int32, device=f"cuda:{dev}")
        rng = np.random.default_rng(27491095 + 4)
        bfs_sources = [int(x) for x in rng.integers(0, n, 4 * a.bfs_sources)]
        eng.set_stream(stream.cuda_stream)
        for s_ in bfs_sources[:2]:
            eng.bfs_device(s_, parent.data_ptr())  # warm-up (also checks the sources)
        torch.cuda.synchronize()
        picked, t_total, steps_total = [], 0.0, 0
        b0, b1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        for s_ in bfs_sources:
            if len(picked) == a.bfs_sources:
                break
            torch.cuda.synchronize()
            b0.record(stream)
            nst = eng.bfs_device(s_, parent.data_ptr())  # returns once the search is done
            b1.record(stream)
            torch.cuda.synchronize()
            dt = b0.elapsed_time(b1) / 1e3
            if nst <= 2:
                continue  # an isolated source: nothing to search
            picked.append(s_)
            t_total += dt
            steps_total += nst
        bfs_ms = dist.max(t_total * 1e3 / max(1, len(picked)))
        bfs = {"workload": f"direction-optimizing BFS of {a.graph.strip()} from {len(picked)} "
                           "sources with out-edges (seeded draw)",
               "ms": round(bfs_ms, 3), "unit": "ms per search (device-resident graph, one "
                                               "launch per search)",
               "gteps": round(m / (bfs_ms / 1e3) / 1e9, 2), "steps_per_search":
                   round(steps_total / max(1, len(picked)), 1), "sources": picked}
        eng.set_stream(None)

    # ---- end to end with the graph uploaded every step (a caller whose graph
    # changes between solves): pr_gpu_upload of the host CSR + pr_gpu_run
    e2e_up = None
    if a.e2e_upload_steps > 0:
        if g is None:
            g = eng.download_graph()  # the generated graph, as a host CSR
        # a graph solved once per upload: the gather sweep (building the
        # slice-blocked layout costs more than it saves on one solve)
        eng.set_sweep_layout("gather")
        per_step, up_sweeps = [], 0
        for i in range(a.e2e_upload_steps + 1):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            eng.upload(g)
            res = eng.run(a.max_iters, a.epsilon, out=host_out)
            dt = time.perf_counter() - t0
            if i > 0:  # the first is a warm-up
                per_step.append(dt)
                up_sweeps += int(res.sweeps[0])
        # host-bound (pageable staging copy and DMA) on a host shared with
        # other jobs, so single steps can be slowed by others' memory traffic:
        # the value uses the median step, min and max are reported beside it
        med_s = dist.max(float(np.median(per_step)))
        sweeps_step = up_sweeps / max(1, len(per_step))
        e2e_up = {
            "value": round(dist.sum(float(m) * sweeps_step) / med_s / 1e9, 3), "unit": "GTEPS",
            "h2d_bytes_per_step": 4 * (n + 1) + 4 * m, "d2h_bytes_per_step": 4 * n,
            "path": "pr_gpu_upload (host CSR, pageable) + pr_gpu_run every step, gather sweep "
                    "layout (one solve per upload)",
            "ms_per_step": round(med_s * 1e3, 3), "statistic": "median step",
            "ms_min": round(dist.max(min(per_step)) * 1e3, 3),
            "ms_max": round(dist.max(max(per_step)) * 1e3, 3),
            "steps": a.e2e_upload_steps,
        }
        eng.set_sweep_layout("auto")
        eng.set_stream(stream.cuda_stream)

    # ---- roofline of the sweep
    peak, peak_src = measured_peak()
    bps = sweep_bytes(n, m, directed)
    avg_sweep_ms = sweep_ms_total / max(sweeps_total, 1)
    achieved = bps / (avg_sweep_ms / 1e3) / 1e9
    traffic = profiled_traffic(a.graph) if blocked else None
    # each kernel of the sweep timed on its own, in one extra solve outside the
    # timed region: CUDA events between separate launches, or, where a solve is
    # one launch, the device's clock from the first sweep to the last
    kms, ksweeps = eng.sweep_kernel_times(a.max_iters, a.epsilon)
    assert len(kms) == (3 if blocked else 1), "sweep layout changed between legs"
    knames = (["slice_partial_kernel<flat pairs>", "slice_partial_kernel<other pairs>",
               "bin_row_kernel"] if blocked
              else ["resident_solve_kernel" if one_launch else "pull_sweep_kernel"])
    kernels = [{"kernel": kn, "ms_per_sweep": round(t, 4), "share": round(t / sum(kms), 4)}
               for kn, t in zip(knames, kms)]
    if blocked:
        # bytes the slice-blocked layout moves per sweep: the stored source
        # ids (2 bytes each, padding included), per (row, slice) pair its
        # dest (4) and its partial written and read (4 + 4) and its position
        # in the bin (2); per row its pair range (4), old and new score (8),
        # next contrib (4) and degree (4); the slices' contribs (4 per vertex)
        layout_bytes = (2 * layout["ids"] + 14 * layout["pairs"] + 24 * n
                        + (4 * (n + 1) if directed else 0))
    else:
        layout_bytes = bps
    # The gather sweep's loads (one 4-byte load per edge at a random address)
    # are bounded by the rate at which L1 misses can be served, measured here
    # on an L2-resident array: the gather roofline beside the HBM one.
    if not blocked:
        from gapbs_b200.pagerank import measure_gather_rate
        gather_peak = measure_gather_rate(64 << 20, dev)
        gather_achieved = m / (avg_sweep_ms / 1e3)

    result = {
        "metric": METRIC,
        "value": round(value, 3),
        "unit": "GTEPS",
        "n_gpus": dist.world,
        "steps": a.steps,
        "warmup": a.warmup,
        "ms_per_step": round(max_ms / a.steps, 4),
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f32",
        "data": "synthetic (reference generator, identical graph)",
        "config": {
            "workload": f"PageRankPull {a.graph.strip()} (Kronecker/uniform per pr_spmv options), "
                        f"damping 0.85, epsilon {a.epsilon}, max_iters {a.max_iters}",
            "sweep_layout": ({"layout": "slice-blocked", "slices": layout["slices"],
                              "bins": layout["bins"], "pairs": layout["pairs"],
                              "stored_ids": layout["ids"], "device_bytes": layout["bytes"]}
                             if blocked else {"layout": "gather"}),
            "num_nodes": n, "num_edges_directed": m, "sweeps_per_step": sweeps_per_step,
            "l2": "256 MB buffer written between steps; graph 4M+4N bytes >> 126 MB L2",
            "parallelism": f"replicas{dist.world}" if dist.world > 1 else "single GPU",
            "graph_build_s": round(build_s, 2),
            "graph_built_on": "gpu (pr_gpu_generate)" if on_gpu else "host",
        },
        "e2e": {
            "value": round(e2e_value, 3), "unit": "GTEPS",
            "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 4 * n,
            "path": "pr_gpu_run (C ABI, host scores buffer, pinned)",
            "upload_once_s": round(upload_s, 3), "upload_once_bytes": upload_bytes,
            "graph_note": ("generated on the device once before timing"
                           if on_gpu else "uploaded once before timing"),
            "ms_per_step": round(e2e_s * 1e3 / a.steps, 4),
        },
        "roofline": {
            "kernel": ("slice-blocked sweep: " + ", ".join(knames) + " (one launch each per "
                       "sweep)") if blocked else knames[0],
            "bound": "hbm",
            "achieved": round(achieved, 1),
            "peak": peak,
            "peak_source": peak_src,
            "unit": "GB/s",
            "frac": round(achieved / peak, 4),
            "traffic": traffic,
            "algorithmic_bytes_per_sweep": bps,
            "avg_sweep_ms": round(avg_sweep_ms, 4),
            "kernels": kernels,
            "kernels_note": "average device ms per sweep of each kernel, "
                            + ("from the first sweep to the last of the one launch "
                               if one_launch else
                               "each launched on its own between CUDA events ")
                            + f"({ksweeps} sweeps, one solve outside the timed region)",
            "layout_bytes_per_sweep": int(layout_bytes),
            "layout_gbs": round(layout_bytes / (avg_sweep_ms / 1e3) / 1e9, 1),
            "layout_frac": round(layout_bytes / (avg_sweep_ms / 1e3) / 1e9 / peak, 4),
        },
        "clocks": clk,
        "gpu_launches": int(launches),
    }
    if not blocked:
        # the gather sweep's ceiling: one random 4-byte load per edge
        result["roofline"]["gather"] = {
            "achieved": round(gather_achieved / 1e9, 2),
            "peak": round(gather_peak / 1e9, 2),
            "unit": "G gathers/s",
            "frac": round(gather_achieved / gather_peak, 4),
            "peak_source": "measured in this run: random 4-byte loads (ld.global.nc) "
                           "from a 64 MB L2-resident array",
        }
    if e2e_up is not None:
        result["e2e_graph_upload_each_step"] = e2e_up
    if verify is not None:
        result["verify"] = verify
    if cc is not None:
        result["cc"] = cc
    if bfs is not None:
        result["bfs"] = bfs
    del flush

    # ---- batched PPR vs sequential single-vector solves (rank 0, N=1 config)
    if not a.no_ppr and dist.rank == 0:
        result["ppr"] = run_ppr(a, dev)
    if not a.no_adjoint and dist.rank == 0:
        result["adjoint"] = run_adjoint(a, dev)
    if not a.no_noalloc and dist.rank == 0:
        try:
            result["noalloc"] = run_noalloc(a, dev)
        except Exception as exc:  # a side leg: its failure must not lose the bench line
            result["noalloc"] = {"error": f"{type(exc).__name__}: {exc}"}

    # ---- CPU baseline on this host (rank 0 at N=1 only)
    if not a.no_cpu_baseline and dist.rank == 0 and dist.world == 1:
        if g is None:
            g = eng.download_graph()  # the generated graph, for the reference on the host
        import oracle
        rg = oracle.RefGraph.from_csr(g) if oracle.ref_available() else None
        result["cpu_baseline"] = cpu_baseline(g, a, sweeps_per_step, max_ms / a.steps, rg)
        if verify is not None and rg is not None:
            # the reference's serial PRVerifier on the same scores, at the
            # device's error e and at the next double above it: false then
            # true only when the reference's error is exactly e
            e_v = verify["error"]
            t0 = time.perf_counter()
            below_e, _ = capture_fd1(rg.verify, scores_v, e_v)
            below_next, _ = capture_fd1(rg.verify, scores_v, float(np.nextafter(e_v, np.inf)))
            sec = (time.perf_counter() - t0) / 2
            verify["reference_cpu_ms"] = round(sec * 1e3, 1)
            verify["reference_cpu_cores"] = 1
            verify["reference_error_equal"] = bool(not below_e and below_next)
            verify["speedup_vs_reference_cpu"] = round(sec * 1e3 / verify["ms"], 1)
        if bfs is not None and bfs["sources"]:
            import oracle
            if oracle.ref_available():
                _, sec = oracle.ref_bfs_csr(g, bfs["sources"])
                bfs["reference_cpu_ms"] = round(sec * 1e3 / len(bfs["sources"]), 3)
                bfs["reference_cpu_cores"] = os.cpu_count() or 1
                bfs["speedup_vs_reference_cpu"] = round(bfs["reference_cpu_ms"] / bfs["ms"], 2)
        if cc is not None:
            import oracle
            if oracle.ref_available():
                _, sec = oracle.ref_cc_afforest_csr(g, trials=2)
                cc["reference_cpu_ms"] = round(sec * 1e3, 3)
                cc["reference_cpu_cores"] = os.cpu_count() or 1
                cc["speedup_vs_reference_cpu"] = round(sec * 1e3 / cc["ms"], 2)
    eng.close()
    return result


def run_ppr(a, dev):
    import torch
    from gapbs_b200 import PageRankEngine
    from gapbs_b200.graph import make_graph
    eng = PageRankEngine(dev)
    if synthetic(a.ppr_graph):
        eng.generate(a.ppr_graph)
        g = eng.download_graph()  # host copy for the seed sets
    else:
        g = make_graph(a.ppr_graph)
        eng.upload(g)
    n, m = g.num_nodes, g.num_edges_directed
    T, sizes = ppr_teleports(g, a.ppr_cols, seed=27491095 + 1)
    stream = torch.cuda.current_stream(dev)
    eng.set_stream(stream.cuda_stream)
    Td = torch.from_numpy(T).to(f"cuda:{dev}")
    out = torch.empty_like(Td)
    cols = [torch.from_numpy(np.ascontiguousarray(T[:, c])).to(f"cuda:{dev}")
            for c in range(a.ppr_cols)]
    out1 = torch.empty(n, dtype=torch.float32, device=f"cuda:{dev}")
    reps = max(1, min(a.steps, 3))
    # batched
    for _ in range(max(1, a.warmup)):
        eng.run_device(a.max_iters, a.epsilon, 0.85, a.ppr_cols, Td.data_ptr(), out.data_ptr())
    torch.cuda.synchronize()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record(stream)
    bsweeps = None
    for _ in range(reps):
        bsweeps, _ = eng.run_device(a.max_iters, a.epsilon, 0.85, a.ppr_cols, Td.data_ptr(),
                                    out.data_ptr())
    e.record(stream)
    torch.cuda.synchronize()
    b_ms = s.elapsed_time(e) / reps
    b_gteps = float(m) * float(bsweeps.sum()) / (b_ms / 1e3) / 1e9
    # sequential single-vector solves
    for c in range(min(2, a.ppr_cols)):
        eng.run_device(a.max_iters, a.epsilon, 0.85, 1, cols[c].data_ptr(), out1.data_ptr())
    torch.cuda.synchronize()
    s.record(stream)
    ssweeps = 0
    for c in range(a.ppr_cols):
        sw, _ = eng.run_device(a.max_iters, a.epsilon, 0.85, 1, cols[c].data_ptr(), out1.data_ptr())
        ssweeps += int(sw[0])
    e.record(stream)
    torch.cuda.synchronize()
    s_ms = s.elapsed_time(e)
    s_gteps = float(m) * ssweeps / (s_ms / 1e3) / 1e9
    # agreement of the two paths (same columns, same tolerance)
    maxdiff = 0.0
    for c in range(0, a.ppr_cols, max(1, a.ppr_cols // 8)):
        eng.run_device(a.max_iters, a.epsilon, 0.85, 1, cols[c].data_ptr(), out1.data_ptr())
        maxdiff = max(maxdiff, float((out[:, c] - out1).abs().sum()))
    schedule = eng.batch_schedule()
    eng.close()
    # Roofline of the batched solve: every column-sweep gathers 4 bytes per
    # edge (one float of each neighbour's contrib row, served mostly by L2);
    # the streams are ids and offsets once per sweep step and old score, new
    # score and next contrib (12 bytes) per vertex and column-sweep.
    col_sweeps = float(bsweeps.sum())
    steps = float(bsweeps.max())
    gathered = 4.0 * m * col_sweeps
    streamed = steps * (4.0 * m + 4.0 * (n + 1)) + 12.0 * n * col_sweeps
    # the ceilings of those gathers: random 256-byte rows (a 64-column tile
    # row) with 16-byte loads from an L2-resident array and from a 1 GB one
    # (the g22 tile's size, served by HBM), measured now
    from gapbs_b200.pagerank import measure_row_gather_rate
    row_peak = measure_row_gather_rate(64 << 20, 4 * 64, dev) / 1e9
    row_peak_hbm = measure_row_gather_rate(1 << 30, 4 * 64, dev) / 1e9
    gathered_gbs = gathered / (b_ms / 1e3) / 1e9
    return {
        "workload": f"{a.ppr_cols} PPR vectors on {a.ppr_graph.strip()} (N={n}, M={m}), seed sets "
                    f"log-uniform in [1,4096] (sizes min {min(sizes)} max {max(sizes)})",
        "roofline": {
            "kernel": "batch_sweep_kernel",
            "gathered_gbs": round(gathered_gbs, 1),
            "streamed_gbs": round(streamed / (b_ms / 1e3) / 1e9, 1),
            "gather": {"achieved": round(gathered_gbs, 1), "peak": round(row_peak, 1),
                       "unit": "GB/s", "frac": round(gathered_gbs / row_peak, 4),
                       "peak_source": "measured in this run: random 256-byte rows (16-byte "
                                      "loads) from a 64 MB L2-resident array",
                       "peak_1gb_array": round(row_peak_hbm, 1),
                       "frac_1gb_array": round(gathered_gbs / row_peak_hbm, 4)},
            "note": "hub rows hit L2, the rest come from HBM (63 % L2 hit at g22 by ncu): "
                    "the rate lies between the L2-resident and the 1 GB-array row-gather "
                    "ceilings",
        },
        "schedule": dict(schedule, chosen_by="autotuner (tile width, then short-row length "
                                             "and L1 hub budget, timed on the first solve)"),
        "batched_gteps": round(b_gteps, 3),
        "batched_ms": round(b_ms, 3),
        "batched_sweeps_total": int(bsweeps.sum()),
        "sequential_gteps": round(s_gteps, 3),
        "sequential_ms": round(s_ms, 3),
        "sequential_sweeps_total": ssweeps,
        "speedup_aggregate_gteps": round(b_gteps / s_gteps, 3),
        "max_l1_batched_vs_single": maxdiff,
    }


def run_noalloc(a, dev):
    """pr_gpu_run_noalloc (the entry point that allocates nothing; its sweep
    has no degree bins) on the largest graph it takes, beside the regular
    entry point (pr_gpu_run_device) on the same graph: device buffers in and
    out, CUDA events on the stream both run on, inputs resident."""
    import ctypes
    import torch
    from gapbs_b200 import PageRankEngine
    from gapbs_b200._native import pr_lib
    eng = PageRankEngine(dev)
    n, m = eng.generate(a.noalloc_graph)
    g = eng.download_graph()
    stream = torch.cuda.current_stream(dev)
    eng.set_stream(stream.cuda_stream)
    d = f"cuda:{dev}"
    out = torch.empty(n, dtype=torch.float32, device=d)
    out_na = torch.empty(n, dtype=torch.float32, device=d)
    in_off = torch.tensor(np.asarray(g.in_offsets, np.int32), device=d)
    in_nbr = torch.tensor(np.asarray(g.in_neighbors, np.int32), device=d)
    reps = max(3, a.steps)
    sweeps = np.zeros(1, np.int32)
    msg = ctypes.create_string_buffer(256)

    def noalloc():
        rc = pr_lib().pr_gpu_run_noalloc(dev, n, m, in_off.data_ptr(), in_nbr.data_ptr(), None,
                                         a.max_iters, a.epsilon, 0.85, out_na.data_ptr(),
                                         sweeps.ctypes.data, None, stream.cuda_stream, msg, 256)
        if rc != 0:
            raise RuntimeError(f"pr_gpu_run_noalloc: {rc} {msg.value.decode()}")
        return int(sweeps[0])

    def regular():
        sw, _ = eng.run_device(a.max_iters, a.epsilon, 0.85, 1, None, out.data_ptr())
        return int(sw[0])

    timed = {}
    for name, fn in (("regular", regular), ("noalloc", noalloc)):
        for _ in range(max(1, a.warmup)):
            fn()
        torch.cuda.synchronize()
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record(stream)
        total = sum(fn() for _ in range(reps))
        e.record(stream)
        torch.cuda.synchronize()
        ms = s.elapsed_time(e) / reps
        timed[name] = (ms, total / reps)
    ref = out.cpu().numpy().astype(np.float64)
    got = out_na.cpu().numpy().astype(np.float64)
    eng.close()
    (r_ms, r_sw), (n_ms, n_sw) = timed["regular"], timed["noalloc"]
    return {"workload": f"PageRankPull {a.noalloc_graph.strip()} (N={n}, M={m}) through "
                        "pr_gpu_run_noalloc, beside pr_gpu_run_device",
            "noalloc_ms": round(n_ms, 3), "noalloc_gteps": round(m * n_sw / n_ms / 1e6, 2),
            "regular_ms": round(r_ms, 3), "regular_gteps": round(m * r_sw / r_ms / 1e6, 2),
            "sweeps": n_sw, "regular_sweeps": r_sw,
            "max_rel_diff": float(np.max(np.abs(got - ref) / np.maximum(np.abs(ref), 1e-30))),
            "statistic": f"mean of {reps} solves (CUDA events, device buffers)"}


def run_adjoint(a, dev):
    """Reverse-mode solve of L = w . s on a weighted graph: forward PPR, then
    the adjoint sweeps and the edge-weight gradient pass, timed with CUDA
    events (host buffers excluded: device-pointer entry points)."""
    import torch
    from gapbs_b200 import PageRankEngine
    eng = PageRankEngine(dev)
    eng.generate(a.adjoint_graph)
    g = eng.download_graph()
    n, m = g.num_nodes, g.num_edges_directed
    rng = np.random.default_rng(27491095 + 3)
    ew = rng.uniform(0.5, 1.5, m).astype(np.float32)
    eng.upload(g, edge_w=ew)
    stream = torch.cuda.current_stream(dev)
    eng.set_stream(stream.cuda_stream)
    t = torch.from_numpy(ppr_teleports(g, 1, seed=27491095 + 3)[0][:, 0].copy()).to(f"cuda:{dev}")
    s = torch.empty(n, dtype=torch.float32, device=f"cuda:{dev}")
    w = torch.from_numpy(rng.normal(size=n).astype(np.float32)).to(f"cuda:{dev}")
    gt = torch.empty(n, dtype=torch.float32, device=f"cuda:{dev}")
    ge = torch.empty(m, dtype=torch.float32, device=f"cuda:{dev}")
    fsw = asw = 0
    for _ in range(max(1, a.warmup)):
        eng.run_device(100, 1e-7, 0.85, 1, t.data_ptr(), s.data_ptr())
        eng.adjoint_device(300, 1e-7, 0.85, w.data_ptr(), s.data_ptr(), gt.data_ptr(),
                           ge.data_ptr())
    torch.cuda.synchronize()
    e0, e1, e2 = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    e0.record(stream)
    fsw, _ = eng.run_device(100, 1e-7, 0.85, 1, t.data_ptr(), s.data_ptr())
    e1.record(stream)
    asw = eng.adjoint_device(300, 1e-7, 0.85, w.data_ptr(), s.data_ptr(), gt.data_ptr(),
                             ge.data_ptr())
    e2.record(stream)
    torch.cuda.synchronize()
    f_ms, a_ms = e0.elapsed_time(e1), e1.elapsed_time(e2)
    eng.close()
    asw = int(asw)
    # a training loop through torch.autograd: forward, backward, SGD step on
    # the edge weights; the graph is uploaded once, each later step hands
    # the new weights to the engine from device memory
    from gapbs_b200.autograd import PageRankContext, personalized_pagerank
    pctx = PageRankContext(g, device=dev, max_iters=100, epsilon=1e-7, adjoint_max_iters=300,
                           adjoint_epsilon=1e-7)
    wt = torch.tensor(ew, device=f"cuda:{dev}", requires_grad=True)

    def train_step():
        sp = personalized_pagerank(t, wt, pctx)
        loss = (w * sp).sum()
        wt.grad = None
        loss.backward()
        with torch.no_grad():
            wt.sub_(1e3 * wt.grad)
            wt.clamp_(min=0.05)

    train_step()  # warm-up: the one graph upload
    torch.cuda.synchronize()
    steps = 10
    t0 = time.perf_counter()
    for _ in range(steps):
        train_step()
    torch.cuda.synchronize()
    train_ms = (time.perf_counter() - t0) * 1e3 / steps
    train = {"steps": steps, "ms_per_step": round(train_ms, 3),
             "graph_uploads_in_timed_steps": pctx.uploads - 1,
             "device_weight_updates_in_timed_steps": pctx.weight_updates,
             "host_device_graph_bytes_per_step": 0,
             "path": "torch.autograd (personalized_pagerank) forward + backward + SGD on edge "
                     "weights; pr_gpu_set_edge_weights_device each step"}
    pctx.engine.close()
    # adjoint sweeps read ids, weights and offsets of the out-rows (8M + 4(N+1))
    # plus 16N of vectors; the gradient pass reads 8M and writes 4M
    adj_bytes = asw * (8.0 * m + 4.0 * (n + 1) + 16.0 * n) + 12.0 * m
    return {
        "workload": f"weighted PPR adjoint on {a.adjoint_graph} (N={n}, M={m}), weights "
                    f"U[0.5,1.5], loss weights N(0,1), epsilon 1e-7",
        "forward_sweeps": int(fsw[0]), "forward_ms": round(f_ms, 3),
        "adjoint_sweeps": asw, "adjoint_ms": round(a_ms, 3),
        "autograd_training": train,
        "adjoint_gteps": round(m * asw / (a_ms / 1e3) / 1e9, 2),
        "adjoint_algorithmic_gbs": round(adj_bytes / (a_ms / 1e3) / 1e9, 1),
    }


def cpu_baseline(g, a, gpu_sweeps, gpu_ms_per_solve, rg=None):
    import oracle
    cores = os.cpu_count() or 1
    n, m = g.num_nodes, g.num_edges_directed
    if rg is not None:
        tot, per = rg.time_pagerank_pull(trials=a.cpu_trials, max_iters=a.max_iters,
                                         epsilon=a.epsilon)
        sweeps = gpu_sweeps
        sec = float(np.mean(per))
        # the reference's pr benchmark: Gauss-Seidel PageRankPullGS on the
        # same graph (its own convergence test, fewer sweeps), for time to
        # solution
        _, log = capture_fd1(rg.pagerank_gs, a.max_iters, a.epsilon, True)
        gs_sweeps = len([ln for ln in log.splitlines() if ln.strip()])
        _, gper = rg.time_pagerank_gs(trials=a.cpu_trials, max_iters=a.max_iters,
                                      epsilon=a.epsilon)
        gsec = float(np.mean(gper))
        return {"value": round(m * sweeps / sec / 1e9, 4), "unit": "GTEPS", "cores": cores,
                "kind": "reference",
                "sample": f"{a.cpu_trials} full PageRankPull solves of the same graph "
                          f"({sweeps:.0f} sweeps each) by the reference compiled from source, "
                          f"OpenMP on {cores} threads; {sec:.3f} s per solve",
                "gauss_seidel": {
                    "kernel": "PageRankPullGS (src/pr.cc:34-61), the reference's pr benchmark",
                    "value": round(m * gs_sweeps / gsec / 1e9, 4), "unit": "GTEPS",
                    "sweeps": gs_sweeps, "s_per_solve": round(gsec, 4), "cores": cores,
                    "sample": f"{a.cpu_trials} full solves of the same graph, OpenMP on "
                              f"{cores} threads",
                    "gpu_speedup_time_to_solution": round(gsec * 1e3 / gpu_ms_per_solve, 2),
                }}
    # port: single-threaded FP32 oracle, 2 sweeps
    t0 = time.perf_counter()
    _, k, _ = oracle.pr_pull_f32(g, max_iters=2, epsilon=0.0)
    sec = time.perf_counter() - t0
    return {"value": round(m * k / sec / 1e9, 4), "unit": "GTEPS", "cores": 1, "kind": "port",
            "sample": f"2 sweeps of the FP32 restatement, one thread, {sec:.3f} s"}


# ---------------------------------------------------------------------------
# reference arm

def capture_fd1(fn, *args):
    sys.stdout.flush()
    saved = os.dup(1)
    with tempfile.TemporaryFile(mode="w+b") as tmp:
        os.dup2(tmp.fileno(), 1)
        try:
            ret = fn(*args)
        finally:
            sys.stdout.flush()
            os.dup2(saved, 1)
            os.close(saved)
        tmp.seek(0)
        return ret, tmp.read().decode()


def run_reference(a, dist: Dist):
    if dist.rank != 0:
        return None
    import oracle
    cores = os.cpu_count() or 1
    if not oracle.ref_available():
        # the oracle port stands in (single-threaded FP32 restatement)
        from gapbs_b200.graph import make_graph
        g = make_graph(a.graph)
        m = g.num_edges_directed
        per = []
        for i in range(a.warmup + a.steps):
            t0 = time.perf_counter()
            _, k, _ = oracle.pr_pull_f32(g, max_iters=2, epsilon=0.0)
            if i >= a.warmup:
                per.append((time.perf_counter() - t0, k))
        sec = sum(p[0] for p in per)
        val = m * sum(p[1] for p in per) / sec / 1e9
        ms_step = sec * 1e3 / a.steps
        kind, sample, cores_used = "port", "2 sweeps per step, FP32 restatement, one thread", 1
    else:
        rg, _ = capture_fd1(oracle.RefGraph.build, a.graph)
        m = rg.num_edges_directed
        s, log = capture_fd1(rg.pagerank_pull, a.max_iters, a.epsilon, True)
        sweeps = len([ln for ln in log.splitlines() if ln.strip()])
        for _ in range(a.warmup):
            rg.time_pagerank_pull(trials=1, max_iters=a.max_iters, epsilon=a.epsilon)
        tot, per = rg.time_pagerank_pull(trials=a.steps, max_iters=a.max_iters, epsilon=a.epsilon)
        val = m * sweeps * a.steps / tot / 1e9
        ms_step = tot * 1e3 / a.steps
        kind, cores_used = "reference", cores
        sample = (f"each step one full PageRankPull solve ({sweeps} sweeps) of {a.graph.strip()} "
                  f"by the reference compiled from source, OpenMP on {cores} threads")
    out = {
        "impl": "reference",
        "metric": METRIC,
        "value": round(val, 4),
        "unit": "GTEPS",
        "n_gpus": dist.world,
        "steps": a.steps,
        "warmup": a.warmup,
        "ms_per_step": round(ms_step, 4),
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f32",
        "data": "synthetic (reference generator)",
        "config": {"workload": f"PageRankPull {a.graph.strip()}, damping 0.85, epsilon "
                               f"{a.epsilon}, max_iters {a.max_iters}"},
        "cpu_baseline": {"value": round(val, 4), "unit": "GTEPS", "cores": cores_used,
                         "kind": kind, "sample": sample},
        "e2e": {"value": round(val, 4), "unit": "GTEPS", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    return out


def main():
    a = parse_args()
    # The reference arm runs on rank 0 alone and needs no process group.
    dist = Dist(init=a.impl != "reference")
    try:
        if a.impl == "reference":
            res = run_reference(a, dist)
        else:
            res = run_ours(a, dist)
        if dist.rank == 0 and res is not None:
            print(json.dumps(res), flush=True)
    finally:
        dist.close()


if __name__ == "__main__":
    main()
