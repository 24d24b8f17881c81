"""Benchmark of the GB300 network RHS on the large-graph throughput workload.

Workload: diffusion on a Barabási–Albert graph, N = 10,000,000 vertices, m = 4
(E ≈ 4e7 edges, power-law hubs), e = w_ij (u_src - u_dst) with w ~ U(0,1), du = Σ e,
u ~ N(0,1), seeded synthetic inputs.  One step = one RHS evaluation `nw(du, u, p, t)`.
The headline line is FP64 (bitwise equal to the sequential reference order); the same
JSON line carries the FP32 run (compensated sums at hubs), the end-to-end figure through
the public API with host buffers, the HBM roofline of the RHS kernel, and the CPU
baseline (the oracle restatement of SequentialExecution / PolyesterExecution).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl gb300|reference]

Under torchrun every rank runs an independent replica (the single-graph RHS does not
shard); value = edges processed by all ranks / max time over ranks.
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
sys.path.insert(0, str(ROOT / "networkdynamics.jl_gb300"))
sys.path.insert(0, str(ROOT))

METRIC = "RHS edges/s (% HBM peak) @10M-vertex"
HEAVY_MIN_DEGREE = 2049  # rows this long run in the heavy-row kernel (kMediumMaxDeg + 1)
NV_DEFAULT = 10_000_000
M_BA = 4
SEED = 1


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=2000)
    ap.add_argument("--warmup", type=int, default=10)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--nv", type=int, default=NV_DEFAULT, help="vertices (smaller for profiling captures)")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline leg")
    ap.add_argument("--no-f32", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-ensemble", action="store_true",
                    help="skip the basin-stability ensemble (FP32 vs FP64 solves/s) leg")
    ap.add_argument("--no-warmstart", action="store_true", help="skip the learned warm-start leg")
    ap.add_argument("--no-dense", action="store_true", help="skip the reference's dense diffusion case")
    ap.add_argument("--cases", action="store_true",
                    help="instead of the headline workload: the reference's benchmark cases at their largest size, "
                         "one JSON line each")
    return ap.parse_args()


def algorithmic_bytes(nv, ne, s):
    """Bytes one RHS must move at ideal caching: read u, write du, read p (w per edge),
    read the CSR row pointers (4 B per vertex) and the incidences (nbr + eid, 8 B each)."""
    return s * (nv + nv + ne) + 4 * (nv + 1) + 2 * ne * 8


def peaks():
    try:
        d = json.loads((ROOT / "MEASURED_PEAKS.json").read_text())
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


def kernel_bytes(g, s):
    """Algorithmic bytes (and FP64 lane operations) of one launch of each RHS kernel for
    diffusion edges with s-byte values.
      edge phase  per edge: src, dst (4 B each), staging slot (2 B); u_src, u_dst, w, y, ybkt (s each)
      row phase   per row: its 16-byte record and du (s); per destination-side incidence its
                  ybkt position (4 B) + ybkt (s); per source-side y (s)
      heavy rows  per row: slot vertex, slot pointer pair (12 B), u_v and du (s each);
                  per incidence the (nbr, eid) pair (8 B), u_nbr and w (s each)
      fused       the whole RHS (algorithmic_bytes)
    Rows of degree > 2048 are the heavy rows."""
    nv, ne = g.nv, g.ne
    ndst = np.bincount(g.dst, minlength=nv)
    nsrc = np.bincount(g.src, minlength=nv)
    heavy = (ndst + nsrc) > HEAVY_MIN_DEGREE - 1
    light = ~heavy
    nh, inc_h = int(heavy.sum()), int((ndst + nsrc)[heavy].sum())
    rows = int(light.sum()) * (16 + s) + int(ndst[light].sum()) * (4 + s) + int(nsrc[light].sum()) * s
    return {
        "edge_phase": (ne * (10 + 5 * s), 2 * ne),
        "row_phase": (rows, int((ndst + nsrc)[light].sum())),
        "heavy_rows": (nh * (12 + 2 * s) + inc_h * (8 + 2 * s), 3 * inc_h),
        "fused": (algorithmic_bytes(nv, ne, s), 3 * 2 * ne),
    }


def profiled_traffic(dtype_tag, nv):
    """DRAM bytes of one RHS from the committed ncu summary of this workload: lines
    `traffic_bytes_per_launch <kernel>: <bytes>`, summed over the kernels; None when absent."""
    f = ROOT / "profiles" / f"rhs_ba{nv // 1_000_000}m_{dtype_tag}.txt"
    if not f.exists():
        return None
    key = "traffic_bytes_per_launch "
    per = {}
    for line in f.read_text().splitlines():
        if line.startswith(key):
            name, _, val = line[len(key):].partition(":")
            try:
                per[name.strip()] = float(val.strip())
            except ValueError:
                pass
    if not per:
        return None
    return {"total": sum(per.values()), "kernels": per, "source": f"profiles/{f.name}"}


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    def __init__(self, index=0):
        self.index = index
        self.samples = []
        self.proc = None

    def __enter__(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={q}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except Exception:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.samples.append([x.strip() for x in line.split(",")])

    def __exit__(self, *exc):
        if self.proc is not None:
            time.sleep(0.25)
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(s[1]) for s in self.samples if len(s) > 2 and s[1].replace(".", "").isdigit()]
        mx = [float(s[2]) for s in self.samples if len(s) > 2 and s[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for s in self.samples:
            for k, name in enumerate(names):
                if len(s) > 5 + k and s[5 + k].lower().startswith("active"):
                    reasons.add(name)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(self.samples)}


def make_workload(nv):
    import nd_gb300 as nd
    g = nd.barabasi_albert(nv, M_BA, seed=SEED)
    u, w = make_inputs(nv, g.ne)
    return g, u, w


def dist_setup(args):
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist
        backend = "gloo" if args.impl == "reference" else "nccl"
        if backend == "nccl":
            import torch
            torch.cuda.set_device(local)
        dist.init_process_group(backend=backend)
    return rank, world, local


def barrier(world):
    if world > 1:
        import torch.distributed as dist
        dist.barrier()


def max_over_ranks(x, world, device=None):
    if world == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def cpu_baseline(g, u, w, seconds=12.0):
    """The oracle on the host cores: the PolyesterExecution restatement on all threads and
    the SequentialExecution restatement on one, each on whole RHS evaluations."""
    from oracle import oracle as O
    on = O.OracleNetwork.from_graph(g, O.V_DIFFUSION, O.E_DIFFUSION)
    res = {}
    for name, fn, threads in (("poly", on.rhs_poly, os.cpu_count() or 1), ("seq", on.rhs, 1)):
        O.load().nd_oracle_set_num_threads(threads)
        fn(u, w)  # warm
        n, t0 = 0, time.perf_counter()
        while True:
            fn(u, w)
            n += 1
            el = time.perf_counter() - t0
            if el > seconds / 2 or n >= 50:
                break
        res[name] = (g.ne * n / el, n, threads, el)
    O.load().nd_oracle_set_num_threads(os.cpu_count() or 1)
    return res


def workload_config(g):
    """The config dict both arms print: the workload and its sizes, nothing arm-specific."""
    deg = np.bincount(g.src, minlength=g.nv) + np.bincount(g.dst, minlength=g.nv)
    B = algorithmic_bytes(g.nv, g.ne, 8)
    return {"workload": f"diffusion on Barabasi-Albert N={g.nv}, m={M_BA}, F64 RHS", "nv": g.nv, "ne": g.ne,
            "incidences": 2 * g.ne, "max_degree": int(deg.max()), "hub_rows": int((deg > 32).sum()),
            "sum_order": "sequential (bitwise = SequentialAggregator)",
            "l2": "no flush: inputs+topology %.2f GB > 129 MB L2" % (B / 1e9)}


def make_inputs(nv, ne):
    rng = np.random.default_rng(SEED)
    return rng.normal(size=nv), rng.uniform(0.0, 1.0, size=ne)


def run_reference(args, rank, world):
    """CPU reference arm: the threaded oracle restatement (PolyesterExecution +
    PolyesterAggregator) on all host cores, same workload, config and metric.  It loads
    nothing of the package: the graph comes from the oracle's copy of the generator."""
    if rank != 0:
        return
    from oracle import oracle as O
    g = O.barabasi_albert(args.nv, M_BA, SEED)
    u, w = make_inputs(g.nv, g.ne)
    on = O.OracleNetwork.from_graph(g, O.V_DIFFUSION, O.E_DIFFUSION)
    threads = os.cpu_count() or 1
    O.load().nd_oracle_set_num_threads(threads)
    for _ in range(max(args.warmup, 3)):
        on.rhs_poly(u, w)
    # each step is one full RHS; a run asked for more steps than ~3 minutes of host time
    # holds is cut to that many (the line says how many ran)
    t0 = time.perf_counter()
    on.rhs_poly(u, w)
    one = time.perf_counter() - t0
    steps = max(1, min(args.steps, int(180.0 / max(one, 1e-6))))
    t0 = time.perf_counter()
    for _ in range(steps):
        on.rhs_poly(u, w)
    el = time.perf_counter() - t0
    val = g.ne * steps / el
    line = {
        "impl": "reference", "metric": METRIC, "value": val, "unit": "edges/s", "n_gpus": args.gpus,
        "steps": steps, "warmup": max(args.warmup, 3), "ms_per_step": 1e3 * el / steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic (seeded BA graph, w~U(0,1), u~N(0,1))", "config": workload_config(g),
        "execution": f"host threads ({threads})",
        "cpu_baseline": {"value": val, "unit": "edges/s", "cores": threads, "kind": "port",
                         "sample": f"{steps} full RHS evaluations (at most ~3 minutes of host time) of the "
                                   "PolyesterExecution+PolyesterAggregator restatement"},
        "e2e": {"value": val, "unit": "edges/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def secondary_leg(line, key, leg):
    """line[key] = leg(), or the error: a secondary leg never costs the headline line."""
    try:
        line[key] = leg()
    except Exception as exc:
        line[key] = {"error": f"{type(exc).__name__}: {exc}"}


def ensemble_leg():
    """Ensemble solves/s, FP32 vs FP64; raises where a state is not a solution."""
    from nd_gb300 import benchmarks as NB
    ens = NB.ensemble(4096)
    keys = ("synchronised_median", "synchronised_p95", "synchronised_max", "synchronised_within_1e-6",
            "median_instance", "instances_within_1e-6", "desynchronised_median", "sync_verdict_agreement")
    return {
        "metric": "ensemble solves/s FP32 vs FP64 @1e-6", "workload": ens["workload"],
        "instances": 4096, "sync_fraction_f64": ens["sync_fraction_f64"],
        "solves_per_s_f32_batched": ens["f32"]["solves_per_s"],
        "solves_per_s_f32x2_batched": ens["f32x2"]["solves_per_s"],
        "solves_per_s_f64_batched": ens["f64"]["solves_per_s"],
        "solves_per_s_plain_f64": ens["plain_f64_per_instance"]["solves_per_s"],
        "f32_batched_vs_plain_f64": ens["f32_batched_vs_plain_f64"],
        "f32x2_batched_vs_plain_f64": ens["f32x2_batched_vs_plain_f64"],
        "f32_batched_vs_f64_batched": ens["f32"]["solves_per_s"] / ens["f64"]["solves_per_s"],
        "final_state_err_vs_f64": {k: {x: ens[f"{k}_final_state_err_vs_f64"][x] for x in keys}
                                   for k in ("f32", "f32x2", "f64_1ulp", "f64_f32params")},
        "note": "f32: FP32 RHS on FP32 parameters; f32x2: double-float RHS (pairs of floats on the FP32 "
                "pipe) on FP64 parameters; f64_1ulp / f64_f32params: FP64 solves with the parameters "
                "perturbed by one ulp / rounded to FP32 (the sensitivity floor); state, error norm and "
                "step control are FP64 in every run",
        "details": ens}


def dense_case_leg(dev, steps=200):
    """The reference's dense diffusion benchmark case (diffusion_static_edge at its largest N,
    WS(3000, 1500): rows of 1500 terms), FP64 and FP32: device time per RHS over back-to-back
    calls on resident buffers, as `bench.py --cases` times it."""
    import torch

    import nd_gb300 as nd
    name, N = CASES[0]
    g, vm, em = _case_networks(N, name)
    net = nd.Network(g, vm, em)
    u, p = case_inputs(name, net, g)
    out = {"case": name, "N": N, "ne": g.ne, "steps": steps}
    stream = torch.cuda.current_stream(dev)
    for tag, dt in (("f64", torch.float64), ("f32", torch.float32)):
        nw = nd.adapt(net, dt)
        ut = torch.from_numpy(u).to(dev, dt)
        pt = torch.from_numpy(p).to(dev, dt) if net.pdim else None
        du = torch.empty_like(ut)
        for _ in range(5):
            nw(du, ut, pt, 0.0, stream=stream)
        torch.cuda.synchronize(dev)
        el = time_device(nw, du, ut, pt, steps, stream)
        out[tag] = {"rhs_us": 1e6 * el / steps, "edges_per_s": g.ne * steps / el}
        del nw, ut, pt, du
    return out


def time_device(nw, du, u, p, steps, stream):
    import torch
    start = torch.cuda.Event(enable_timing=True)
    stop = torch.cuda.Event(enable_timing=True)
    start.record(stream)
    for _ in range(steps):
        nw(du, u, p, 0.0, stream=stream)
    stop.record(stream)
    stop.synchronize()
    return start.elapsed_time(stop) / 1e3


def run_gb300(args, rank, world, local):
    import torch

    import nd_gb300 as nd
    dev = torch.device(f"cuda:{local}")
    torch.cuda.set_device(dev)
    g, u_h, w_h = make_workload(args.nv)
    nv, ne = g.nv, g.ne
    stream = torch.cuda.current_stream(dev)
    net = nd.Network(g, nd.diffusion_vertex(), nd.diffusion_edge())
    nw = nd.adapt(net, torch.float64)
    info = nw.info()
    u = torch.from_numpy(u_h).to(dev)
    p = torch.from_numpy(w_h).to(dev)
    du = torch.empty_like(u)
    for _ in range(max(args.warmup, 3)):
        nw(du, u, p, 0.0)
    torch.cuda.synchronize()
    nw.kernel_times()  # reset the launch counters
    barrier(world)
    with ClockSampler(local) as clk:
        torch.cuda.synchronize()
        barrier(world)
        t = time_device(nw, du, u, p, args.steps, stream)
        torch.cuda.synchronize()
        barrier(world)
    counts = nw.kernel_times()
    t = max_over_ranks(t, world, dev)
    ms = 1e3 * t / args.steps
    value = world * ne * args.steps / t
    hbm, peak_kind = peaks()
    B = algorithmic_bytes(nv, ne, 8)
    # per-kernel device times: the same RHS again with every launch bracketed by CUDA events
    kt = min(args.steps, 500)
    nw.set_kernel_timing(True)
    time_device(nw, du, u, p, kt, stream)
    times = nw.kernel_times()
    nw.set_kernel_timing(False)
    kb = kernel_bytes(g, 8)
    kernels = {}
    for kind, (n, tot) in times.items():
        if n == 0:
            continue
        avg = tot / 1e3 / n
        kbytes, kops = kb[kind]
        kernels[kind] = {"launches": n, "avg_ms": 1e3 * avg, "share": None, "bytes_per_launch": kbytes,
                         "achieved_gbs": kbytes / avg / 1e9, "fp64_lane_ops_per_launch": kops}
    # heavy rows run on the handle's side stream, overlapped with the other kernels: the
    # dominant kernel is the longest one on the caller's stream (the critical path), and
    # shares are over those kernels (the ncu launch list serialises every launch)
    main = [k for k in kernels if k != "heavy_rows"]
    total_ms = sum(kernels[k]["avg_ms"] * kernels[k]["launches"] for k in main)
    for kind, k in kernels.items():
        k["stream"] = "side (overlapped)" if kind == "heavy_rows" else "caller"
        k["share"] = k["avg_ms"] * k["launches"] / total_ms if (total_ms and kind in main) else None
    dom = max(main, key=lambda k: kernels[k]["avg_ms"] * kernels[k]["launches"])
    traffic = profiled_traffic("f64", nv)
    rhs_gbs = B / (t / args.steps) / 1e9
    line = {
        "metric": METRIC, "value": value, "unit": "edges/s", "n_gpus": world, "steps": args.steps,
        "warmup": max(args.warmup, 3), "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded BA graph, w~U(0,1), u~N(0,1))",
        "config": workload_config(g),
        "execution": "replicas, one per GPU" if world > 1 else "single GPU",
        "edges_per_s": value, "incidences_per_s": 2 * value, "rhs_evals_per_s": world * args.steps / t,
        "roofline": {"bound": "hbm", "kernel": "whole RHS (%s)" % " + ".join(kernels), "achieved": rhs_gbs,
                     "peak": hbm, "unit": "GB/s", "frac": rhs_gbs / hbm, "peak_kind": peak_kind,
                     "algorithmic_bytes_per_rhs": B,
                     "traffic": traffic["total"] if traffic else None,
                     "traffic_per_kernel": traffic["kernels"] if traffic else None,
                     "traffic_source": traffic["source"] if traffic else None,
                     "dominant_kernel": dom, "kernels": kernels,
                     "note": "achieved = the RHS's algorithmic bytes 8(2N+E) + 4(N+1) + 16E (read u, write du, "
                             "read w; CSR row pointers and incidences, each byte once) / timed ms_per_step; "
                             "traffic = DRAM bytes of one RHS, summed over its kernels, from the committed ncu "
                             "summary; kernels[*].bytes_per_launch are each kernel's own design bytes "
                             "(intermediate buffers included), timed over %d event-bracketed RHS calls" % kt},
        "gpu_launches": sum(n for n, _ in counts.values()),
        "gpu_launches_by_kernel": {k: n for k, (n, _) in counts.items() if n},
    }
    # the other FP64 summation modes, for comparison (same workload, fewer steps)
    ks = min(args.steps, 200)
    modes = {}
    for mode in ("sequential_hw", "tree"):
        nw.set_sum_order(mode)
        nw(du, u, p, 0.0)
        tm = time_device(nw, du, u, p, ks, stream)
        modes[mode] = {"ms_per_step": 1e3 * tm / ks, "edges_per_s": ne * ks / tm}
    nw.set_sum_order("sequential")
    # the single fused kernel over the destination-sorted CSR (every incidence evaluates its
    # edge from u and p; the layout for edge lists in any order)
    nw.set_layout("fused")
    nw(du, u, p, 0.0)
    tm = time_device(nw, du, u, p, ks, stream)
    fused_out = du.clone()
    nw.set_layout("auto")
    nw(du, u, p, 0.0)
    torch.cuda.synchronize()
    modes["fused"] = {"ms_per_step": 1e3 * tm / ks, "edges_per_s": ne * ks / tm,
                      "same_bits_as_two_phase": bool(torch.equal(fused_out, du))}
    del fused_out
    line["f64_modes"] = modes
    # FP32 variant (compensated sums at hubs)
    if not args.no_f32:
        nw32 = nd.adapt(net, torch.float32)
        u32, p32 = u.float(), p.float()
        du32 = torch.empty_like(u32)
        for _ in range(3):
            nw32(du32, u32, p32, 0.0)
        torch.cuda.synchronize()
        t32 = time_device(nw32, du32, u32, p32, args.steps, stream)
        t32 = max_over_ranks(t32, world, dev)
        B32 = algorithmic_bytes(nv, ne, 4)
        ref = torch.empty_like(u)
        nw(ref, u, p, 0.0)
        err = (du32.double() - ref).abs().max().item()
        nw32.kernel_times()
        nw32.set_kernel_timing(True)
        time_device(nw32, du32, u32, p32, min(args.steps, 200), stream)
        kt32 = nw32.kernel_times()
        nw32.set_kernel_timing(False)
        line["f32"] = {"value": world * ne * args.steps / t32, "unit": "edges/s", "ms_per_step": 1e3 * t32 / args.steps,
                       "achieved_gbs": B32 / (t32 / args.steps) / 1e9,
                       "frac": B32 / (t32 / args.steps) / 1e9 / hbm, "max_abs_err_vs_f64": err,
                       "kernels_avg_ms": {k: tot / n for k, (n, tot) in kt32.items() if n}}
        traffic32 = profiled_traffic("f32", nv)
        if traffic32:
            line["f32"].update({"traffic": traffic32["total"], "traffic_per_kernel": traffic32["kernels"],
                                "traffic_source": traffic32["source"]})
        del nw32, u32, p32, du32
    # end to end through the public API with pinned host buffers: every step copies its
    # inputs (u, p) host->device and its result du device->host.  Two buffer sets and
    # three streams pipeline step k's RHS with step k+1's upload and step k-1's download.
    if not args.no_e2e:
        ke = min(args.steps, 200)
        uh = torch.from_numpy(u_h).pin_memory()
        ph = torch.from_numpy(w_h).pin_memory()
        duh = [torch.empty(nv, dtype=torch.float64).pin_memory() for _ in range(2)]
        ub = [u, torch.empty_like(u)]
        pb = [p, torch.empty_like(p)]
        dub = [du, torch.empty_like(du)]
        s_up = torch.cuda.Stream(dev)
        s_down = torch.cuda.Stream(dev)
        ev = lambda: torch.cuda.Event()  # noqa: E731
        uploaded = [ev(), ev()]
        computed = [ev(), ev()]
        downloaded = [ev(), ev()]

        def e2e_steps(k):
            for i in range(k):
                b = i & 1
                with torch.cuda.stream(s_up):
                    if i >= 2:
                        s_up.wait_event(computed[b])  # buffers b are free once step i-2's RHS ran
                    ub[b].copy_(uh, non_blocking=True)
                    pb[b].copy_(ph, non_blocking=True)
                    uploaded[b].record(s_up)
                stream.wait_event(uploaded[b])
                if i >= 2:
                    stream.wait_event(downloaded[b])  # du buffer b was read back
                nw(dub[b], ub[b], pb[b], 0.0, stream=stream)
                computed[b].record(stream)
                with torch.cuda.stream(s_down):
                    s_down.wait_event(computed[b])
                    duh[b].copy_(dub[b], non_blocking=True)
                    downloaded[b].record(s_down)
            stream.wait_stream(s_down)

        e2e_steps(4)
        torch.cuda.synchronize()
        barrier(world)
        start = torch.cuda.Event(enable_timing=True)
        stop = torch.cuda.Event(enable_timing=True)
        start.record(stream)
        e2e_steps(ke)
        stop.record(stream)
        stop.synchronize()
        te = max_over_ranks(start.elapsed_time(stop) / 1e3, world, dev)
        line["e2e"] = {"value": world * ne * ke / te, "unit": "edges/s", "steps": ke,
                       "h2d_bytes_per_step": int(uh.numel() * 8 + ph.numel() * 8),
                       "d2h_bytes_per_step": int(duh[0].numel() * 8),
                       "pipeline": "2 buffer sets; upload, RHS and download on 3 streams"}
        torch.cuda.synchronize()
        ok = np.array_equal(duh[(ke - 1) & 1].numpy(), dub[(ke - 1) & 1].cpu().numpy())
        line["e2e"]["result_matches_device"] = bool(ok)
    line["clocks"] = clk.summary()
    if world == 1 and not args.no_dense:
        secondary_leg(line, "reference_dense_case", lambda: dense_case_leg(dev))
    # the second half of the headline metric: ensemble solves/s, FP32 vs FP64, and the
    # learned warm start (single-GPU runs; the instances are independent replicas)
    if world == 1 and not (args.no_ensemble and args.no_warmstart):
        from nd_gb300 import benchmarks as NB
        del nw, u, p, du
        torch.cuda.empty_cache()
        if not args.no_ensemble:
            secondary_leg(line, "ensemble", ensemble_leg)
            torch.cuda.empty_cache()
        if not args.no_warmstart:
            secondary_leg(line, "warm_start", lambda: {
                "metric": "Newton iterations to residual 1e-10, cold / warm", **NB.warmstart()})
            torch.cuda.empty_cache()
    if rank == 0 and world == 1 and not args.no_cpu:
        res = cpu_baseline(g, u_h, w_h)
        v, n, thr, el = res["poly"]
        line["cpu_baseline"] = {"value": v, "unit": "edges/s", "cores": thr, "kind": "port",
                                "sample": f"{n} full RHS evaluations ({el:.1f} s) of the threaded "
                                          "PolyesterExecution+PolyesterAggregator restatement"}
        v1, n1, _, el1 = res["seq"]
        line["cpu_baseline_sequential"] = {"value": v1, "unit": "edges/s", "cores": 1, "kind": "port",
                                           "sample": f"{n1} full RHS evaluations ({el1:.1f} s) of the "
                                                     "SequentialExecution+SequentialAggregator restatement"}
    if rank == 0:
        print(json.dumps(line), flush=True)


# The reference's benchmark cases (benchmark/benchmark_cases.jl:20-102) at their largest N.
# Graphs.jl's watts_strogatz(N, 3, 0.8) links div(3, 2) = 1 ring neighbour per side before
# rewiring, which is k = 2 here.  powergrid_inhomogeneous_pq gives every PQ bus its own
# component, so 50,001 vertex batches at N = 10^5.
def _case_networks(N, name):
    import nd_gb300 as nd
    if name == "diffusion_static_edge":
        return nd.watts_strogatz(N, N // 2, 0.0, seed=1), nd.diffusion_vertex(), nd.diffusion_edge_unit()
    if name == "diffusion_ode_edge":
        return nd.watts_strogatz(N, N // 2, 0.0, seed=1), nd.diffusion_vertex(), nd.diffusion_dedge()
    g = nd.watts_strogatz(N, 2, 0.8, seed=1)
    if name == "kuramoto_homogeneous":
        return g, nd.kuramoto_vertex_2d(), nd.static_kuramoto_edge()
    if name == "powergrid":
        kinds = np.random.default_rng(1).permutation(np.repeat([0, 1], N // 2))
        return g, [nd.pqnode() if k == 0 else nd.generator() for k in kinds], nd.piline()
    if name == "powergrid_inhomogeneous_pq":  # every PQ bus closes over its own P, Q
        rng = np.random.default_rng(1)
        P, Q = -rng.random(N // 2), -rng.random(N // 2)
        vm = [nd.pqnode_inhomogeneous(P[i], Q[i]) for i in range(N // 2)] + [nd.generator() for _ in range(N - N // 2)]
        return g, [vm[i] for i in rng.permutation(N)], nd.piline()
    kinds = np.random.default_rng(1).permutation(np.repeat([0, 1], N // 2))
    return g, [nd.kuramoto_vertex_1d() if k == 0 else nd.kuramoto_vertex_2d() for k in kinds], \
        nd.static_kuramoto_edge()


def case_inputs(name, net, g):
    """Seeded u, p of a benchmark case: N(0,1) states and U(0.5,1.5) parameters; the power
    grids get line and machine data in the ranges of per-unit grid models."""
    rng = np.random.default_rng(2)
    u = rng.normal(size=net.dim)
    p = rng.uniform(0.5, 1.5, size=net.pdim)
    if name.startswith("powergrid"):
        p = net.pflat(vertex={"P": rng.uniform(-1, 1, g.nv), "Q": rng.uniform(-1, 1, g.nv), "H": 5.0,
                              "D": 0.1, "Ω": 2 * np.pi * 50, "E_f": 1.0, "T_d_dash": 7.0, "T_q_dash": 0.5,
                              "X_d_dash": 0.3, "X_q_dash": 0.6, "X_d": 1.8, "X_q": 1.7},
                      edge={"L": 1e-3, "R": 0.05, "C1": 1e-5, "C2": 1e-5})
        u = 1.0 + 0.1 * rng.normal(size=net.dim)
    return u, p


CASES = (("diffusion_static_edge", 3000), ("diffusion_ode_edge", 3000), ("kuramoto_homogeneous", 100_000),
         ("kuramoto_heterogeneous", 100_000), ("powergrid", 100_000), ("powergrid_inhomogeneous_pq", 100_000))


def run_cases(args):
    """GPU RHS time of every reference benchmark case (FP64 and FP32, CUDA events over
    back-to-back calls on resident buffers, as the reference's @benchmark of nw(du, u, p, NaN)),
    with the CPU oracle (sequential on one core, threaded on all cores) on the same inputs."""
    import torch

    import nd_gb300 as nd
    from nd_gb300 import _capi as capi
    from oracle import oracle as O
    dev = torch.device("cuda:0")
    torch.cuda.set_device(dev)
    hbm = peaks()[0]
    for name, N in CASES:
        g, vm, em = _case_networks(N, name)
        net = nd.Network(g, vm, em)
        u, p = case_inputs(name, net, g)
        line = {"case": name, "N": N, "ne": g.ne, "dim": net.dim, "pdim": net.pdim,
                "vertex_batches": len(net.vertex_batches), "edge_batches": len(net.edge_batches)}
        for tag, dt, s in (("f64", torch.float64, 8), ("f32", torch.float32, 4)):
            nw = nd.adapt(net, dt)
            ut = torch.from_numpy(u).to(dev, dt)
            pt = torch.from_numpy(p).to(dev, dt) if net.pdim else None
            du = torch.empty_like(ut)
            stream = torch.cuda.current_stream()
            for _ in range(max(3, args.warmup)):
                nw(du, ut, pt, 0.0, stream=stream)
            nw.kernel_times()
            steps = max(10, min(args.steps, 500))
            torch.cuda.synchronize()
            el = time_device(nw, du, ut, pt, steps, stream)
            launches = {k: n // steps for k, (n, _) in nw.kernel_times().items() if n}
            # per-kernel device time from a second, event-bracketed pass
            nw.set_kernel_timing(True)
            time_device(nw, du, ut, pt, 50, stream)
            kernel_us = {k: 1e3 * ms / n for k, (n, ms) in nw.kernel_times().items() if n}
            nw.set_kernel_timing(False)
            algo = s * (2 * net.dim + net.pdim) + 4 * (g.nv + 1) + 2 * g.ne * 8
            line[tag] = {"rhs_us": 1e6 * el / steps, "edges_per_s": g.ne * steps / el,
                         "algorithmic_gbs": algo * steps / el / 1e9,
                         "hbm_frac_of_measured": algo * steps / el / 1e9 / hbm,
                         "kernels_per_rhs": launches, "kernel_us": kernel_us,
                         "path": "batched" if "batched_rows" in launches else "homogeneous"}
        vb = [m.kind for m in net.vertex_batches]
        eb = [(m.kind, capi.COUPLINGS[m.coupling]) for m in net.edge_batches]
        consts = [m.constants or (0.0, 0.0) for m in net.vertex_batches]
        on = O.OracleNetwork.from_batches(g.nv, g.src, g.dst, vb, net.vertex_batch, eb, net.edge_batch,
                                          vertex_constants=consts)
        for tag, fn, threads in (("cpu_sequential", on.rhs, 1), ("cpu_threaded", on.rhs_poly, os.cpu_count() or 1)):
            O.load().nd_oracle_set_num_threads(threads)
            fn(u, p)
            n, t0 = 0, time.perf_counter()
            while True:
                fn(u, p)
                n += 1
                sec = time.perf_counter() - t0
                if sec > 3.0 or n >= 200:
                    break
            line[tag] = {"rhs_us": 1e6 * sec / n, "cores": threads, "kind": "port", "evaluations": n}
        O.load().nd_oracle_set_num_threads(os.cpu_count() or 1)
        line["speedup_f64_vs_cpu_threaded"] = line["cpu_threaded"]["rhs_us"] / line["f64"]["rhs_us"]
        print(json.dumps(line), flush=True)


def main():
    args = parse()
    if args.cases:
        run_cases(args)
        return
    rank, world, local = dist_setup(args)
    if args.impl == "reference":
        run_reference(args, rank, world)
    else:
        run_gb300(args, rank, world, local)
    if world > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
