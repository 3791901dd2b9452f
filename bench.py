#!/usr/bin/env python
"""bench.py -- srgemm throughput on B200 through libsimd2.

Default workload: the nine-semiring srgemm sweep at M = N = K = 4096
(min_plus, plus_mul, max_plus, max_min, max_mul, min_mul, min_max, or_and,
minus_square).  One step runs all nine once.  Inputs are seeded synthetic
matrices with the sweep's value distributions (integer-valued FP32 in
[1,1000] with 20% +-inf add-identities for the min/max semirings, U(0,1] for
the *_mul ones, N(0,1) for plus_mul / minus_square, uint8 Bernoulli(0.01)
for or_and).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl simd2|reference]

With N > 1 (torchrun, one rank per GPU) every rank runs the sweep on its
own inputs (independent problems, no collective in the data path): weak
scaling, value = all ranks' operations / max-over-ranks time.

``--impl reference`` times the reference's own CPU srgemm
(escalab/SIMD2 kernel/host_srgemm.h, compiled unchanged into
oracle/_ref/libref.so; the C restatement in oracle/ if that library is
absent) on every host core, on a bounded row sample of the same workload.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

SWEEP_OPS = ("min_plus", "plus_mul", "max_plus", "max_min", "max_mul", "min_mul", "min_max", "or_and",
             "minus_square")
METRIC = "srgemm Gop/s & % CUDA-core/tensor peak; batched APSP graphs/s vs plain path"
SMS = 148
LANES = 128


def parse_args():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=30)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", choices=("simd2", "reference"), default="simd2")
    p.add_argument("--n", type=int, default=4096, help="M = N = K of the sweep")
    p.add_argument("--ref-rows", type=int, default=max(8, os.cpu_count() or 1),
                   help="rows per semiring in the CPU sample (one per host core)")
    p.add_argument("--ops", default=",".join(SWEEP_OPS),
                   help="comma-separated subset of the sweep (profiling runs use one semiring)")
    p.add_argument("--no-extras", action="store_true",
                   help="skip the batched-closure / learned-dispatch / APSP-512 measurements")
    p.add_argument("--batched-count", type=int, default=4096)
    p.add_argument("--batched-n", type=int, default=0,
                   help="with --workload batched: every graph of this size (ER, p = 0.1) instead of the mixed set "
                        "(one size class)")
    p.add_argument("--knn-q", type=int, default=16384)
    p.add_argument("--knn-r", type=int, default=65536)
    p.add_argument("--workload", choices=("sweep", "batched", "knn", "rowpanel", "orand"), default="sweep",
                   help="sweep: the nine-semiring srgemm line (default); batched: only the batched closure "
                        "(used for profiling runs); knn: the k-NN modes; rowpanel: one or_and closure with "
                        "X's rows split across the ranks")
    p.add_argument("--rowpanel-n", type=int, default=16384)
    p.add_argument("--no-e2e", action="store_true")
    p.add_argument("--no-cpu-baseline", action="store_true")
    return p.parse_args()


def measured_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return json.load(f), "measured"
    except OSError:
        return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "sm_max_mhz": 1965.0}, "fallback"


# --------------------------------------------------------------------------
# clocks during the timed region
# --------------------------------------------------------------------------
class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.path = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None
        time.sleep(0.15)
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
        return False

    def summary(self):
        sm, mx, reasons = [], [], set()
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        try:
            with open(self.path) as f:
                for line in f:
                    parts = [x.strip() for x in line.split(",")]
                    if len(parts) < 9:
                        continue
                    try:
                        sm.append(float(parts[1]))
                        mx.append(float(parts[2]))
                    except ValueError:
                        continue
                    for nm, v in zip(names, parts[5:9]):
                        if v.lower() == "active":
                            reasons.add(nm)
            os.unlink(self.path)
        except OSError:
            pass
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "reasons": sorted(reasons),
                "samples": len(sm)}


# --------------------------------------------------------------------------
# CPU baseline: the reference's host_srgemm on a bounded row sample
# --------------------------------------------------------------------------
def cpu_sample_inputs(n, rows, seed=11):
    from simd2_b200 import datagen
    out = {}
    for i, op in enumerate(SWEEP_OPS):
        # rows x n slice of A, full B, rows x n slice of C, same distributions
        a, _, c = datagen.semiring_operands(op, rows, n, n, seed=seed + i)
        _, b, _ = datagen.semiring_operands(op, 1, n, n, seed=seed + 100 + i)
        out[op] = (a, b, c)
    return out


def cpu_sweep(inputs, threads):
    """Runs one sampled sweep on the CPU; returns (ops, seconds, kind)."""
    import oracle
    use_ref = oracle.ref_lib() is not None
    kind = "reference" if use_ref else "port"
    ops = 0.0
    t0 = time.perf_counter()
    for op, (a, b, c) in inputs.items():
        if op == "or_and" and use_ref:
            oracle.srgemm(op, a.astype(np.int32), b.astype(np.int32), c.astype(np.int32), do_epilogue=True,
                          threads=threads, use_ref=True)
        else:
            oracle.srgemm(op, a, b, c, do_epilogue=True, threads=threads, use_ref=use_ref)
        ops += 2.0 * a.shape[0] * b.shape[1] * a.shape[1]
    return ops, time.perf_counter() - t0, kind


def run_reference_arm(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return 0
    threads = os.cpu_count() or 1
    inputs = cpu_sample_inputs(args.n, args.ref_rows)
    for _ in range(max(args.warmup, 0)):
        cpu_sweep(inputs, threads)
    tot_ops, tot_s, kind = 0.0, 0.0, "port"
    for _ in range(args.steps):
        o, s, kind = cpu_sweep(inputs, threads)
        tot_ops += o
        tot_s += s
    gops = tot_ops / tot_s / 1e9
    sample = (f"{args.ref_rows} rows x {args.n} x {args.n} per semiring, all nine semirings per step "
              f"(host_srgemm on row panels, one thread per core)")
    line = {
        "impl": "reference", "metric": METRIC, "value": gops, "unit": "Gop/s", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": tot_s / args.steps * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": f"nine-semiring srgemm sweep M=N=K={args.n} (or_and uint8, int32 for host_srgemm)",
                   "sample": sample},
        "cpu_baseline": {"value": gops, "unit": "Gop/s", "cores": threads, "kind": kind, "sample": sample},
        "e2e": {"value": gops, "unit": "Gop/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
    }
    print(json.dumps(line), flush=True)
    return 0


# --------------------------------------------------------------------------
# GPU arm
# --------------------------------------------------------------------------
# Dispatch slots (lane-cycles) per (x),(+) pair of the CUDA-core kernels on the sweep's
# values: on 16-bit codes an add-min takes one, a selection three instructions of two
# per four pairs; FP32 products (no codes) a packed multiply and a three-operand min,
# two each for two pairs.
SLOTS_PER_PAIR = {"min_plus": 1.0, "max_plus": 1.0, "max_min": 1.5, "min_max": 1.5, "max_mul": 2.0, "min_mul": 2.0}


def issue_peak_gops(op, sm_max):
    """Dispatch bound of one CUDA-core semiring, two operations a pair."""
    return SMS * LANES * sm_max * 1e6 / 1e9 * 2.0 / SLOTS_PER_PAIR[op]


def traffic_from_profile(key="srgemm_sk_kernel min_plus 4096^3"):
    """DRAM bytes per launch of a kernel, from the byte counts kept beside the
    ncu summaries (profiles/dram_traffic.json)."""
    try:
        with open(os.path.join(ROOT, "profiles", "dram_traffic.json")) as f:
            return float(json.load(f)[key]["dram_bytes_per_launch"])
    except (OSError, KeyError, ValueError):
        return None


def batched_sharded(args, dev, rank, world, op="min_plus", reps=3):
    """Batched closure over `world` ranks: every rank builds the same seeded
    graph list, closes its size-balanced shard in one persistent launch
    captured in a CUDA graph, and the slowest rank's device time of a graph
    replay is the job's time (no collective in the data path; only the
    timing is reduced).  The inputs are restored before each replay, outside
    the timed region."""
    import torch

    import simd2_b200 as s2
    from simd2_b200 import datagen
    from simd2_b200.shard import assign_graphs, max_over_ranks

    if getattr(args, "batched_n", 0):
        graphs = [datagen.closure_graph(op, args.batched_n, 0.1, seed=i) for i in range(args.batched_count)]
    else:
        graphs = datagen.batched_graphs(args.batched_count, 32, 1024, seed=3, op=op)
    mine = assign_graphs([g.shape[0] for g in graphs], world)[rank]
    mats = [torch.from_numpy(graphs[g]).to(dev) for g in mine]
    origs = [m.clone() for m in mats]
    plan = s2.BatchedClosure(op, mats)
    plan.run()  # warm-up outside the capture (sets the kernel's shared-memory attribute)
    torch.cuda.synchronize()
    torch._foreach_copy_(mats, origs)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.run()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    times = []
    for _ in range(reps):
        torch._foreach_copy_(mats, origs)
        torch.cuda.synchronize()
        ev0.record()
        graph.replay()
        ev1.record()
        torch.cuda.synchronize()
        times.append(ev0.elapsed_time(ev1))
    its, nc = plan.iters()
    del graph
    plan.close()
    local_ms = min(times)
    ms = max_over_ranks(local_ms, device=dev) if world > 1 else local_ms
    ops = sum(2.0 * graphs[g].shape[0] ** 3 * it for g, it in zip(mine, its))
    if world > 1:
        ops_t = torch.tensor([ops], dtype=torch.float64, device=dev)
        torch.distributed.all_reduce(ops_t)
        ops = float(ops_t.item())
    res = {"semiring": op, "graphs": len(graphs), "n_gpus": world, "batched_ms": ms,
           "graphs_per_s": len(graphs) / ms * 1e3, "gops_dense_equivalent": ops / ms / 1e6, "not_converged": nc,
           "how": "one persistent launch per rank on an n^3-balanced shard, captured in a CUDA graph; CUDA-event time "
                  f"of a graph replay (best of {reps}), max over ranks"}
    return res, graphs, mats, mine


def fp64_errors(got, want, scale=None):
    """Error of a float32 result against its FP64 value: max abs, max rel over
    the entries at least as large as the result's rms (near-zero sums make the
    elementwise ratio meaningless), normwise (max abs / max |FP64|) and, with
    ``scale`` = the sum of the absolute terms, max |err| / scale."""
    import torch
    d = (got.double() - want).abs()
    mag = want.abs()
    rms = float(torch.sqrt((want * want).mean()))
    big = mag >= rms
    out = {"max_abs_err": float(d.max()), "max_rel_err": float((d[big] / mag[big]).max()) if bool(big.any()) else None,
           "normwise_rel_err": float(d.max() / mag.max())}
    if scale is not None:
        out["max_err_over_abs_sum"] = float((d / scale).max())
    return out


def sum_op_errors(op, A, B, C, D):
    """FP64 (torch, on the GPU) errors of a plus_mul / minus_square result
    D = A (x) B (+) C."""
    import torch
    A64, B64, C64 = A.double(), B.double(), C.double()
    if op == "plus_mul":
        want = A64 @ B64 + C64
        scale = A64.abs() @ B64.abs() + C64.abs()
    else:  # sum_k (a_ik - b_kj)^2 = |a_i|^2 + |b_j|^2 - 2 a_i . b_j
        an = (A64 * A64).sum(1, keepdim=True)
        bn = (B64 * B64).sum(0, keepdim=True)
        want = an + bn - 2.0 * (A64 @ B64) + C64
        scale = 2.0 * (an + bn) + C64.abs()
    e = fp64_errors(D, want, scale)
    del A64, B64, C64, want, scale
    return e


def knn_errors(query, ref, dist, idx, sample=2048, k=16):
    """The k-NN result against FP64 on the first ``sample`` queries: distance
    errors (all returned pairs, and the near-duplicate queries whose nearest
    distance is below 0.1), and index agreement position by position as the
    reference's PLD test counts it, plus as sets."""
    import torch
    q = query[:sample].double()
    r = ref.double()
    d2 = (q * q).sum(1, keepdim=True) + (r * r).sum(1)[None, :] - 2.0 * (q @ r.T)
    cand = torch.topk(d2, k + 8, dim=1, largest=False).indices
    del d2
    exact = ((q[:, None, :] - r[cand]) ** 2).sum(2)  # FP64 sum of squares of the candidates
    # order by (distance, index): ties keep the lower reference index
    key_order = torch.argsort(cand, dim=1)
    cand = torch.gather(cand, 1, key_order)
    exact = torch.gather(exact, 1, key_order)
    order = torch.argsort(exact, dim=1, stable=True)[:, :k]
    want_idx = torch.gather(cand, 1, order)
    want_d = torch.sqrt(torch.gather(exact, 1, order))
    got_d = dist[:sample].double()
    got_i = idx[:sample].long()
    rel = (got_d - want_d).abs() / want_d.clamp_min(1e-300)
    near = want_d[:, 0] < 0.1
    pos = (got_i == want_idx).double().mean()
    sets = sum(len(set(a.tolist()) & set(b.tolist())) for a, b in zip(got_i.cpu(), want_idx.cpu())) / (sample * k)
    return {"queries_checked": sample, "max_abs_err": float((got_d - want_d).abs().max()),
            "max_rel_err": float(rel.max()), "near_duplicate_queries": int(near.sum()),
            "near_duplicate_max_rel_err": float(rel[near].max()) if bool(near.any()) else None,
            "index_agreement": float(pos), "index_set_agreement": float(sets),
            "how": "FP64 distances of the first queries to every reference (torch on the GPU), exact FP64 sums of "
                   "squares for the 24 nearest, ordered by (distance, index)"}


def min_plus_8192(dev, reps=3):
    """min_plus srgemm at M = N = K = 8192 with C (integer-valued FP32 in
    [1,1000], 20 % +inf): CUDA-event kernel time from the library's own
    events on the launching stream, and the call's time with its operand
    preparation."""
    import torch

    import simd2_b200 as s2

    n = 8192
    gen = torch.Generator(device=dev)
    gen.manual_seed(8192)

    def ints():
        x = torch.randint(1, 1001, (n, n), device=dev, generator=gen).float()
        x[torch.rand((n, n), device=dev, generator=gen) < 0.2] = float("inf")
        return x

    A, B, C = ints(), ints(), ints()
    D = torch.empty_like(A)
    s2.srgemm("min_plus", A, B, C, do_epilogue=True, D=D)  # warm-up
    torch.cuda.synchronize()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with s2.KernelTimer() as kt:
        ev0.record()
        for _ in range(reps):
            s2.srgemm("min_plus", A, B, C, do_epilogue=True, D=D)
        ev1.record()
        torch.cuda.synchronize()
    kms, launches, _ = kt.by_kind["simt"]
    kms /= max(launches, 1)
    peaks, kind = measured_peaks()
    sm_max = float(peaks.get("sm_max_mhz", 1965.0))
    peak = issue_peak_gops("min_plus", sm_max)
    gops = 2.0 * n ** 3 / kms / 1e6
    del A, B, C, D
    return {"kernel_ms": kms, "call_ms": ev0.elapsed_time(ev1) / reps, "gops": gops, "peak_gops": peak,
            "frac": gops / peak, "peak_source": f"{SMS} SMs x {LANES} pairs x {sm_max:.0f} MHz ({kind} sm_max_mhz)",
            "how": f"srgemm_sk_kernel on 16-bit codes, {reps} launches with C; kernel time from CUDA events on the launching stream"}


def learned_dispatch_mixed(dev, params, weights_path, count=64):
    """min_plus APSP closures of the 64 mixed-density R-MAT graphs (n in
    {4096, 8192, 16384}, average degree 4..4096) under three policies of
    simd2_closure_ex: the plain dense path, the hand-written rules (sparse
    steps under fixed thresholds, then the autotuner's best fixed dense
    configuration) and the learned dispatch (the MLP chooses every step,
    sparse or dense).  Wall clock per call (each call synchronizes); outputs
    are compared bit for bit with the dense path's."""
    import torch

    import simd2_b200 as s2
    from simd2_b200 import datagen

    with open(weights_path) as f:
        rules_cfg = int(json.load(f).get("training", {}).get("best_fixed_config", s2.config_id(2, True)))
    arms = (("dense", {"dispatch": "dense"}), ("rules", {"dispatch": "rules", "config": rules_cfg}),
            ("learned", {"dispatch": "learned", "mlp_params": params}))
    # warm-up per size: workspaces and kernels outside the timing
    for n in (4096, 8192, 16384):
        g = datagen.rmat_graph_device(n, 8.0, seed=1, device=dev)
        for _, kw in arms:
            s2.closure_ex("min_plus", g.clone(), **kw)
        del g
    rows, tot = [], {a: 0.0 for a, _ in arms}
    identical = True
    for n, deg, seed in datagen.rmat_mixed_set(count):
        g = datagen.rmat_graph_device(n, deg, seed=seed, device=dev)
        res, ref, ref_it = {}, None, None
        for name, kw in arms:
            X = g.clone()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            it = s2.closure_ex("min_plus", X, **kw)
            res[name] = (time.perf_counter() - t0) * 1e3
            if ref is None:
                ref, ref_it = X, it
            else:
                identical &= it == ref_it and bool(torch.equal(X.view(torch.int32), ref.view(torch.int32)))
                del X
        # the learned steps' choices, from a recorded (untimed) call
        r = s2.closure_ex("min_plus", g.clone(), record=True, **dict(arms)["learned"])
        cfgs = "".join("s" if c == s2.SPARSE_CONFIG else str(c) for c in r["configs"])
        for a in res:
            tot[a] += res[a]
        rows.append({"n": n, "degree": deg, "iters": ref_it, **{f"{a}_ms": round(v, 3) for a, v in res.items()},
                     "learned_steps": cfgs})
        del g, ref
    return {"graphs": len(rows), "dense_ms": tot["dense"], "rules_ms": tot["rules"], "learned_ms": tot["learned"],
            "speedup_learned_vs_dense": tot["dense"] / tot["learned"],
            "speedup_rules_vs_dense": tot["dense"] / tot["rules"],
            "mlp_gain_learned_vs_rules": tot["rules"] / tot["learned"], "outputs_identical": identical,
            "rules_dense_config": s2.config_desc(rules_cfg),
            "learned_steps_legend": "per step: s = CSR SpGEMM step, else the dense config id (split = 1 << (id & 3), "
                                    "skip = id >> 2)",
            "per_graph": rows,
            "how": "simd2_closure_ex wall clock per graph (synchronous calls, no recording); R-MAT a=.57 b=.19 c=.19 "
                   "drawn on the GPU (datagen.rmat_mixed_set / rmat_graph_device), weights 1..100"}


def or_and_step(dev, n=16384, reps=3):
    """One or_and srgemm D = X (x) X (+) X at N = 16384 on a 0/1 byte matrix of
    density 0.5 (a squaring step after the closure has filled in): kernel time
    from the library's CUDA events, against the nominal dense FP4 rate."""
    import torch

    import simd2_b200 as s2

    gen = torch.Generator(device=dev)
    gen.manual_seed(16384)
    X = (torch.rand((n, n), device=dev, generator=gen) < 0.5).to(torch.uint8)
    D = torch.empty_like(X)
    s2.srgemm("or_and", X, X, X, do_epilogue=True, D=D)
    torch.cuda.synchronize()
    with s2.KernelTimer() as kt:
        for _ in range(reps):
            s2.srgemm("or_and", X, X, X, do_epilogue=True, D=D)
        torch.cuda.synchronize()
    kms, launches, _ = kt.by_kind["tensor"]
    kms /= max(launches, 1)
    tops = 2.0 * n ** 3 / kms / 1e9
    del X, D
    # The peak stated is the nominal dense FP4 rate (four times the nominal dense BF16
    # 2.25 PFLOP/s); no library call here runs 0/1 matrices at that rate to measure it by.
    nominal = 9000.0
    peaks, _ = measured_peaks()
    return {"kernel_ms": kms, "tops": tops, "peak_tops": nominal, "frac": tops / nominal,
            "peak_source": "nominal dense FP4 (9 POPS per B200)",
            "four_times_measured_bf16_tops": 4.0 * float(peaks.get("bf16_tflops", 1590.0)),
            "how": "tc_gemm2_kernel<1> (tcgen05 kind::mxf4 on SM pairs), 0/1 bytes of density 0.5 with C, kernel time "
                   "from CUDA events"}


def extra_measurements(args, dev):
    """The metric's other two parts, on one GPU: batched APSP graphs/s against
    per-graph launches, and the learned dispatch against the plain dense path
    (plus the N=512 ER APSP closure)."""
    import torch

    import simd2_b200 as s2
    from simd2_b200 import costmodel, datagen

    out = {}
    # --- plain APSP, directed ER N=512 p=0.05 (weights 1..100), closure to fixed point
    x = torch.from_numpy(datagen.er_graph(512, 0.05, seed=1)).to(dev)
    res = {}
    weights = os.path.join(ROOT, "simd2_b200", "costmodel_weights.json")
    params = costmodel.load(weights, dev) if os.path.exists(weights) else None
    if params is not None:
        # the plain dense path's split-K by size, as the autotuner measured it
        s2.set_dense_configs(costmodel.load_dense_table(weights))
    for mode in ("dense", "learned") if params is not None else ("dense",):
        X = x.clone()
        r = s2.closure_ex("min_plus", X, dispatch=mode, mlp_params=params, record=True)  # configs, warm-up
        best = None
        for _ in range(5):
            X = x.clone()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            it = s2.closure_ex("min_plus", X, dispatch=mode, mlp_params=params)
            dt = (time.perf_counter() - t0) * 1e3
            best = dt if best is None else min(best, dt)
        res[mode] = {"ms": best, "iters": it, "configs": [s2.config_desc(c) for c in r["configs"]],
                     "gops": 2.0 * 512 ** 3 * it / best / 1e6}
    out["apsp_er512"] = res

    # --- batched closure: graphs with N log-uniform in [32,1024], p in U[0.01,0.3],
    # min_plus APSP and max_min maximum capacity, each against simd2_closure per graph
    out["batched_apsp"] = {}
    for op in ("min_plus", "max_min"):
        res_b, graphs, closed, _ = batched_sharded(args, dev, 0, 1, op=op)
        mats = [torch.from_numpy(g).to(dev) for g in graphs]
        s2.closure(op, mats[0].clone())  # warm-up: the per-graph path's workspace
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        its = [s2.closure(op, m) for m in mats]
        torch.cuda.synchronize()
        pms = (time.perf_counter() - t0) * 1e3
        same = all(torch.equal(a.view(torch.int32), b.view(torch.int32)) for a, b in zip(mats, closed))
        res_b.update({"plain_ms": pms, "plain_graphs_per_s": len(graphs) / pms * 1e3,
                      "speedup_vs_plain": pms / res_b["batched_ms"], "outputs_identical_to_plain": same,
                      "plain_how": "simd2_closure per graph in a host loop (wall clock around synchronize)",
                      "plain_iters_total": int(sum(its))})
        out["batched_apsp"][op] = res_b
        del mats, closed

    # --- paths: closure with a predecessor matrix, and the MST from the min_max closure
    paths = {}
    xp = torch.from_numpy(datagen.er_graph(4096, 0.05, seed=1)).to(dev)

    def best_ms(fn, reps=3):
        fn(xp.clone())  # warm-up
        best = None
        for _ in range(reps):
            X = xp.clone()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            r = fn(X)
            torch.cuda.synchronize()
            dt = (time.perf_counter() - t0) * 1e3
            best = dt if best is None else min(best, dt)
        return best, r

    pred_ms, (pred_it, _) = best_ms(lambda X: s2.closure_pred("min_plus", X))
    plain_ms, plain_it = best_ms(lambda X: s2.closure("min_plus", X))
    paths["closure_pred_er4096"] = {
        "ms": pred_ms, "iters": pred_it, "gops": 2.0 * 4096 ** 3 * pred_it / pred_ms / 1e6,
        "plain_closure_ms": plain_ms, "plain_iters": plain_it, "cost_vs_plain": pred_ms / plain_ms,
        "how": "simd2_closure_pred wall clock (X and P to the fixed point) vs simd2_closure on the same ER graph"}
    mst_ms, mst_r = best_ms(lambda X: s2.mst(X))
    paths["mst_er4096"] = {"ms": mst_ms, "edges": int(len(mst_r[0])), "closure_iters": int(mst_r[3]),
                           "how": "simd2_mst wall clock: min_max closure, candidate scan, host Kruskal over the "
                                  "candidates"}
    out["paths"] = paths
    del xp

    # --- the headline size: min_plus srgemm at 8192^3 on the sweep's value distribution
    out["min_plus_8192"] = min_plus_8192(dev)
    # --- or_and on the FP4 tensor cores: one dense squaring step at N=16384
    out["or_and_16384_step"] = or_and_step(dev)

    # --- dense-contraction workloads at full size (tensor cores)
    cfg4 = {}
    n4 = 16384
    rng = np.random.default_rng(44)
    m4 = 2 * n4
    X = torch.zeros((n4, n4), dtype=torch.uint8, device=dev)
    X[torch.from_numpy(rng.integers(0, n4, m4)).to(dev), torch.from_numpy(rng.integers(0, n4, m4)).to(dev)] = 1
    X.fill_diagonal_(1)
    s2.closure("or_and", X.clone())  # warm-up
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    it4 = s2.closure("or_and", X)
    ms4 = (time.perf_counter() - t0) * 1e3
    cfg4["or_and_closure_16384"] = {"ms": ms4, "iters": it4, "gops_dense_equivalent": 2.0 * n4 ** 3 * it4 / ms4 / 1e6,
                                    "how": "simd2_closure_orand_u8 wall clock: CSR SpGEMM steps while X is sparse, then FP4 "
                                           "tcgen05 per squaring"}
    del X
    q, r = datagen.point_cloud(16384, 65536, 128, seed=4, dup_frac=0.05)
    Q, R = torch.from_numpy(q).to(dev), torch.from_numpy(r).to(dev)
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for mode in ("fused", "materialised"):
        s2.knn(Q, R, 16, mode=mode)  # warm-up at full size (workspace growth stays outside the timing)
        torch.cuda.synchronize()
        with s2.KernelTimer() as kt:
            ev0.record()
            kd, ki = s2.knn(Q, R, 16, mode=mode)
            ev1.record()
            torch.cuda.synchronize()
        kms = ev0.elapsed_time(ev1)
        dist_ms = kt.by_kind.get("tensor", (0, 0, 0))[0]
        cfg4[f"knn_16384x65536x128_k16_{mode}"] = {
            "ms": kms, "queries_per_s": 16384 / kms * 1e3, "gops": 2.0 * 16384 * 65536 * 128 / kms / 1e6,
            "how": "simd2_knn_ex, CUDA events: " + (
                "selection inside the BF16 hi/lo distance MMA's epilogue, then a per-query merge" if mode == "fused"
                else "BF16 hi/lo minus_square blocks of 1 GiB written, then top-k + sqrt")}
        # distance kernels' own time (both passes of the fused mode); BF16 hi/lo = 3 MMAs per product
        peaks, peak_source = measured_peaks()
        bf16_tf = 3 * 2.0 * 16384 * 65536 * 128 / dist_ms / 1e9 if dist_ms > 0 else None
        cfg4[f"knn_16384x65536x128_k16_{mode}"]["distance_kernel"] = {
            "ms": dist_ms, "bf16_tflops": bf16_tf,
            "frac": bf16_tf / float(peaks["bf16_tflops"]) if bf16_tf else None,
            "peak": float(peaks["bf16_tflops"]), "peak_source": f"{peak_source} bf16_tflops (cuBLAS burst)"}
        if mode == "fused":
            cfg4[f"knn_16384x65536x128_k16_{mode}"]["distance_kernel"]["traffic"] = traffic_from_profile(
                "knn_fused_kernel<8> Q=16384 R=65536 D=128 k=16")
            cfg4[f"knn_16384x65536x128_k16_{mode}"]["fp64_error"] = knn_errors(Q, R, kd, ki)
        del kd, ki
    del Q, R
    # --- very sparse inputs: semiring SpGEMM and the hybrid sparse/dense closure
    sp = {}
    xs = datagen.er_graph(16384, 4 / 16384, seed=1)
    Xs = torch.from_numpy(xs).to(dev)
    As = s2.csr_from_dense(Xs, "min_plus")
    s2.spgemm("min_plus", As, As, 16384, C=As)  # warm-up
    ev0.record()
    Ds = s2.spgemm("min_plus", As, As, 16384, C=As)
    ev1.record()
    torch.cuda.synchronize()
    sp["spgemm_step_ms"] = ev0.elapsed_time(ev1)
    sp["nnz_in"], sp["nnz_out"] = int(As[1].numel()), int(Ds[1].numel())
    s2.srgemm("min_plus", Xs, Xs, Xs, do_epilogue=True)
    ev0.record()
    s2.srgemm("min_plus", Xs, Xs, Xs, do_epilogue=True)
    ev1.record()
    torch.cuda.synchronize()
    sp["dense_step_ms"] = ev0.elapsed_time(ev1)
    s2.closure_sparse("min_plus", As)  # warm-up: workspaces and capacity buffers allocated outside the timing
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    _, sp["hybrid_closure_iters"] = s2.closure_sparse("min_plus", As)
    torch.cuda.synchronize()
    sp["hybrid_closure_ms"] = (time.perf_counter() - t0) * 1e3
    t0 = time.perf_counter()
    sp["dense_closure_iters"] = s2.closure("min_plus", Xs)
    torch.cuda.synchronize()
    sp["dense_closure_ms"] = (time.perf_counter() - t0) * 1e3
    sp["how"] = ("ER n=16384, average degree 4, min_plus: one X (+) X(x)X step as CSR SpGEMM vs the dense srgemm "
                 "(CUDA events); closure as sparse steps until density 1/32 then the dense gated closure, vs the dense "
                 "closure throughout (wall clock)")
    del Xs, As, Ds
    cfg4["sparse_er16384_deg4"] = sp
    gen = torch.Generator(device=dev)
    gen.manual_seed(8192)
    A = torch.randn((8192, 8192), device=dev, generator=gen)
    B = torch.randn((8192, 8192), device=dev, generator=gen)
    Dp = s2.srgemm("plus_mul", A, B)
    torch.cuda.synchronize()
    with s2.KernelTimer() as kt8:
        ev0.record()
        for _ in range(3):
            s2.srgemm("plus_mul", A, B, D=Dp)
        ev1.record()
        torch.cuda.synchronize()
    pms = ev0.elapsed_time(ev1) / 3
    # the call includes the BF16 hi/lo split of A and B; the kernel's own time beside it
    kms8 = kt8.by_kind.get("tensor", (0, 0, 0))[0] / 3
    peaks, peak_source = measured_peaks()
    cfg4["plus_mul_8192"] = {"ms": pms, "gops": 2.0 * 8192 ** 3 / pms / 1e6,
                             "bf16_equiv_tflops": 3 * 2.0 * 8192 ** 3 / pms / 1e9,
                             "kernel_ms": kms8,
                             "kernel_bf16_equiv_tflops": 3 * 2.0 * 8192 ** 3 / kms8 / 1e9 if kms8 > 0 else None,
                             "kernel_frac": (3 * 2.0 * 8192 ** 3 / kms8 / 1e9) / float(peaks["bf16_tflops"])
                             if kms8 > 0 else None,
                             "peak_source": f"{peak_source} bf16_tflops (cuBLAS burst)",
                             "fp64_error": sum_op_errors("plus_mul", A, B, torch.zeros_like(A), Dp)}
    del A, B, Dp
    out["dense_contraction"] = cfg4

    # --- learned dispatch on mixed-density R-MAT (a=.57 b=.19 c=.19): plain dense path,
    # the hand-written rules, and the MLP's choices
    if params is not None:
        out["learned_dispatch"] = learned_dispatch_mixed(dev, params, weights)
    return out


def main():
    global SWEEP_OPS
    args = parse_args()
    SWEEP_OPS = tuple(op for op in args.ops.split(",") if op)
    if args.impl == "reference":
        return run_reference_arm(args)

    import torch
    import torch.distributed as dist

    import simd2_b200 as s2
    from simd2_b200 import datagen

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        import datetime
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120), device_id=dev)

    def barrier():
        if world > 1:
            dist.barrier()

    if args.workload == "knn":
        from simd2_b200 import datagen
        q, r = datagen.point_cloud(args.knn_q, args.knn_r, 128, seed=4, dup_frac=0.05)
        Q, R = torch.from_numpy(q).to(dev), torch.from_numpy(r).to(dev)
        out = {"workload": f"knn Q={args.knn_q} R={args.knn_r} D=128 k=16"}
        for mode in ("fused", "materialised"):
            for _ in range(max(args.warmup, 1)):
                s2.knn(Q, R, 16, mode=mode)
            ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            with s2.KernelTimer() as kt:
                ev0.record()
                for _ in range(args.steps):
                    s2.knn(Q, R, 16, mode=mode)
                ev1.record()
                torch.cuda.synchronize()
            ms = ev0.elapsed_time(ev1) / args.steps
            out[mode] = {"ms": ms, "queries_per_s": args.knn_q / ms * 1e3,
                         "distance_kernel_ms": kt.by_kind.get("tensor", (0, 0, 0))[0] / args.steps}
        if rank == 0:
            print(json.dumps(out), flush=True)
        return 0

    if args.workload == "orand":
        # one or_and reachability closure per rank (independent replicas), the
        # configuration-4 graph: CSR steps while X is sparse, then FP4 delta steps
        n = args.rowpanel_n
        rng = np.random.default_rng(44)
        m = 2 * n
        base = torch.zeros((n, n), dtype=torch.uint8, device=dev)
        base[torch.from_numpy(rng.integers(0, n, m)).to(dev), torch.from_numpy(rng.integers(0, n, m)).to(dev)] = 1
        base.fill_diagonal_(1)
        X = base.clone()
        s2.closure("or_and", X)  # warm-up
        times, its = [], 0
        for _ in range(max(args.steps, 1)):
            X.copy_(base)
            barrier()
            torch.cuda.synchronize()
            ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            ev0.record()
            its = s2.closure("or_and", X)
            ev1.record()
            torch.cuda.synchronize()
            times.append(ev0.elapsed_time(ev1))
        ms = sorted(times)[len(times) // 2]
        if world > 1:
            from simd2_b200.shard import max_over_ranks
            ms = max_over_ranks(ms, device=dev)
        if rank == 0:
            print(json.dumps({"workload": f"or_and closure n={n} (edge probability 2/n, seed 44)", "ms": ms,
                              "iters": its, "gops_dense_equivalent": 2.0 * n ** 3 * its / ms / 1e6, "n_gpus": world,
                              "how": "simd2_closure_orand_u8 on every rank; CUDA events, median of steps, max over "
                                     "ranks"}), flush=True)
        if world > 1:
            dist.destroy_process_group()
        return 0

    if args.workload == "rowpanel":
        from simd2_b200.shard import closure_rowpanel, max_over_ranks, panel_bounds
        n = args.rowpanel_n
        rng = np.random.default_rng(44)
        m = 2 * n  # or_and reachability closure, edge probability 2/n
        x = np.zeros((n, n), np.uint8)
        x[rng.integers(0, n, m), rng.integers(0, n, m)] = 1
        np.fill_diagonal(x, 1)
        P, bounds = panel_bounds(n, world)
        start, stop = bounds[rank]
        base = torch.zeros((P, n), dtype=torch.uint8, device=dev)
        base[: stop - start] = torch.from_numpy(x[start:stop]).to(dev)
        del x
        block = base.clone()
        closure_rowpanel("or_and", block, n)  # warm-up (same collective sequence on every rank)
        times, its = [], 0
        for _ in range(max(args.steps, 1)):
            block.copy_(base)
            barrier()
            torch.cuda.synchronize()
            ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            ev0.record()
            its = closure_rowpanel("or_and", block, n)
            ev1.record()
            torch.cuda.synchronize()
            barrier()
            times.append(ev0.elapsed_time(ev1))
        ms = sorted(times)[len(times) // 2]
        if world > 1:
            ms = max_over_ranks(ms, device=dev)
        if rank == 0:
            print(json.dumps({"workload": f"or_and closure n={n}, rows split over {world} rank(s)", "ms": ms,
                              "iters": its, "gops": 2.0 * n ** 3 * its / ms / 1e6, "n_gpus": world,
                              "how": "closure_rowpanel: all-gather of the row blocks, simd2_closure_panel_step, "
                                     "all-reduce(MAX) of the change flag per squaring; CUDA events, median "
                                     "of steps, max over ranks"}), flush=True)
        if world > 1:
            dist.destroy_process_group()
        return 0

    if args.workload == "batched":
        res = {op: batched_sharded(args, dev, rank, world, op=op)[0] for op in ("min_plus", "max_min")}
        if rank == 0:
            what = (f"batched closure, {args.batched_count} ER graphs of n={args.batched_n}, p=0.1" if args.batched_n
                    else "batched closure")
            print(json.dumps({"workload": what, **res}), flush=True)
        if world > 1:
            dist.destroy_process_group()
        return 0

    n = args.n
    s2.lib()
    # inputs: resident in HBM for `value`, pinned on the host for `e2e`
    host, devb = {}, {}
    for i, op in enumerate(SWEEP_OPS):
        a, b, c = datagen.semiring_operands(op, n, n, n, seed=1000 * rank + i)
        host[op] = tuple(torch.from_numpy(x).pin_memory() for x in (a, b, c))
        devb[op] = tuple(x.to(dev, non_blocking=True) for x in host[op])
    outs = {op: torch.empty((n, n), dtype=devb[op][2].dtype, device=dev) for op in SWEEP_OPS}
    torch.cuda.synchronize()

    def step():
        for op in SWEEP_OPS:
            A, B, C = devb[op]
            s2.srgemm(op, A, B, C, do_epilogue=True, D=outs[op])

    for _ in range(max(args.warmup, 3)):
        step()
    torch.cuda.synchronize()
    barrier()

    stream = torch.cuda.current_stream()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    launches0 = s2.launch_count()
    with ClockSampler(local) as clk:
        torch.cuda.synchronize()
        barrier()
        with s2.KernelTimer() as kt:
            ev0.record(stream)
            for _ in range(args.steps):
                step()
            ev1.record(stream)
            torch.cuda.synchronize()
        barrier()
    launches = s2.launch_count() - launches0
    ms = ev0.elapsed_time(ev1)
    ms_t = torch.tensor([ms], device=dev)
    if world > 1:
        dist.all_reduce(ms_t, op=dist.ReduceOp.MAX)
    ms_max = float(ms_t.item())
    ops_per_step = 2.0 * n ** 3 * len(SWEEP_OPS)
    value = ops_per_step * args.steps * world / (ms_max / 1e3) / 1e9
    assert s2.device_status() == 0, "a kernel reported a device-side error"

    # per-semiring kernel throughput (one timed launch each, after the sweep)
    per_op = {}
    for op in SWEEP_OPS:
        A, B, C = devb[op]
        with s2.KernelTimer() as t1:
            for _ in range(3):
                s2.srgemm(op, A, B, C, do_epilogue=True, D=outs[op])
        per_op[op] = t1.ops / (t1.kernel_ms / 1e3) / 1e9
    # FP64 error of the two summing semirings' sweep results (the last launch's D)
    sweep_err = {}
    for op in ("plus_mul", "minus_square"):
        if op in SWEEP_OPS:
            A, B, C = devb[op]
            sweep_err[op] = sum_op_errors(op, A, B, C, outs[op])
            torch.cuda.synchronize()

    # e2e through the public API with host buffers: H2D inputs, srgemm, D2H result,
    # pipelined over two buffer sets and three streams.
    e2e = None
    if not args.no_e2e:
        s_in, s_cmp, s_out = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Stream()
        slots = [{op: (torch.empty_like(devb[op][0]), torch.empty_like(devb[op][1]), torch.empty_like(devb[op][2]),
                       torch.empty_like(outs[op])) for op in SWEEP_OPS} for _ in range(2)]
        host_out = {op: torch.empty((n, n), dtype=outs[op].dtype).pin_memory() for op in SWEEP_OPS}
        bi = sum(sum(x.numel() * x.element_size() for x in host[op]) for op in SWEEP_OPS)
        bo = sum(host_out[op].numel() * host_out[op].element_size() for op in SWEEP_OPS)

        def e2e_step(free_ev):
            # Every semiring has its own device buffers; the only reuse is the
            # same semiring's buffers one step later, so H2D of op j waits for
            # nothing but the D2H of op j in the previous step.
            for j, op in enumerate(SWEEP_OPS):
                slot = slots[j % 2][op]
                with torch.cuda.stream(s_in):
                    if free_ev.get(op) is not None:
                        s_in.wait_event(free_ev[op])
                    for hx, dx in zip(host[op], slot[:3]):
                        dx.copy_(hx, non_blocking=True)
                    in_ev = torch.cuda.Event()
                    in_ev.record(s_in)
                with torch.cuda.stream(s_cmp):
                    s_cmp.wait_event(in_ev)
                    s2.srgemm(op, slot[0], slot[1], slot[2], do_epilogue=True, D=slot[3], stream=s_cmp)
                    c_ev = torch.cuda.Event()
                    c_ev.record(s_cmp)
                with torch.cuda.stream(s_out):
                    s_out.wait_event(c_ev)
                    host_out[op].copy_(slot[3], non_blocking=True)
                    f_ev = torch.cuda.Event()
                    f_ev.record(s_out)
                free_ev[op] = f_ev

        free = {}
        for _ in range(2):
            e2e_step(free)
        torch.cuda.synchronize()
        barrier()
        t0 = time.perf_counter()
        for _ in range(max(1, args.steps // 3)):
            e2e_step(free)
        torch.cuda.synchronize()
        e2e_s = time.perf_counter() - t0
        e2e_steps = max(1, args.steps // 3)
        et = torch.tensor([e2e_s], device=dev)
        if world > 1:
            dist.all_reduce(et, op=dist.ReduceOp.MAX)
        e2e = {"value": ops_per_step * e2e_steps * world / float(et.item()) / 1e9, "unit": "Gop/s",
               "h2d_bytes_per_step": bi, "d2h_bytes_per_step": bo,
               "how": "pinned host buffers; per semiring H2D(A,B,C) -> srgemm -> D2H(D) on three streams "
                      "(copy in, compute, copy out), device buffers per semiring; wall clock around synchronize"}

    clocks = clk.summary()
    peaks, peak_kind = measured_peaks()
    sm_max = float(peaks.get("sm_max_mhz", 1965.0))
    # the six semirings do the same number of pairs: the harmonic mean of their bounds
    simt_run = [op for op in SLOTS_PER_PAIR if op in args.ops.split(",")] or list(SLOTS_PER_PAIR)
    simt_peak = len(simt_run) / sum(1.0 / issue_peak_gops(op, sm_max) for op in simt_run)
    simt_ms, simt_n, simt_ops = kt.by_kind["simt"]
    tc_ms, tc_n, tc_ops = kt.by_kind["tensor"]
    achieved = simt_ops / (simt_ms / 1e3) / 1e9 if simt_ms > 0 else None
    traffic = traffic_from_profile()
    # tensor-core family: plus_mul / minus_square issue 3 BF16 MMAs per product term
    # (hi*hi, hi*lo, lo*hi), or_and one FP4 MMA at four times the BF16 rate; both are
    # expressed as BF16-equivalent FLOP/s against the measured cuBLAS BF16 peak.
    tc_equiv = 0.0
    for op in SWEEP_OPS:
        if op in ("plus_mul", "minus_square"):
            tc_equiv += 3 * 2.0 * n ** 3 * args.steps
        elif op == "or_and":
            tc_equiv += 0.25 * 2.0 * n ** 3 * args.steps
    bf16_peak = float(peaks.get("bf16_tflops", 1590.0))

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        threads = os.cpu_count() or 1
        inputs = cpu_sample_inputs(n, args.ref_rows)
        o, s_, kind = cpu_sweep(inputs, threads)
        cpu = {"value": o / s_ / 1e9, "unit": "Gop/s", "cores": threads, "kind": kind,
               "sample": f"{args.ref_rows} rows x {n} x {n} per semiring, all nine semirings, one sweep"}

    extras = {}
    if not args.no_extras:
        if world == 1:
            extras = extra_measurements(args, dev)
        else:
            extras = {"batched_apsp": {op: batched_sharded(args, dev, rank, world, op=op)[0]
                                       for op in ("min_plus", "max_min")}}
    if world > 1:
        lt = torch.tensor([launches], dtype=torch.float64, device=dev)
        dist.all_reduce(lt)
        launches = int(lt.item())

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": "Gop/s", "n_gpus": world, "steps": args.steps,
            "warmup": max(args.warmup, 3), "ms_per_step": ms_max / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": f"nine-semiring srgemm sweep M=N=K={n} (or_and uint8 0/1 density 0.01)",
                       "l2": "inputs larger than L2: 9 semirings x (A,B,C) x 64 MiB rotated every step",
                       "parallelism": f"independent sweep per rank x{world}"},
            "per_semiring_kernel_gops": per_op,
            "fp64_error": dict(sweep_err, how="full 4096 x 4096 results against FP64 (torch on the GPU): max abs, max "
                                              "rel over entries >= the rms, normwise, and max |err| / sum of |terms|; "
                                              "min/max semirings and or_and are bit-exact (tests)"),
            "roofline": {"bound": "cuda_core_issue",
                         "kernel": "srgemm_sk_kernel (min_plus, max_plus, max_min, max_mul, min_mul, min_max)",
                         "achieved": achieved, "peak": simt_peak, "unit": "Gop/s",
                         "frac": achieved / simt_peak if achieved else None, "traffic": traffic,
                         "peak_source": f"{SMS} SMs x {LANES} lanes x {sm_max:.0f} MHz ({peak_kind} sm_max_mhz); "
                                        "2 ops per (x),(+) pair; dispatch slots per pair: " + json.dumps(SLOTS_PER_PAIR),
                         "share_of_kernel_time": simt_ms / (simt_ms + tc_ms) if simt_ms + tc_ms > 0 else None,
                         "timed_launches": simt_n},
            "roofline_tensor": {"bound": "tensor", "kernel": "tc_gemm2_kernel on SM pairs (plus_mul, minus_square, or_and)",
                                "achieved": tc_equiv / (tc_ms / 1e3) / 1e12 if tc_ms > 0 else None,
                                "peak": bf16_peak, "unit": "TFLOP/s (BF16-equivalent)",
                                "frac": (tc_equiv / (tc_ms / 1e3) / 1e12) / bf16_peak if tc_ms > 0 else None,
                                "peak_source": f"{peak_kind} bf16_tflops (cuBLAS burst)", "timed_launches": tc_n,
                                "traffic": traffic_from_profile("tc_gemm2_kernel plus_mul 4096^3"),
                                "traffic_of": "one plus_mul 4096^3 launch with C (ncu dram read + write)"},
            "cpu_baseline": cpu,
            "e2e": e2e,
            "gpu_launches": launches,
            "clocks": clocks,
        }
        mp = line["per_semiring_kernel_gops"].get("min_plus") if line.get("per_semiring_kernel_gops") else None
        if mp:
            # the reference's one recorded measurement of this path: the cuASR
            # min_plus srgemm kernel at 4096^3, 27.32 ms on an RTX 3080-class
            # Ampere board (2 * 4096^3 / 27.32 ms = 5031 Gop/s); another GPU, so
            # this is context, not vs_baseline
            line["published_comparison"] = {
                "kernel": "min_plus srgemm 4096^3, kernel time", "published_gops": 2.0 * 4096 ** 3 / 27.32e-3 / 1e9,
                "published_hw": "Ampere, RTX 3080 class, SM 1.44 GHz", "this_gops": mp,
                "ratio": mp / (2.0 * 4096 ** 3 / 27.32e-3 / 1e9)}
        line.update(extras)
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
