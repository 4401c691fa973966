#!/usr/bin/env python
"""Benchmark of the PDHG LP hot path on B200.

Workload: the large seeded LP (m=1,000,000, n=2,000,000, ~21.1M nonzeros,
Zipf(1.5) column degrees clamped at 2000 and thinned, values +-10^U[-3,3];
vikalp_b200.synthetic.workload_large_lp). Synthetic data: no dataset exists
for this path.

A step is one check interval of 64 PDHG iterations over that LP. `value` is
PDHG iterations per second of the reference scheme (pdhg.cpp:87-151, the
same algorithm the reference arm runs on the CPU) on resident device data,
timed with CUDA events on the solver's stream between a barrier + synchronize
on both sides; whole-job = the sum over ranks (each rank solves its own copy:
replicas, no collective on the path). The same line carries:
  e2e            the same metric through the C ABI from host arrays (model
                 upload, device setup, iterations, results copied back)
  halpern        iterations/s of the restarted Halpern scheme, fp64 and mixed
  time_to_tol    time and iterations to 1e-6 relative KKT, fp64 vs mixed, on
                 the small LP and on the bench's large LP (its points
                 re-evaluated by the C oracle; --no-ttt skips the large LP)
  spmv           GB/s of the sparse product kernel, A x and A'y, fp64 / fp32
  batched        768 LPs (512 shared-matrix node relaxations + 256 independent
                 LPs) to 1e-6 relative KKT in two batches, mixed and fp64, vs
                 the plain fp64 engine one instance at a time (sampled)
  adjoint        256 LPs solved and differentiated (gradients w.r.t. b and A)
                 in batches, errors against the CPU FP64 KKT gradient
  time_to_tol.qp the convex QP (n=5e5, m=2e5), fp64 vs mixed
  roofline       the sparse-pass kernel against measured HBM bandwidth
  reference_cuda the reference's own CUDA backend (cuSPARSE) on the same GPU
  cpu_baseline   the reference's CPU implementation on this host
`python bench.py --impl reference` times the reference's own CPU PDHG
iteration (oracle/_ref, compiled from the reference sources) on the same LP.
"""

from __future__ import annotations

import argparse
import json
import os
import re
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

CHUNK = 64  # iterations per step (one device-side check interval)
METRIC = "PDHG LP iterations/s (reference scheme; m=1e6 n=2e6 nnz=21.1M); time to 1e-6 rel KKT and SpMV GB/s in-line"


def measured_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


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
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except (OSError, ValueError):
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.samples.append([s.strip() for s in line.split(",")])

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(s[1]) for s in self.samples if len(s) > 8 and s[1].replace(".", "").isdigit()]
        mx = [float(s[2]) for s in self.samples if len(s) > 8 and s[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for s in self.samples if len(s) > 8 for i in range(4)
                          if s[5 + i].lower().startswith("active")})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.samples)}


def profile_traffic(kernel_name):
    """DRAM bytes per launch of a fused pass (the column or the row pass of the
    reference-scheme iteration on the large LP) from its committed ncu summary,
    with the kernel variant that capture pinned: (bytes, variant, file)."""
    name = "col_pass_large_lp.md" if kernel_name.startswith("column") else "row_pass_large_lp.md"
    p = os.path.join(ROOT, "profiles", name)
    if not os.path.exists(p):
        return None, None, name
    text = open(p).read()
    m = re.search(r"traffic_bytes_per_launch:\s*([0-9.eE+]+)", text)
    v = re.search(r"Kernel: variant (\d+)", text)
    return (float(m.group(1)) if m else None), (int(v.group(1)) if v else None), name


def spmv_figures(inst, torch, stream):
    """GB/s of the sparse product kernel (A x and A'y, fp64 and fp32), live CUDA events."""
    import vikalp_b200 as vk
    out = {}
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device="cuda")
    for prec, dt in (("fp64", torch.float64), ("fp32", torch.float32)):
        A = vk.SpMat(inst.row_offsets, inst.col_idx, inst.values, inst.m, inst.n,
                     "fp64" if prec == "fp64" else "mixed")
        for tr in (False, True):
            xl, yl = (inst.m, inst.n) if tr else (inst.n, inst.m)
            x = torch.rand(xl, dtype=dt, device="cuda")
            y = torch.zeros(yl, dtype=dt, device="cuda")
            for _ in range(3):
                A.apply(x.data_ptr(), y.data_ptr(), tr, stream.cuda_stream)
            ts = []
            for _ in range(10):
                flush.zero_()
                e0 = torch.cuda.Event(enable_timing=True)
                e1 = torch.cuda.Event(enable_timing=True)
                e0.record(stream)
                A.apply(x.data_ptr(), y.data_ptr(), tr, stream.cuda_stream)
                e1.record(stream)
                torch.cuda.synchronize()
                ts.append(e0.elapsed_time(e1))
            ms = statistics.median(ts)
            out[f"{prec}_{'At_y' if tr else 'A_x'}"] = {
                "ms": round(ms, 4), "bytes": A.bytes(tr), "gbs": round(A.bytes(tr) / ms / 1e6, 1),
                "variant": A.variant(tr)}
        A.close()
    return out


def time_to_tolerance(inst, label, limit, time_limit=float("inf"), check=False):
    """Both precisions of the Halpern scheme to 1e-6 relative KKT. With check,
    the returned point's relative KKT is evaluated again by the C oracle (the
    checker, not the thing timed) and the mixed answer's error against the
    float64 answer is reported."""
    import vikalp_b200 as vk
    res, pts = {}, {}
    for prec in ("fp64", "mixed"):
        with vk.Pdhg(inst, algorithm="halpern", precision=prec, iteration_limit=limit,
                     relative_tolerance=1e-6, time_limit_seconds=time_limit) as h:
            r = h.solve(duals=False)
        pts[prec] = r
        res[prec] = {"status": r["status"], "iterations": r["iterations"], "fp32_iterations": r["fp32_iterations"],
                     "iterate_s": round(r["iterate_seconds"], 4), "solve_s": round(r["solve_seconds"], 4),
                     "rel_kkt": max(r["rel_primal"], r["rel_dual"], r["rel_gap"]), "objective": r["objective"]}
        if check:
            from oracle.oracle import Oracle
            k = Oracle().rel_kkt(inst, r["x"], r["y"])
            res[prec]["rel_kkt_by_c_oracle"] = max(k["rel_primal"], k["rel_dual"], k["rel_gap"])
    f64, mx = pts["fp64"], pts["mixed"]
    res["mixed_vs_fp64"] = {
        "objective_rel_diff": abs(mx["objective"] - f64["objective"]) / (1 + abs(f64["objective"])),
        "x_rel_diff": float(np.linalg.norm(mx["x"] - f64["x"]) / max(np.linalg.norm(f64["x"]), 1e-300))}
    f, mx = res["fp64"], res["mixed"]
    if f["status"] == "Optimal" and mx["status"] == "Optimal":
        res["mixed_speedup_vs_fp64"] = round(f["iterate_s"] / mx["iterate_s"], 3)
    res["workload"] = label
    return res


def batched_figures():
    """The batched workload: 512 node relaxations of one LP (m=50,000, n=100,000,
    6 nonzeros per column, 1-12 tightened variables each) and 256 independent
    LPs (m log-uniform on [500, 20000], n=2m, 8 per column), all to 1e-6
    relative KKT. Batched: one vk_batch_solve_together call (both batches set up,
    then both device loops in flight on their own streams); wall time from host
    arrays to results. Also timed: the two batches one after the other, and the
    plain-FP64 comparison, which solves every one of the 768 instances one by
    one with the single-instance float64 engine (a resident model for the
    nodes, create + solve for each independent LP)."""
    import vikalp_b200 as vk
    from vikalp_b200 import synthetic
    node_lp = synthetic.lp_uniform(50000, 100000, 6, seed=2025)
    lo, hi = synthetic.bnb_nodes(node_lp, 512, seed=7)
    indep = synthetic.workload_independent_lps(256)
    tol = dict(iteration_limit=200000, relative_tolerance=1e-6, time_limit_seconds=300)

    def summary(rs, wall):
        status = {}
        for r in rs:
            status[r["status"]] = status.get(r["status"], 0) + 1
        return {"wall_s": round(wall, 3), "status": status, "max_iterations": int(max(r["iterations"] for r in rs)),
                "max_rel_kkt": float(max(max(r["rel_primal"], r["rel_dual"], r["rel_gap"]) for r in rs))}

    answers = {}

    def together(prec):
        t0 = time.perf_counter()
        nodes, lps = vk.batch_solve_together(node_lp, 512, indep, lo, hi, precision=prec, **tol)
        out = summary(nodes + lps, time.perf_counter() - t0)
        out["shared_iterate_s"] = round(nodes[0]["iterate_seconds"], 3)
        out["independent_iterate_s"] = round(lps[0]["iterate_seconds"], 3)
        answers[prec] = nodes + lps
        return out

    def one_after_other(prec):
        t0 = time.perf_counter()
        nodes = vk.batch_solve_shared(node_lp, 512, lo, hi, precision=prec, **tol)
        t1 = time.perf_counter()
        lps = vk.batch_solve(indep, precision=prec, **tol)
        out = summary(nodes + lps, time.perf_counter() - t0)
        out.update(shared_s=round(t1 - t0, 3), independent_s=round(time.perf_counter() - t1, 3))
        return out

    out = {"workload": "512 node LPs sharing A (m=5e4 n=1e5 nnz=600k, 1-12 tightened bounds) + 256 independent LPs "
                       "(m log-uniform 500..20000, n=2m, 8/col; 19.7M nnz), to 1e-6 relative KKT",
           "mixed": together("mixed"), "fp64_batched": together("fp64"),
           "mixed_one_batch_after_the_other": one_after_other("mixed")}
    # the mixed answers against the float64 ones, instance by instance
    obj = [abs(a["objective"] - b["objective"]) / (1 + abs(b["objective"]))
           for a, b in zip(answers["mixed"], answers["fp64"])]
    out["mixed_vs_fp64"] = {"max_objective_rel_diff": float(max(obj)), "median_objective_rel_diff":
                            float(statistics.median(obj))}
    # plain float64, every instance one by one
    # (one untimed solve of each kind first, so no one-time cost of the path enters)
    node_t, indep_t, statuses = [], [], {}
    with vk.Pdhg(node_lp, algorithm="halpern", precision="fp64", **tol) as h:
        h.solve(lower=lo[0], upper=hi[0], duals=False)
        t_all = time.perf_counter()
        for b in range(512):
            t = time.perf_counter()
            r = h.solve(lower=lo[b], upper=hi[b], duals=False)
            node_t.append(time.perf_counter() - t)
            statuses[r["status"]] = statuses.get(r["status"], 0) + 1
    vk.solve(indep[0], algorithm="halpern", precision="fp64", **tol)
    for inst in indep:
        t = time.perf_counter()
        r = vk.solve(inst, algorithm="halpern", precision="fp64", **tol)
        indep_t.append(time.perf_counter() - t)
        statuses[r["status"]] = statuses.get(r["status"], 0) + 1
    measured = sum(node_t) + sum(indep_t)
    out["plain_fp64_one_by_one"] = {"measured_s": round(measured, 3), "nodes_s": round(sum(node_t), 3),
                                    "independent_s": round(sum(indep_t), 3), "status": statuses,
                                    "instances": len(node_t) + len(indep_t),
                                    "slowest_node_s": round(max(node_t), 4),
                                    "slowest_independent_s": round(max(indep_t), 4)}
    out["speedup_mixed_batched_vs_plain_fp64"] = round(measured / out["mixed"]["wall_s"], 2)
    return out


def adjoint_figures(count=256, checked=3):
    """The differentiable-LP workload: `count` LPs (m=1000, n=2000, 8 nonzeros
    per column, distinct seeds), solved in one batch (mixed precision, float64
    polish to 1e-9 relative KKT), then gradients of L = g'x* (g ~ N(0,1)) with
    respect to b and the values of A in one adjoint batch. Errors: relative
    2-norm against the CPU FP64 active-set gradient at HiGHS's optimum on the
    first `checked` instances."""
    import vikalp_b200 as vk
    from oracle import adjoint as oadj
    from vikalp_b200 import synthetic
    lps = [synthetic.lp_uniform(1000, 2000, 8, seed=7000 + s) for s in range(count)]
    rng = np.random.default_rng(99)
    gs = [rng.standard_normal(i.n) for i in lps]
    t0 = time.perf_counter()
    sols = vk.batch_solve(lps, precision="mixed", iteration_limit=500000, relative_tolerance=1e-9,
                          time_limit_seconds=300)
    t_solve = time.perf_counter() - t0
    t0 = time.perf_counter()
    grads = vk.lp_adjoint(lps, [s["x"] for s in sols], [s["y"] for s in sols], gs)
    t_adj = time.perf_counter() - t0
    errs = {"b": [], "A": []}
    for k in range(checked):
        x, y = oadj.highs_solve(lps[k])
        want = oadj.kkt_gradient(lps[k], x, y, gs[k])
        for key in errs:
            errs[key].append(float(np.linalg.norm(grads[k][key] - want[key]) / np.linalg.norm(want[key])))
    status = {}
    for s in sols:
        status[s["status"]] = status.get(s["status"], 0) + 1
    return {"workload": f"{count} LPs m=1000 n=2000 nnz=16k (distinct seeds), L = g'x*, g ~ N(0,1)",
            "solve_s": round(t_solve, 3), "solve_status": status, "adjoint_s": round(t_adj, 3),
            "adjoint_max_lsqr_iterations": int(max(g["iterations"] for g in grads)),
            "adjoint_status": sorted({g["status"] for g in grads}),
            "max_rel_err_vs_cpu_fp64_kkt": {k: max(v) for k, v in errs.items()},
            "checked_instances": checked}


def reference_cuda_rate(inst, iterations=64):
    """Iterations/s of the same pdhg.cpp:92-130 call sequence on the reference's
    own CUDA backend (cuda/cuda_ops.cu, cuSPARSE CSR SpMV with int64 indices,
    built for sm_100a into oracle/_ref/libvkref_cuda.so) on this GPU: the
    GPU-to-GPU comparison. None when that build is absent."""
    from oracle.oracle import Oracle, ReferenceCuda
    try:
        ref = ReferenceCuda()
    except (FileNotFoundError, OSError):
        return None
    step = 0.99 / max(1.0, Oracle().operator_bound(inst.row_offsets, inst.col_idx, inst.values, inst.n))
    ref.pdhg_replay_cuda(inst, step, 2)  # warm-up (cuSPARSE handle, workspaces)
    secs, _, _ = ref.pdhg_replay_cuda(inst, step, iterations)
    return {"value": round(iterations / secs, 2), "unit": "iter/s", "iterations": iterations,
            "note": "the reference's own CUDA backend (cuSPARSE CSR ALG1, int64 indices, host-finished "
                    "norm_inf twice per iteration) replaying the pdhg.cpp:92-130 call sequence on the same "
                    "LP and GPU; comparison only"}


def reference_cpu_rate(inst, budget_s, warmup=3):
    """Iterations/s of the reference's own CPU PDHG iteration (pdhg.cpp:92-130 call
    sequence through its CPU ExecutionBackend), a bounded sample sized by budget_s
    after an untimed run of `warmup` iterations (which also sizes the sample)."""
    from oracle.oracle import Reference
    from oracle.oracle import Oracle
    ref = Reference()
    step = 0.99 / max(1.0, Oracle().operator_bound(inst.row_offsets, inst.col_idx, inst.values, inst.n))
    secs_w, _, _ = ref.pdhg_replay(inst, step, warmup)
    iters = max(1, min(200, int(budget_s / max(secs_w / warmup, 1e-6))))
    secs, _, _ = ref.pdhg_replay(inst, step, iters)
    return iters / secs, iters, secs


def reference_cpu_end_to_end(small_budget_s=20.0, each_budget_s=8.0):
    """The reference's own end-to-end CPU solve, vikalp::solve(model, options)
    with the default backend preference (its CPU backend, oracle/_ref compiled
    from its sources), on the small LP and on bounded samples of the other
    LP workloads: 4 of the 256 differentiable-workload LPs and 4 of the 256
    independent LPs of the batched workload (sizes spread over the range).
    Each run stops at the reference's own tolerance (1e-6 absolute residuals)
    or at its time budget; the returned point's relative KKT is evaluated by
    the C oracle (the checker). Baseline only."""
    from oracle.oracle import Oracle
    from oracle.oracle import Reference
    from vikalp_b200 import synthetic
    ref, orc = Reference(), Oracle()

    def one(inst, budget):
        t = time.perf_counter()
        r = ref.solve(inst, iteration_limit=10_000_000, time_limit_seconds=budget, primal_tolerance=1e-6,
                      dual_tolerance=1e-6)
        secs = time.perf_counter() - t
        k = orc.rel_kkt(inst, r["x"], r["y"])
        return {"status": r["status"], "iterations": r["iterations"], "seconds": round(secs, 2),
                "rel_kkt": max(k["rel_primal"], k["rel_dual"], k["rel_gap"]), "backend": r["backend"]}

    out = {"small_lp": one(synthetic.workload_small_lp(), small_budget_s)}
    adj = [synthetic.lp_uniform(1000, 2000, 8, seed=7000 + s) for s in (0, 85, 170, 255)]
    out["adjoint_lps_sample"] = [one(i, each_budget_s) for i in adj]
    indep = synthetic.workload_independent_lps(256)
    order = sorted(range(256), key=lambda i: indep[i].m)
    out["independent_lps_sample"] = [dict(one(indep[i], each_budget_s), m=indep[i].m) for i in
                                     (order[0], order[85], order[170], order[255])]
    out["note"] = (f"1 core; per-instance budget {small_budget_s:.0f} s (small LP) / {each_budget_s:.0f} s "
                   "(samples); the reference stops on its absolute 1e-6 residuals")
    return out


def reference_cpu_steps(inst, steps, warmup, budget_s):
    """The reference arm's timing: `warmup` untimed then `steps` timed steps of
    the reference's own CPU PDHG iteration (pdhg.cpp:92-130 call sequence through
    its CPU ExecutionBackend), each step a bounded sample of `per_step`
    iterations (at most one 64-iteration chunk) sized so that the whole run
    stays within about `budget_s` seconds. Returns (iterations/s, per_step,
    timed seconds); steps x ms_per_step equals the timed seconds."""
    from oracle.oracle import Oracle
    from oracle.oracle import Reference
    ref = Reference()
    step = 0.99 / max(1.0, Oracle().operator_bound(inst.row_offsets, inst.col_idx, inst.values, inst.n))
    probe, _, _ = ref.pdhg_replay(inst, step, 2)
    per_iter = max(probe / 2, 1e-6)
    per_step = int(max(1, min(CHUNK, budget_s / ((steps + warmup) * per_iter))))
    ref.pdhg_replay(inst, step, warmup * per_step)
    secs, _, _ = ref.pdhg_replay(inst, step, steps * per_step)
    return steps * per_step / secs, per_step, secs


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["b200", "reference"], default="b200")
    ap.add_argument("--no-ttt", action="store_true", help="skip timing the large LP to 1e-6 relative KKT")
    ap.add_argument("--ttt-seconds", type=float, default=120.0, help="time cap per precision for the large LP")
    ap.add_argument("--no-extras", action="store_true")
    ap.add_argument("--no-batched", action="store_true", help="skip the batched-workload figures")
    ap.add_argument("--profile-spmv", choices=["fp64", "fp32"], default=None,
                    help="only run the sparse-product kernel 5 times on the large LP (for ncu captures)")
    ap.add_argument("--transpose", action="store_true", help="with --profile-spmv: A'y instead of A x")
    ap.add_argument("--profile-shared", type=int, default=0,
                    help="only run the 512-node shared-matrix batch for this many iterations (for ncu captures)")
    ap.add_argument("--profile-iter", type=int, default=0,
                    help="only run this many reference-scheme iterations on the large LP (for ncu captures)")
    ap.add_argument("--profile-halpern", choices=["fp64", "mixed"], default=None,
                    help="only run 256 Halpern-scheme iterations on the large LP (for ncu captures)")
    args = ap.parse_args()
    if args.profile_spmv:
        return profile_spmv(args.profile_spmv, args.transpose)
    if args.profile_iter:
        return profile_iterations(args.profile_iter)
    if args.profile_halpern:
        return profile_halpern(args.profile_halpern)
    if args.profile_shared:
        return profile_shared(args.profile_shared)
    K, W = max(1, args.steps), max(3, args.warmup)
    from vikalp_b200 import replicas
    from vikalp_b200 import synthetic
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    config = {"workload": "lp m=1,000,000 n=2,000,000 nnz~21.1M (Zipf 1.5 column degrees, |a| in 1e-3..1e3)",
              "step": f"{CHUNK} PDHG iterations", "inputs_vs_l2": "inputs larger than L2 (~0.6 GB of matrix per iteration)",
              "parallelism": f"replicas x{ws}"}

    if args.impl == "reference":
        # rank 0 alone times the reference's CPU code; no process group
        if int(os.environ.get("RANK", "0")) != 0:
            return 0
        inst = synthetic.workload_large_lp(seed=12345)
        cores = 1
        try:
            rate, per_step, secs = reference_cpu_steps(inst, K, W, budget_s=100.0)
        except FileNotFoundError:  # its CPU build is made from its source tree
            print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref is not built here"}))
            return 0
        sample = (f"{K} steps of {per_step} iterations each (a bounded sample of the {CHUNK}-iteration step) of "
                  f"the pdhg.cpp:92-130 ExecutionBackend call sequence on the large LP, after {W} untimed steps "
                  f"(its own setup is O(n*nnz) and cannot run)")
        line = {"metric": METRIC, "value": round(rate, 4), "unit": "iter/s", "n_gpus": args.gpus, "steps": K,
                "warmup": W, "ms_per_step": round(secs / K * 1e3, 3), "higher_is_better": True,
                "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic", "impl": "reference",
                "config": dict(config, parallelism="1 CPU core (the reference backend is single-threaded)",
                               reference_step=f"{per_step} PDHG iterations"),
                "cpu_baseline": {"value": round(rate, 4), "unit": "iter/s", "cores": cores, "kind": "reference",
                                 "sample": sample},
                "e2e": {"value": round(rate, 4), "unit": "iter/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
        print(json.dumps(line))
        return 0

    ranks = replicas.init()
    ws, rank, local = ranks.world, ranks.rank, ranks.local
    import torch

    import vikalp_b200 as vk
    torch.cuda.set_device(local)
    stream = torch.cuda.current_stream()
    inst = synthetic.workload_large_lp(seed=12345 + rank)
    # ---- value: resident data, reference scheme -------------------------------
    h = vk.Pdhg(inst, algorithm="reference", check_every=CHUNK)
    # warm-up: W steps
    replicas.barrier(ranks)
    torch.cuda.synchronize()
    _ = solve_with_limit(h, W * CHUNK)
    replicas.barrier(ranks)
    torch.cuda.synchronize()
    with ClockSampler(local) as clk:
        replicas.barrier(ranks)
        torch.cuda.synchronize()
        r = solve_with_limit(h, K * CHUNK)
        torch.cuda.synchronize()
        replicas.barrier(ranks)
    iters = r["iterations"]
    value, t_dev = replicas.whole_job_rate(ranks, iters, r["iterate_seconds"])
    ms_per_step = t_dev / (iters / CHUNK) * 1e3
    launches = r["kernel_launches"]
    # per-kernel device times of the same passes on the same handle (eager
    # launches with CUDA events on the solver's stream, right after the timed region)
    prof = h.profile(2 * CHUNK) if rank == 0 else None
    h.close()
    # ---- e2e: through the C ABI from host arrays ---------------------------------
    # nine calls (each: create with upload and device setup, solve, results
    # back); the median is reported: the host side (page faults of fresh
    # result arrays, driver allocations, a shared host's other work) varies
    # from call to call, by up to ~0.7 s on some boxes
    runs, creates = [], []
    for _ in range(9):
        replicas.barrier(ranks)
        t0 = time.perf_counter()
        with vk.Pdhg(inst, algorithm="reference", iteration_limit=K * CHUNK, primal_tolerance=0.0,
                     dual_tolerance=0.0) as he:
            creates.append(time.perf_counter() - t0)
            r2 = he.solve()
        torch.cuda.synchronize()
        runs.append(replicas.whole_job_rate(ranks, r2["iterations"], time.perf_counter() - t0))
    e2e_rate, t_e2e = sorted(runs)[len(runs) // 2]
    h2d = (inst.row_offsets.nbytes + inst.col_idx.nbytes + inst.values.nbytes + inst.c.nbytes +
           inst.var_lower.nbytes + inst.var_upper.nbytes + inst.row_lower.nbytes + inst.row_upper.nbytes)
    d2h = 8 * (3 * inst.n + 3 * inst.m)  # x, variable duals; y, row duals
    steps_e2e = max(1, r2["iterations"] // CHUNK)
    e2e = {"value": round(e2e_rate, 3), "unit": "iter/s",
           "h2d_bytes_per_step": int(h2d / steps_e2e), "d2h_bytes_per_step": int(d2h / steps_e2e),
           "seconds": round(t_e2e, 3), "runs_seconds": [round(t, 3) for _, t in runs],
           "create_seconds": [round(t, 3) for t in creates],
           "note": "create (upload + device setup) + solve + results, pageable host arrays; median of 9 calls"}
    line = {"metric": METRIC, "value": round(value, 3), "unit": "iter/s", "n_gpus": ws, "steps": iters // CHUNK,
            "warmup": W, "ms_per_step": round(ms_per_step, 3), "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic", "config": config,
            "clocks": clk.summary(), "e2e": e2e, "gpu_launches": int(launches)}
    if rank == 0:
        peak, peak_kind = measured_peaks()
        total = sum(p["ms"] * p["launches"] for p in prof)
        dom = max(prof, key=lambda p: p["ms"] * p["launches"])
        achieved = dom["bytes"] / (dom["ms"] * 1e-3) / 1e9
        traffic, cap_variant, cap_file = profile_traffic(dom["name"])
        live = re.search(r"variant (\d+)", dom["name"])
        live_variant = int(live.group(1)) if live else None
        line["roofline"] = {"bound": "hbm", "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
                            "frac": round(achieved / peak, 4), "traffic": traffic,
                            "traffic_source": f"ncu capture committed in profiles/{cap_file} (kernel variant "
                                              f"{cap_variant}); the timed run's pass ran variant {live_variant}"
                                              + ("" if cap_variant == live_variant else
                                                 " (a different variant: the capture's bytes are indicative)"),
                            "kernel": f"{dom['name']} of the reference-scheme iteration (fp64, FAST order)",
                            "peak_kind": f"{peak_kind} (MEASURED_PEAKS.json hbm_gbs)",
                            "algorithmic_bytes": int(dom["bytes"]), "ms": round(dom["ms"], 4),
                            "passes": [{"kernel": p["name"], "ms": round(p["ms"], 4), "share": round(p["ms"] * p["launches"] / total, 3),
                                        "gbs": round(p["bytes"] / (p["ms"] * 1e-3) / 1e9, 1) if p["bytes"] else None}
                                       for p in prof]}
    if rank == 0 and not args.no_extras:
        sp = spmv_figures(inst, torch, stream)
        line["spmv"] = sp
        # Halpern scheme iteration rate (fp64 and mixed)
        hal = {}
        for prec in ("fp64", "mixed"):
            with vk.Pdhg(inst, algorithm="halpern", precision=prec, check_every=CHUNK) as hh:
                # the first solve tunes the passes and captures the graphs; the second is timed
                solve_with_limit(hh, 2 * CHUNK, rel_tol=0.0)
                rr = solve_with_limit(hh, 10 * CHUNK, rel_tol=0.0)
            hal[prec] = {"iter_per_s": round(rr["iterations"] / rr["iterate_seconds"], 2),
                         "iterations": rr["iterations"]}
        line["halpern"] = hal
        small = synthetic.workload_small_lp()
        ttt = {"small_lp": time_to_tolerance(small, "lp m=2000 n=5000 nnz=40000", 400000)}
        if not args.no_ttt:
            ttt["large_lp"] = time_to_tolerance(inst, "lp m=1e6 n=2e6 nnz=21.1M (the bench's LP)", 2_000_000,
                                                time_limit=args.ttt_seconds, check=True)
        line["time_to_tol"] = ttt
        if not args.no_batched:
            line["batched"] = batched_figures()
            line["adjoint"] = adjoint_figures()
            line["time_to_tol"]["qp"] = time_to_tolerance(synthetic.workload_qp(), "qp m=2e5 n=5e5 A nnz=3M Q nnz=1.1M",
                                                          400000, time_limit=120)
        line["reference_cuda"] = reference_cuda_rate(inst)
        if ws == 1:
            try:
                line["cpu_reference_end_to_end"] = reference_cpu_end_to_end()
                rate, n_it, secs = reference_cpu_rate(inst, budget_s=20.0)
                line["cpu_baseline"] = {"value": round(rate, 4), "unit": "iter/s", "cores": 1, "kind": "reference",
                                        "sample": f"{n_it} iterations of the reference's pdhg.cpp:92-130 call sequence "
                                                  f"(its CPU ExecutionBackend) on the large LP, {secs:.1f} s"}
            except FileNotFoundError:  # the reference's CPU build is made from its source tree
                line["cpu_baseline"] = {"unavailable": "oracle/_ref is not built here"}
    if rank == 0:
        print(json.dumps(line))
    replicas.finish(ranks)
    return 0


def profile_iterations(iterations):
    """`iterations` reference-scheme iterations (fp64, FAST order) on the large LP, for ncu captures."""
    import torch

    import vikalp_b200 as vk
    from vikalp_b200 import synthetic
    inst = synthetic.workload_large_lp()
    with vk.Pdhg(inst, algorithm="reference", check_every=CHUNK) as h:
        r = h.solve(iteration_limit=iterations, primal_tolerance=0.0, dual_tolerance=0.0, duals=False)
    torch.cuda.synchronize()
    print(f"ok iterations={r['iterations']} status={r['status']}")
    return 0


def profile_halpern(precision, iterations=256):
    """`iterations` Halpern-scheme iterations on the large LP (the passes the
    time-to-tolerance figure runs), for ncu captures."""
    import torch

    import vikalp_b200 as vk
    from vikalp_b200 import synthetic
    inst = synthetic.workload_large_lp()
    with vk.Pdhg(inst, algorithm="halpern", precision=precision, check_every=CHUNK) as h:
        r = h.solve(iteration_limit=iterations, relative_tolerance=0.0, duals=False)
    torch.cuda.synchronize()
    print(f"ok iterations={r['iterations']} status={r['status']}")
    return 0


def profile_shared(iterations):
    """The batched workload's node half (512 relaxations of the m=5e4, n=1e5 LP,
    mixed precision) capped at `iterations`, for ncu captures of its SpMM passes."""
    import vikalp_b200 as vk
    from vikalp_b200 import synthetic
    node_lp = synthetic.lp_uniform(50000, 100000, 6, seed=2025)
    lo, hi = synthetic.bnb_nodes(node_lp, 512, seed=7)
    rs = vk.batch_solve_shared(node_lp, 512, lo, hi, precision="mixed", iteration_limit=iterations,
                               relative_tolerance=1e-6)
    print(f"ok status={rs[0]['status']} iterations={rs[0]['iterations']}")
    return 0


def profile_spmv(prec, transpose):
    """Five launches of the sparse-product kernel (PlainEpi) on the large LP."""
    import torch

    import vikalp_b200 as vk
    from vikalp_b200 import synthetic
    inst = synthetic.workload_large_lp()
    dt = torch.float64 if prec == "fp64" else torch.float32
    A = vk.SpMat(inst.row_offsets, inst.col_idx, inst.values, inst.m, inst.n, "fp64" if prec == "fp64" else "mixed")
    xl, yl = (inst.m, inst.n) if transpose else (inst.n, inst.m)
    x = torch.rand(xl, dtype=dt, device="cuda")
    y = torch.zeros(yl, dtype=dt, device="cuda")
    for _ in range(5):
        A.apply(x.data_ptr(), y.data_ptr(), transpose, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    print(f"ok variant={A.variant(transpose)} bytes={A.bytes(transpose)}")
    return 0


def solve_with_limit(h, limit, rel_tol=0.0):
    """One vk_pdhg_solve with a fixed iteration budget (tolerances 0: runs the full budget)."""
    return h.solve(duals=False, iteration_limit=limit, primal_tolerance=0.0, dual_tolerance=0.0,
                   relative_tolerance=rel_tol)


if __name__ == "__main__":
    sys.exit(main())
