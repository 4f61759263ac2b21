"""Benchmark of the B200 PDHG engine on the config-2 LP.

Workload: the seeded random LP with m=40,000 rows, n=80,000 columns and
512,025 nonzeros (6.4 per column, 1% of the rows hold 10% of the nonzeros),
solved by restarted-Halpern PDHG to relative KKT 1e-6.  One step = one full
solve from the cold start.

Metric: time to relative KKT 1e-6, in seconds (lower is better), of the chosen
form -- mixed precision: FP32 iterates, FP64 checks, FP64 verification and
polish -- with the plain FP64 form's time on the same LP reported beside it.
  value : device time of the PDHG loop (CUDA events on the engine's stream),
          with the prepared problem already resident in HBM; L2 is flushed
          (a 512 MiB write) before every step.
  e2e   : the chosen form through the public C ABI (b2p_solve_pdhg) from host
          arrays: host preprocessing, host->device upload, the loop and the
          device->host read of x and y, wall clock per step.
N > 1 (torchrun): N independent replicas of the same solve, one per GPU
("replicas only": a single LP is not partitioned); the reported time is the
maximum over ranks.

``--impl reference`` times the reference's own multithreaded CPU PDHG
(oracle/_ref/libpramana_ref.so, built from the reference sources) on the
host's cores: every timed step is one full solve of the same LP to the same
tolerance (the warm-up steps are short samples).

``--workload family`` runs the learned-warm-start workload instead: a
164 x 324 refinery-planning LP family with 16 parameters (6 crude prices
U(40, 120), 10 demand scales U(0.8, 1.2)); --train members solved by batched
cold PDHG to 1e-6 as training data, the PCA basis and the BF16 tensor-core
MLP trained on the GPU, then --steps held-out batches of --batch members
solved to certified relative KKT 1e-6 from a cold start, from the nearest
training solution and from the network's prediction, plus plain FP64
single-LP solves of a sample of members (the per-instance baseline).

Other workloads (each prints its own line; see their functions):
  multi      uneven batch of config-2-generator LPs through the multi-LP engine
  sweep      256 crude-price cases of the full refinery LP as a shared-A batch
  router     the router's per-engine timings and the refitted model
  plan       the reference's headline refinery plan (plan_60x156) to 1e-4 / 1e-6
  families   the batched leg of the reference's published repeated-solve runs
  calibrate  the reference's six per-iteration calibration LPs
  gemm       the warm-start network's tcgen05 BF16 GEMM at its shapes (TFLOP/s)
  sweep-tol  256-case crude-price sweep of the refinery LP to certified rel KKT 1e-6
``--impl reference --reference-backend gpu`` times the reference's own GPU
backend on this GPU (config-2, or --workload plan / families / calibrate).
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path[:0] = [ROOT, os.path.join(ROOT, "optimized-gpu-accelerator_b200")]

METRIC = "time-to-1e-6 rel KKT (s) & SpMV HBM GB/s: chosen form vs plain FP64 PDHG, B200"
TOL = 1e-6
SEED = 2
CPU_SAMPLE_ITERS = 4096
REF_ITERS_TO_TOL = 20288  # loop iterations of the reference CPU PDHG on this LP to 1e-6 (20,287 reported + 1)


def workload_config(lp, world=1):
    """The workload both arms print, identical for the engine and the reference."""
    return {"workload": f"config-2 random LP m={lp.num_rows} n={lp.num_cols} nnz={lp.nnz} "
                        f"(1% rows hold 10% nnz), seed {SEED}, to rel KKT {TOL:g}",
            "form": "mixed precision (plain FP64 form timed beside it)", "check_every": 64,
            "l2": "flushed before every step (512 MiB device write); the LP itself (~20 MB/iteration) is L2-resident "
                  "within a solve",
            "parallelism": f"replicas x{world}" if world > 1 else "single GPU"}


def answer_errors(objective):
    """Relative objective error of a config-2 answer against the reference's
    FP64 CPU PDHG answer at TOL and against the exact optimum (its dual
    simplex), both stored by tests/golden/make_answers_golden.py."""
    try:
        with open(os.path.join(ROOT, "tests", "golden", "answers.json")) as f:
            a = json.load(f)["config2"]
    except (OSError, KeyError, ValueError):
        return {}
    ref, exact = a[f"{TOL:g}"]["objective"], a["exact"]["objective"]
    return {"objective_rel_err_vs_fp64_oracle": abs(objective - ref) / (1 + abs(ref)),
            "objective_rel_err_vs_exact": abs(objective - exact) / (1 + abs(exact))}


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms while running."""
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index: int):
        self.dev = device_index
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.dev}", f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except (OSError, FileNotFoundError):
            self.proc = None
        return self

    def _read(self):
        for ln in self.proc.stdout:
            self.lines.append(ln.strip())

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            p = [x.strip() for x in ln.split(",")]
            if len(p) < 9:
                continue
            try:
                sm.append(float(p[1]))
                mx.append(float(p[2]))
            except ValueError:
                continue
            for nm, v in zip(names, p[5:9]):
                if v.lower() == "active":
                    reasons.add(nm)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "reasons": sorted(reasons),
                "samples": len(sm)}


def measured_peak():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(p) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    except (OSError, KeyError, ValueError):
        return 6650.0, "fallback"


def ncu_traffic(kernel: str):
    """DRAM bytes (read + write) per unit of work of `kernel` -- the unit the
    roofline uses -- from the committed ncu summary, if any."""
    p = os.path.join(ROOT, "profiles", f"{kernel}_c2_traffic.txt")
    try:
        with open(p) as f:
            for ln in f:
                if ln.startswith("dram_bytes_per_unit:"):
                    return float(ln.split(":", 1)[1])
    except OSError:
        pass
    return None


def cpu_reference_sample(lp, iters: int, threads: int):
    """Reference CPU PDHG (oracle/_ref) for a fixed number of iterations; returns s/iteration."""
    from oracle import oracle as O
    O.set_ref_threads(threads)
    t0 = time.perf_counter()
    O.solve(lp, "ref", tolerance=1e-30, max_iterations=iters)
    wall = time.perf_counter() - t0
    st = O.solve.last_stats
    return st["solve_seconds"] / iters, wall, st


def cpu_reference_solve(lp, threads: int):
    """One full solve of the reference CPU PDHG (oracle/_ref) to TOL from the
    host arrays: (loop seconds, wall seconds, result, stats)."""
    from oracle import oracle as O
    O.set_ref_threads(threads)
    t0 = time.perf_counter()
    r = O.solve(lp, "ref", tolerance=TOL)
    wall = time.perf_counter() - t0
    return O.solve.last_stats["solve_seconds"], wall, r, O.solve.last_stats


def run_reference_gpu(args):
    """--impl reference --reference-backend gpu: the reference's own GPU
    backend (its NVRTC-compiled FP64 kernels, compute_90 PTX run through the
    driver's JIT) on this GPU, full solves of config-2 to 1e-6 (or, with
    --workload plan, of the plan to --plan-tol): the same-hardware comparison
    for this engine.  Not the contract's reference arm, which is the CPU."""
    from oracle import oracle as O
    if not O.available("ref"):
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/libpramana_ref.so was not built"}))
        return 0
    from pramana_b200 import generators as G
    O.solve(G.config1(1), "ref", backend="gpu", tolerance=1e-30, max_iterations=1)
    if O.solve.last_stats["backend"] != "gpu":
        print(json.dumps({"impl": "reference", "unavailable": "the reference's GPU backend did not come up "
                                                               "(it fell back to its CPU backend)"}))
        return 0
    if args.workload in ("families", "calibrate", "sweep"):
        return run_reference_gpu_sets(args, O, G)
    if args.workload == "plan":
        sys.path.insert(0, os.path.join(ROOT, "tests"))
        import lp_cases
        lp, _ = lp_cases.load_plan(args.plan)
        tol, name = args.plan_tol, f"{args.plan} after presolve, to rel KKT {args.plan_tol:g}"
    else:
        lp, tol, name = G.config2(SEED), TOL, workload_config(G.config2(SEED))["workload"]
    loops, walls, kern = [], [], []
    for s in range(args.warmup + args.steps):
        t0 = time.perf_counter()
        r = O.solve(lp, "ref", backend="gpu", tolerance=tol)
        wall = time.perf_counter() - t0
        st = O.solve.last_stats
        if st["backend"] != "gpu":
            print(json.dumps({"impl": "reference", "unavailable": "the reference's GPU backend did not come up "
                                                                   "(it fell back to its CPU backend)"}))
            return 0
        if s >= args.warmup:
            loops.append(st["solve_seconds"])
            walls.append(wall)
            kern.append(st["kernel_seconds"])
    value = statistics.mean(loops)
    line = {"metric": METRIC if args.workload != "plan" else f"time to rel KKT {tol:g} (s), reference refinery plan",
            "value": value, "unit": "s", "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": value * 1e3, "higher_is_better": False, "scaling": "weak", "vs_baseline": None,
            "dtype": "f64", "data": "as the engine's arm", "config": {"workload": name},
            "impl": "reference", "reference_backend": "gpu (the reference's NVRTC kernels, compute_90 PTX, driver JIT)",
            "iterations": st["iterations"], "restarts": st["restarts"], "relative_kkt": r.relative_kkt,
            "kernel_seconds": statistics.mean(kern),
            "e2e": {"value": statistics.mean(walls), "unit": "s", "h2d_bytes_per_step": None,
                    "d2h_bytes_per_step": None}}
    print(json.dumps(line))
    return 0


def run_reference_gpu_sets(args, O, G):
    """The reference's GPU backend on the published families (one batched
    solve per family, 1e-6, 200,000 iterations at most), on the six
    calibration LPs (512 iterations each) or on the 256-case refinery price
    sweep (--sweep-iters iterations of its solvePdhgBatch): loop seconds, wall
    seconds and iterations per item, for the same-hardware comparison."""
    items = []
    if args.workload == "families":
        sys.path.insert(0, os.path.join(ROOT, "tests"))
        import lp_cases
        for fam in lp_cases.FAMILIES:
            lp, cases, _, _ = lp_cases.load_family(fam)
            loops, walls = [], []
            for s in range(args.warmup + args.steps):
                t0 = time.perf_counter()
                rs = O.solve(lp, "ref", cases=cases, backend="gpu", tolerance=1e-6, max_iterations=200000)
                if s >= args.warmup:
                    walls.append(time.perf_counter() - t0)
                    loops.append(O.solve.last_stats["solve_seconds"])
            items.append({"family": fam, "loop_seconds": statistics.mean(loops), "wall_seconds": statistics.mean(walls),
                          "iterations": O.solve.last_stats["iterations"],
                          "solved": sum(r.status == 1 for r in rs), "backend": O.solve.last_stats["backend"]})
    elif args.workload == "sweep":
        import numpy as np
        from pramana_b200 import warmstart as W
        fam = W.RefineryFamily(seed=5)
        rng = np.random.default_rng(9)
        levels = np.linspace(40.0, 120.0, args.cases)
        prices = np.stack([rng.permutation(levels) for _ in range(fam.crudes)], axis=1)
        cases = [fam.case(p) for p in np.hstack([prices, np.ones((args.cases, fam.num_params - fam.crudes))])]
        per, its = [], []
        for s in range(args.warmup + args.steps):
            O.solve(fam.base, "ref", cases=cases, backend="gpu", tolerance=1e-4, max_iterations=args.sweep_iters)
            st = O.solve.last_stats
            if s >= args.warmup:
                per.append(st["solve_seconds"] / st["iterations"])
                its.append(st["iterations"])
        items.append({"cases": args.cases, "iterations_per_step": its, "seconds_per_iteration": statistics.mean(per),
                      "backend": st["backend"]})
    else:
        for scale in G.CALIBRATION_SCALES:
            lp = G.calibration_lp(scale)
            per = []
            for s in range(args.warmup + args.steps):
                O.solve(lp, "ref", backend="gpu", tolerance=1e-30, max_iterations=512)
                st = O.solve.last_stats
                if s >= args.warmup:
                    per.append(st["solve_seconds"] / st["iterations"])
            items.append({"nnz": lp.nnz, "seconds_per_iteration": statistics.mean(per), "backend": st["backend"]})
    print(json.dumps({"impl": "reference", "reference_backend": "gpu (the reference's NVRTC kernels, compute_90 PTX, "
                                                               "driver JIT)", "workload": args.workload,
                      "steps": args.steps, "warmup": args.warmup, "items": items}))
    return 0


def run_reference(args, rank, world):
    """--impl reference: the reference's own CPU PDHG on this host's cores,
    every timed step one full solve of the same LP to the same tolerance."""
    if rank != 0:
        return 0
    if args.reference_backend == "gpu":
        return run_reference_gpu(args)
    if args.steps < 1:
        raise SystemExit("--steps must be >= 1")
    from pramana_b200 import generators as G
    from oracle import oracle as O
    lp = G.config2(SEED)
    threads = os.cpu_count() or 1
    if not O.available("ref"):
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/libpramana_ref.so was not built"}))
        return 0
    # warm-up: bounded samples (thread pool, page cache); timed: full solves
    for _ in range(args.warmup):
        cpu_reference_sample(lp, 512, threads)
    loops, walls, its = [], [], []
    for _ in range(args.steps):
        loop, wall, r, st = cpu_reference_solve(lp, threads)
        assert r.status == 1, r.status
        loops.append(loop)
        walls.append(wall)
        its.append(r.iterations)
    value = statistics.mean(loops)
    sample = (f"{args.steps} full solves to rel KKT {TOL:g} ({its[-1]} iterations each), loop time; the "
              f"{args.warmup} warm-up steps are 512-iteration samples")
    line = {"metric": METRIC, "value": value, "unit": "s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": value * 1e3, "higher_is_better": False, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded generator)",
            "config": workload_config(lp, world), "impl": "reference",
            "run": {"iterations": its[-1], "relative_kkt": r.relative_kkt, "wall_seconds": statistics.mean(walls)},
            "cpu_baseline": {"value": value, "unit": "s", "cores": threads, "kind": "reference", "sample": sample},
            "e2e": {"value": value, "unit": "s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))
    return 0


# Sizes of the refinery-planning family (generators.refinery_lp, unit row and
# column scales): small 164 x 324 (1,072 nonzeros), medium 1,692 x 3,528
# (14,982), large 5,064 x 11,376 (57,178).
FAMILY_SIZES = {
    "small": dict(periods=2, regions=1, units=4, streams=4, properties=2, scale_exponent=0.0),
    "medium": dict(periods=6, regions=2, units=6, streams=6, properties=3, pools=12, scale_exponent=0.0),
    "large": dict(periods=12, regions=2, units=8, streams=8, properties=4, pools=12, scale_exponent=0.0),
}
FAMILY_SIZE = FAMILY_SIZES["small"]
FAMILY_METRIC = "wall time per 1,024-member refinery family batch to certified rel KKT 1e-6 (s), learned warm start"


def run_family(args, rank, world):
    """--workload family: learned warm start vs cold and nearest-neighbour starts."""
    import numpy as np
    import torch

    from pramana_b200 import pdhg
    from pramana_b200 import warmstart as W
    from pramana_b200.mlp import TrainOptions

    if world > 1 and rank != 0:
        return 0
    torch.cuda.set_device(0)
    size = FAMILY_SIZES[args.family_size]
    fam = W.RefineryFamily(seed=5, **size)
    precision = {"fp64": 0, "mixed": 1}[args.precision]
    # the batched engine's form, and the plain FP64 single-LP form of the per-instance baseline
    opts = pdhg.PdhgOptions(tolerance=TOL, maxIterations=args.family_max_iters, precision=precision)
    plain = pdhg.PdhgOptions(tolerance=TOL, maxIterations=args.family_max_iters, precision=0)
    t0 = time.perf_counter()
    P_train = fam.sample(args.train, 100)
    tr = W.solve_family(fam, P_train, opts, batch=args.batch, engine=args.engine)
    gen_s = time.perf_counter() - t0
    ok = tr.status == 1
    lw = W.LearnedWarmStart(fam, seed=1)
    losses = lw.fit(P_train[ok], tr.X[ok], tr.Y[ok],
                    TrainOptions(epochs=args.epochs, batch=512, lr=1e-3, lr_final=1e-5, seed=2))
    nn = W.NearestWarmStart(fam).fit(P_train[ok], tr.X[ok], tr.Y[ok])
    use_w = args.family_weights == "nearest" and args.engine == "multi"
    est = W.WorkEstimate(fam).fit(P_train[ok], tr.iterations[ok], tr.weights[ok] if use_w else None)
    strategies = {"cold": None, "nearest": nn, "learned": lw}

    def start_weights(name, params):
        # warm-started strategies also start from the nearest members' primal weights
        return est.predict_weight(params) if use_w and name != "cold" else None

    # untimed warm-up batches (module loads, variant tuning, pools): the first at full size, the
    # others of 128 members
    for w in range(args.warmup):
        size_w = args.batch if w == 0 else min(args.batch, 128)
        Pw = fam.sample(size_w, 900 + w)
        W.solve_warm(fam, Pw, lw, opts, batch=args.batch, engine=args.engine, work=est.predict(Pw),
                     weights=start_weights("learned", Pw), warm_max_iterations=args.warm_max_iters,
                     continue_failed=args.continue_failed)
    acc = {k: {"seconds": [], "solve_seconds": [], "iterations": [], "certified": [], "fallback": [], "kkt": []}
           for k in strategies}
    with ClockSampler(0) as clk:
        for step in range(args.steps):
            P = fam.sample(args.batch, 200 + step)
            for name, pred in strategies.items():
                torch.cuda.synchronize()
                t1 = time.perf_counter()
                r, cert, redo = W.solve_warm(fam, P, pred, opts, batch=args.batch, engine=args.engine,
                                             work=est.predict(P), weights=start_weights(name, P),
                                             warm_max_iterations=args.warm_max_iters,
                                             continue_failed=args.continue_failed)
                wall = time.perf_counter() - t1
                a = acc[name]
                a["seconds"].append(wall)
                a["solve_seconds"].append(r.solve_seconds)
                a["iterations"].append(r.iterations)
                a["certified"].append(cert["certified"])
                a["fallback"].append(redo if pred is not None else np.zeros(len(P), dtype=bool))
                a["kkt"].append(cert["kkt"][:, 3])
    # per-instance baseline: plain FP64 single-LP solves, one member at a time
    P = fam.sample(args.per_instance_sample, 700)
    per = []
    its1 = []
    for p in P:
        lp = fam.instance(p)
        torch.cuda.synchronize()
        t1 = time.perf_counter()
        r = pdhg.solvePdhg(lp, plain)
        per.append(time.perf_counter() - t1)
        its1.append(r.iterations)
    per_instance_batch = statistics.mean(per) * args.batch
    out = {}
    for name, a in acc.items():
        it = np.concatenate(a["iterations"])
        out[name] = {"seconds_per_batch": statistics.mean(a["seconds"]),
                     "solve_seconds_per_batch": statistics.mean(a["solve_seconds"]),
                     "iterations_mean": float(it.mean()), "iterations_median": float(np.median(it)),
                     "iterations_p95": float(np.percentile(it, 95)), "iterations_max": int(it.max()),
                     "certified_fraction": float(np.concatenate(a["certified"]).mean()),
                     "certification_failures": int((~np.concatenate(a["certified"])).sum()),
                     "fallback_fraction": float(np.concatenate(a["fallback"]).mean()),
                     "max_relative_kkt": float(np.concatenate(a["kkt"]).max())}
    value = out["learned"]["seconds_per_batch"]
    b = fam.base
    line = {"metric": FAMILY_METRIC, "value": value, "unit": "s", "n_gpus": 1, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": value * 1e3, "higher_is_better": False, "scaling": "weak",
            "vs_baseline": None,
            "dtype": {"fp64": "f64 PDHG", "mixed": "f32 iterates / f64 checks, re-measure and polish"}[args.precision]
            + ", bf16 MLP with f32 accumulation", "data": "synthetic (seeded)",
            "workload": "family",
            "config": {"workload": f"refinery-planning family ({args.family_size}), {b.num_rows} rows x "
                                   f"{b.num_cols} cols, {b.nnz} nnz ({size}), 16 parameters; {args.train} training "
                                   f"members, {args.steps} x {args.batch} held-out members, to rel KKT {TOL:g}",
                       "precision": args.precision,
                       "step": "one held-out batch solved and certified per strategy",
                       "launch_order": "members in decreasing predicted work (mean cold iterations of the 4 nearest "
                                       "training members), every strategy",
                       "warm_max_iterations": args.warm_max_iters or args.family_max_iters,
                       "fallback": ("members that fail certification continue from their final point and "
                                    "primal weight, then what still fails re-solves cold" if args.continue_failed else
                                    "members that fail certification re-solved cold by the same engine"),
                       "primal_weights": ("warm strategies start from the geometric mean of the 4 nearest training "
                                          "members' final primal weights" if use_w else "default (||c|| / ||b||)"),
                       "engine": {"multi": "multi-LP engine (AUTO form: one thread block per member)",
                                  "batch": "shared-A batch engine (k-interleaved cases)"}[args.engine],
                       "network": lw.widths, "pca_rank": lw.rank, "pca_explained": lw.basis.explained,
                       "l2": "inputs re-uploaded per batch; the batch state (~4 MB) is L2-resident"},
            "strategies": out,
            "training": {"members": args.train, "solved": int(ok.sum()), "data_generation_s": gen_s,
                         "mlp_train_s": lw.train_seconds, "epochs": args.epochs,
                         "final_loss": float(losses[-1]), "first_loss": float(losses[0])},
            "per_instance_fp64": {"members_timed": len(per), "seconds_per_member": statistics.mean(per),
                                  "iterations_mean": float(np.mean(its1)),
                                  "seconds_per_batch_extrapolated": per_instance_batch},
            "speedup_vs_per_instance_fp64": per_instance_batch / value,
            "clocks": clk.summary()}
    print(json.dumps(line))
    return 0


ROUTER_METRIC = "held-out geo-mean regret of the B200-calibrated engine router (time of chosen engine / fastest)"


def router_instances():
    """Seeded LPs from four generator families (the calibration set)."""
    from pramana_b200 import generators as G
    out = []
    for i, m in enumerate([100, 200, 400, 800, 1500, 3000, 6000]):
        for d in (3.0, 6.0):
            out.append(("random", f"random_m{m}_d{d:g}", G.random_lp(m, 2 * m, d, int(0.6 * m), 500 + 10 * i + int(d))))
    for i, m in enumerate([500, 1000, 2000, 4000, 8000]):
        out.append(("skewed", f"skewed_m{m}", G.random_lp(m, 2 * m, 6.4, int(0.6 * m), 700 + i, heavy_row_frac=0.01,
                                                          heavy_nnz_frac=0.1)))
    for i, (T, R_, U, S, Q, e) in enumerate([(1, 1, 2, 3, 2, 0.0), (2, 1, 4, 4, 2, 0.0), (3, 1, 4, 4, 2, 0.0),
                                             (2, 2, 4, 6, 3, 0.0), (4, 2, 6, 6, 3, 0.0), (1, 1, 2, 3, 2, 1.0),
                                             (2, 1, 4, 4, 2, 1.0), (3, 2, 4, 6, 3, 1.0)]):
        out.append(("refinery", f"refinery_{T}x{R_}x{U}x{S}x{Q}_e{e:g}",
                    G.refinery_lp(periods=T, regions=R_, units=U, streams=S, properties=Q, pools=10, seed=900 + i,
                                  scale_exponent=e)))
    for i, lp in enumerate(G.uneven_family(6, 1e4, 6e4, seed=11)):
        out.append(("uneven", f"uneven_{i}_nnz{lp.nnz}", lp))
    return out


def run_router(args, rank, world):
    """--workload router: every LP of the calibration set solved by the four
    engines the router chooses between -- this library's GPU PDHG through the
    public call ("pdhg-gpu") and the reference's CPU engines on this host's
    cores (dual simplex, interior point with crossover, CPU PDHG; oracle/_ref)
    -- with a time limit; the router's log-linear model is fitted on these
    timings, validated on held-out LPs, and written in Router::load's format."""
    import torch

    from oracle import oracle as O
    from pramana_b200 import pdhg
    from pramana_b200 import router as R

    if world > 1 and rank != 0:
        return 0
    torch.cuda.set_device(0)
    if not O.available("ref"):
        print(json.dumps({"workload": "router", "unavailable": "oracle/_ref/libpramana_ref.so was not built"}))
        return 0
    threads = os.cpu_count() or 1
    O.set_ref_threads(threads)
    limit = args.router_limit
    tol = 1e-6
    insts = router_instances()
    pdhg.solvePdhg(insts[0][2], pdhg.PdhgOptions(tolerance=tol))  # module load, pools
    records, rows = [], []
    for fam, name, lp in insts:
        times, stats = {}, {}
        # the reference's CPU PDHG wrapper sets PRAMANA_DISABLE_GPU (C setenv) to
        # keep the reference off the GPU; this engine honours the variable too
        os.unsetenv("PRAMANA_DISABLE_GPU")
        t0 = time.perf_counter()
        r = pdhg.solvePdhg(lp, pdhg.PdhgOptions(tolerance=tol, timeLimit=limit))
        t = time.perf_counter() - t0
        times["pdhg-gpu"], stats["pdhg-gpu"] = (t if r.status == "Optimal" else None), r.status
        t0 = time.perf_counter()
        o = O.solve(lp, "ref", tolerance=tol, time_limit=limit)
        t = time.perf_counter() - t0
        times["pdhg-cpu"], stats["pdhg-cpu"] = (t if o.status == 1 else None), int(o.status)
        for e in ("dual", "ipm"):
            s = O.timed_solve(lp, e, limit)
            times[e], stats[e] = (s["seconds"] if s["status"] == "Optimal" else None), s["status"]
        rec = R.Record(name=name, family=fam, features=R.features(lp), times=times, limit=limit, statuses=stats)
        records.append(rec)
        rows.append({"instance": name, "family": fam, **{f"t_{e}": times[e] for e in R.ENGINES},
                     **{f"status_{e}": stats[e] for e in R.ENGINES}, **rec.features})
    val = R.validate(records, tolerance=tol)
    W = R.fit(records)
    os.makedirs(args.router_out, exist_ok=True)
    R.write_model(os.path.join(args.router_out, "router_model_b200.json"), W, len(records),
                  note=f"fitted on {len(records)} seeded LPs timed on one B200 and {threads} host threads; "
                       f"time limit {limit:g} s, rel KKT {tol:g} for the PDHG engines")
    with open(os.path.join(args.router_out, "router_runs.json"), "w") as fh:
        json.dump(rows, fh, indent=1)
    line = {"metric": ROUTER_METRIC, "value": val["router_held_out"]["geo_mean_regret"], "unit": "x",
            "n_gpus": 1, "steps": 1, "warmup": 1, "higher_is_better": False, "scaling": "weak", "vs_baseline": None,
            "dtype": "f64", "data": "synthetic (seeded)", "workload": "router",
            "config": {"workload": f"{len(records)} LPs from 4 generator families (random, skewed, refinery, "
                                   f"uneven config-2), 4 engines each, time limit {limit:g} s, 5-fold held-out",
                       "timing": "a calibration pass, not a repeated bench: each LP solved once per engine (as "
                                 "the reference's router fitting times them), after one warm-up solve",
                       "host_threads": threads},
            "validation": val, "weights": W}
    print(json.dumps(line))
    return 0


SWEEP_METRIC = "HBM GB/s of the batched PDHG kernels: 256-case crude-price sweep of the full refinery LP (shared A)"


def run_plan(args, rank, world):
    """--workload plan: a refinery planning LP of the reference's published
    runs (default plan_60x156, 135,876 x 191,568 after presolve, 561,067
    nonzeros; tests/golden/plans/, made by tests/golden/make_plan_golden.py)
    solved to --plan-tol (default 1e-4, the tolerance of the reference's
    published headline run) in the plain FP64 and the mixed form: device time
    of the loop (problem resident in HBM), end to end through solvePdhg from
    host arrays, and the reference's CPU PDHG on this host's cores for the
    first --cpu-sample-iters iterations, scaled to the published iteration
    count.  The line also carries the reference's published times for the
    same run (other hardware)."""
    import torch
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    import lp_cases
    from pramana_b200 import _lib, pdhg

    torch.cuda.set_device(0)
    dev = torch.cuda.current_device()
    lp, pub = lp_cases.load_plan(args.plan)
    run = "pdhg-cpu_raw1e-4" if args.plan_tol >= 1e-4 else "pdhg-gpu_raw1e-6"
    p = pub[run]
    flush = torch.empty(512 * 1024 * 1024, dtype=torch.uint8, device=f"cuda:{dev}")
    forms = {}
    launches = 0
    with ClockSampler(dev) as clk:
        for name, prec in (("plain_fp64", _lib.PRECISION_FP64), ("mixed", _lib.PRECISION_MIXED)):
            po = pdhg.PdhgOptions(tolerance=args.plan_tol, device=dev, precision=prec)
            eng = pdhg.Engine(lp, po)
            times = []
            for s in range(args.warmup + args.steps):
                flush.zero_()
                torch.cuda.synchronize()
                r = eng.solve()[0]
                st = eng.last_stats
                assert r.status == "Optimal", r.status
                if s >= args.warmup:
                    times.append(st.kernel_seconds)
                    launches += st.kernel_launches
            forms[name] = {"value": statistics.mean(times), "iterations": r.iterations + 1,
                           "restarts": st.restarts, "relative_kkt": r.relativeKkt, "objective": r.objective,
                           "kernel_form": {1: "fused", 2: "resident"}.get(st.kernel_mode, "?")}
            eng.close()
    chosen = min(forms, key=lambda f: forms[f]["value"])
    po = pdhg.PdhgOptions(tolerance=args.plan_tol, device=dev,
                          precision=_lib.PRECISION_MIXED if chosen == "mixed" else _lib.PRECISION_FP64)
    e2e = []
    for s in range(args.warmup + args.steps):
        flush.zero_()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        r = pdhg.solvePdhg(lp, po)
        if s >= args.warmup:
            e2e.append(time.perf_counter() - t0)
    cpu = None
    if not args.no_cpu_baseline:
        from oracle import oracle as O
        if O.available("ref"):
            threads = os.cpu_count() or 1
            spi, wall, _ = cpu_reference_sample(lp, args.cpu_sample_iters, threads)
            cpu = {"value": spi * p["iterations"], "unit": "s", "cores": threads, "kind": "reference",
                   "sample": f"first {args.cpu_sample_iters} of {p['iterations']} iterations of the same LP "
                             f"({wall:.1f} s), scaled by iteration count"}
    line = {"metric": f"time to rel KKT {args.plan_tol:g} (s), reference refinery plan", "value": forms[chosen]["value"],
            "unit": "s", "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": forms[chosen]["value"] * 1e3, "higher_is_better": False, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64" if chosen == "plain_fp64" else "f32 iterates, f64 checks and polish",
            "data": "the reference's generated refinery planning model, presolved by its own presolve",
            "workload": "plan",
            "config": {"workload": f"{args.plan} after presolve: m={lp.num_rows} n={lp.num_cols} nnz={lp.nnz}, "
                                   f"to rel KKT {args.plan_tol:g}", "chosen_form": chosen,
                       "l2": "flushed before every step (512 MiB device write)"},
            "forms": forms,
            "published_reference_run": {k: p[k] for k in ("iterations", "restarts", "relative_kkt", "objective",
                                                          "solve_seconds") if k in p} | {"hardware": p["device"]},
            "e2e": {"value": statistics.mean(e2e), "unit": "s", "h2d_bytes_per_step": r.stats.bytesUploaded,
                    "d2h_bytes_per_step": r.stats.bytesDownloaded},
            "gpu_launches": launches, "clocks": clk.summary(), "cpu_baseline": cpu}
    if rank == 0:
        print(json.dumps(line))
    return 0


C3_METRIC = "time to rel KKT 1e-6 (s), full-size config-3 refinery LP, mixed precision"


def run_c3(args, rank, world):
    """--workload c3: the config-3 refinery planning LP at full size (the
    generator's 12 periods x 6 crudes x 10 units x 15 pools x 10 regions,
    48,072 x 99,144, 756,660 nonzeros), with unit row and column scales and
    with the 10^U(-3,3) rescaling, each solved once per (tolerance 1e-4 /
    1e-6, plain FP64 / mixed) under --c3-max-iters: status, iterations,
    device time, the KKT recomputed on the device from the returned point,
    the mixed answer's distance to the FP64 one, and the outward-rounded
    dual bound over the constraint-implied column bounds.  One solve per
    form: a 1e-6 solve is ~2,000,000 iterations (~20 s)."""
    import numpy as np
    import torch

    from pramana_b200 import _lib, pdhg
    from pramana_b200 import generators as G
    from pramana_b200.model import LpCase

    if world > 1 and rank != 0:
        return 0
    torch.cuda.set_device(0)
    results = {}
    launches = 0
    with ClockSampler(0) as clk:
        for scaling, expo in (("unit", 0.0), ("rescaled", 3.0)):
            lp = G.refinery_lp(seed=5, scale_exponent=expo)
            lo, up = pdhg.impliedBounds(lp)
            box = [LpCase(col_lower=lo[0], col_upper=up[0])]
            for tol in (1e-4, 1e-6):
                ref = None
                for form, prec in (("fp64", _lib.PRECISION_FP64), ("mixed", _lib.PRECISION_MIXED)):
                    r = pdhg.solvePdhg(lp, pdhg.PdhgOptions(tolerance=tol, maxIterations=args.c3_max_iters,
                                                            precision=prec))
                    launches += r.stats.kernelLaunches
                    kkt = pdhg.kktResidual(lp, r.x, r.rowDual)[0]
                    lb = pdhg.safeDualBound(lp, r.rowDual, box)[0]["bound"] + lp.obj_offset
                    rec = {"status": r.status, "iterations": r.iterations, "fp32_iterations": r.stats.fp32Iterations,
                           "seconds": r.stats.kernelSeconds, "objective": r.objective,
                           "relative_kkt": float(kkt[3]), "kkt_parts": [float(v) for v in kkt[:3]],
                           "certified_bound": lb,
                           "bound_gap": (abs(r.objective - lb) / (1 + abs(r.objective))) if np.isfinite(lb) else None}
                    if ref is None:
                        ref = r
                    else:
                        rec["objective_vs_fp64"] = abs(r.objective - ref.objective) / (1 + abs(ref.objective))
                        rec["x_vs_fp64"] = float(np.linalg.norm(r.x - ref.x) / (1 + np.linalg.norm(ref.x)))
                    results[f"{scaling}_{tol:g}_{form}"] = rec
    head = results["unit_1e-06_mixed"]
    cpu = None
    if not args.no_cpu_baseline:
        from oracle import oracle as O
        if O.available("ref"):
            lp = G.refinery_lp(seed=5, scale_exponent=0.0)
            threads = os.cpu_count() or 1
            spi, wall, _ = cpu_reference_sample(lp, args.cpu_sample_iters, threads)
            cpu = {"value": spi * head["iterations"], "unit": "s", "cores": threads, "kind": "reference",
                   "sample": f"first {args.cpu_sample_iters} iterations of the unit-scale LP ({wall:.1f} s), "
                             f"scaled to the mixed 1e-6 solve's {head['iterations']} iterations"}
    line = {"metric": C3_METRIC, "value": head["seconds"], "unit": "s", "n_gpus": 1, "steps": 1, "warmup": 0,
            "ms_per_step": head["seconds"] * 1e3, "higher_is_better": False, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32 iterates, f64 checks and polish (the fp64 forms: f64)",
            "data": "synthetic (seeded generator)", "workload": "c3",
            "config": {"workload": "refinery LP 48072 rows x 99144 cols, 756660 nnz (12 periods, 6 crudes, 10 units, "
                                   "15 pools, 10 regions), unit scales and 10^U(-3,3)-rescaled, to rel KKT 1e-4 and "
                                   f"1e-6, at most {args.c3_max_iters} iterations per solve",
                       "steps": "one solve per form (about 20 s each at 1e-6)"},
            "results": results, "gpu_launches": launches, "clocks": clk.summary(), "cpu_baseline": cpu}
    print(json.dumps(line))
    return 0


def run_families(args, rank, world):
    """--workload families: the batched-PDHG leg of the reference's published
    repeated-solve experiment (compareFamilyStrategies; tests/golden/families/,
    made by tests/golden/make_family_golden.py): per family, K crude-price or
    crude-availability cases of a refinery plan in one solvePdhgBatch call
    (1e-6, at most 200,000 iterations) from host arrays, then the
    outward-rounded dual bound over constraint-implied column bounds for every
    solved case, timed together as the reference times its strategy; the
    published figures of the same runs (other hardware) ride along."""
    import torch
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    import lp_cases
    from pramana_b200 import pdhg

    torch.cuda.set_device(0)
    dev = torch.cuda.current_device()
    rows = {}
    launches = 0
    with ClockSampler(dev) as clk:
        for fam in lp_cases.FAMILIES:
            lp, cases, exact, pub = lp_cases.load_family(fam)
            po = pdhg.PdhgOptions(tolerance=1e-6, maxIterations=200000, device=dev)
            times = []
            for s in range(args.warmup + args.steps):
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                st = pdhg.PdhgStats()
                rs = pdhg.solvePdhgBatch(lp, cases, po, batchStats=st)
                cert = lp_cases.family_certified(lp, cases, rs, pdhg.safeDualBound, pdhg.impliedBounds)
                if s >= args.warmup:
                    times.append(time.perf_counter() - t0)
                    launches += st.kernelLaunches
            solved = [b for b, r in enumerate(rs) if r.status == "Optimal"]
            err = max((abs(rs[b].objective - exact[b]) / max(1.0, abs(exact[b])) for b in solved), default=0.0)
            rows[fam] = {"seconds": statistics.mean(times), "kernel_seconds": st.kernelSeconds,
                         "iterations": st.iterations, "cases": len(cases), "solved": len(solved), "certified": cert,
                         "max_relative_error": err,
                         "published_gpu": {k: pub["gpu"][k] for k in ("seconds", "iterations", "solved", "certified",
                                                                      "max_relative_error")},
                         "published_cpu_seconds": pub["cpu"]["seconds"], "published_device": pub["device"]}
    total = sum(r["seconds"] for r in rows.values())
    line = {"metric": "seconds per batched family solve + safe bounds (reference's repeated-solve experiment)",
            "value": total, "unit": "s", "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": total * 1e3, "higher_is_better": False, "scaling": "weak", "vs_baseline": None,
            "dtype": "f64", "data": "the reference's refinery plans and published parameter grids",
            "workload": "families",
            "config": {"workload": "4 published families: plan_10x12 CR03 price / availability (64 cases each), "
                                   "plan_20x12 CR07 price (64), plan_20x52 CR05 availability (32); 1e-6, "
                                   "200,000 iterations at most; value = sum over the families"},
            "families": rows, "gpu_launches": launches, "clocks": clk.summary(), "cpu_baseline": None}
    if rank == 0:
        print(json.dumps(line))
    return 0


def run_calibrate(args, rank, world):
    """--workload calibrate: the reference's PDHG per-iteration calibration
    (calibrateBandwidth, src/parametric/parametric.cpp:531-585) on this
    engine: its six random transportation-like LPs (1e3 to 1e6 rows, 8k to 8M
    nonzeros; generators.calibration_lp), 512 iterations of the plain FP64
    form each (tolerance 1e-30), seconds per iteration from the device loop
    and from the host's loop clock, and the reference's "effective GB/s"
    (24 nnz + 80 (m + n) bytes per iteration).  The reference's CPU PDHG on
    this host's cores runs a bounded sample of each instance (cpu_baseline);
    the published laptop figures (tests/golden/calibration_published.json)
    ride along."""
    import torch
    from pramana_b200 import _lib, pdhg
    from pramana_b200 import generators as G

    torch.cuda.set_device(0)
    dev = torch.cuda.current_device()
    with open(os.path.join(ROOT, "tests", "golden", "calibration_published.json")) as f:
        pub = json.load(f)
    iters = 512
    rows = []
    launches = 0
    cpu_rows = []
    threads = os.cpu_count() or 1
    with ClockSampler(dev) as clk:
        for k, scale in enumerate(G.CALIBRATION_SCALES):
            lp = G.calibration_lp(scale)
            po = pdhg.PdhgOptions(tolerance=1e-30, maxIterations=iters, device=dev, precision=_lib.PRECISION_FP64)
            eng = pdhg.Engine(lp, po)
            dev_t, host_t = [], []
            for s in range(args.warmup + args.steps):
                eng.solve()
                st = eng.last_stats
                if s >= args.warmup:
                    dev_t.append(st.kernel_seconds / st.iterations)
                    host_t.append(st.solve_seconds / st.iterations)
                    launches += st.kernel_launches
            eng.close()
            per = statistics.mean(dev_t)
            model_bytes = 24.0 * lp.nnz + 80.0 * (lp.num_rows + lp.num_cols)
            p = pub["scales"][k]
            rows.append({"rows": lp.num_rows, "cols": lp.num_cols, "nnz": lp.nnz,
                         "seconds_per_iteration": per, "host_loop_seconds_per_iteration": statistics.mean(host_t),
                         "effective_GBs": model_bytes / per / 1e9,
                         "published_gpu_seconds_per_iteration": p["gpu_seconds_per_iteration"],
                         "published_cpu_seconds_per_iteration": p["cpu_seconds_per_iteration"],
                         "speedup_vs_published_gpu": p["gpu_seconds_per_iteration"] / per})
    if not args.no_cpu_baseline:
        from oracle import oracle as O
        if O.available("ref"):
            for scale in G.CALIBRATION_SCALES:
                lp = G.calibration_lp(scale)
                n_s = 128 if lp.nnz < 1e6 else 32
                spi, wall, _ = cpu_reference_sample(lp, n_s, threads)
                cpu_rows.append({"nnz": lp.nnz, "seconds_per_iteration": spi, "sample_iterations": n_s})
    big = rows[-1]
    line = {"metric": "PDHG seconds per iteration, the reference's calibration LPs (largest: 8M nonzeros)",
            "value": big["seconds_per_iteration"], "unit": "s", "n_gpus": 1, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": big["seconds_per_iteration"] * iters * 1e3,
            "higher_is_better": False, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "the reference's calibration generator (SplitMix64 seed 7), restated", "workload": "calibrate",
            "config": {"workload": "6 random transportation-like LPs, 1e3..1e6 rows, 512 iterations each; "
                                   "value = the 1e6-row instance"},
            "scales": rows, "published_hardware": {"gpu": pub["gpu"], "cpu_threads": pub["cpu_threads"]},
            "gpu_launches": launches, "clocks": clk.summary(),
            "cpu_baseline": ({"value": cpu_rows[-1]["seconds_per_iteration"], "unit": "s", "cores": threads,
                              "kind": "reference", "sample": "per scale: " + json.dumps(cpu_rows)}
                             if cpu_rows else None)}
    if rank == 0:
        print(json.dumps(line))
    return 0


def run_sweep(args, rank, world):
    """--workload sweep: 256 cases of the full-size refinery LP (the config-3
    generator: 42,072 rows, 97,344 columns, 748,910 nonzeros, rows and columns
    rescaled by 10^U(-3,3)) whose 6 crude prices sweep a seeded grid over
    40-120 $/bbl, solved as one shared-A batch (k-interleaved vectors).  PDHG
    does not bring this rescaled LP to rel KKT 1e-4 within 200,000 iterations,
    so a step is a fixed block of --sweep-iters iterations (rel KKT 1e-4,
    capped), and the line reports the batch kernels' bandwidth."""
    import numpy as np
    import torch

    from pramana_b200 import pdhg
    from pramana_b200 import warmstart as W

    if world > 1 and rank != 0:
        return 0
    torch.cuda.set_device(0)
    fam = W.RefineryFamily(seed=5)
    base = fam.base
    K = args.cases
    rng = np.random.default_rng(9)
    levels = np.linspace(40.0, 120.0, K)
    prices = np.stack([rng.permutation(levels) for _ in range(fam.crudes)], axis=1)
    params = np.hstack([prices, np.ones((K, fam.num_params - fam.crudes))])
    cases = [fam.case(p) for p in params]
    iters = args.sweep_iters
    opts = pdhg.PdhgOptions(tolerance=1e-4, maxIterations=iters)
    flush = torch.empty(512 * 1024 * 1024, dtype=torch.uint8, device="cuda:0")
    eng = pdhg.Engine(base, opts, cases)
    for _ in range(args.warmup):
        eng.solve()
    dev = []
    with ClockSampler(0) as clk:
        for _ in range(args.steps):
            flush.zero_()
            torch.cuda.synchronize()
            rs = eng.solve()
            dev.append(eng.last_stats.kernel_seconds)
    st = eng.last_stats
    t_dev = statistics.mean(dev)
    # per-kernel times and bytes: one profiled solve (events around every launch)
    eng.set_profiling(True)
    flush.zero_()
    torch.cuda.synchronize()
    eng.solve()
    eng.set_profiling(False)
    prof = {}
    for cls, name in ((0, "k_primal"), (1, "k_dual")):
        n_l, ms = eng.kernel_times(cls)
        prof[name] = {"launches": n_l, "avg_us": ms / n_l * 1e3, "bytes_per_launch": eng.kernel_bytes(cls),
                      "gbs": eng.kernel_bytes(cls) / (ms / n_l / 1e3) / 1e9}
    eng.close()
    # the same batch in the mixed form: the FP32 k-interleaved kernels (classes 3 and 4)
    eng32 = pdhg.Engine(base, pdhg.PdhgOptions(tolerance=1e-4, maxIterations=iters, precision=1), cases)
    eng32.solve()
    eng32.set_profiling(True)
    flush.zero_()
    torch.cuda.synchronize()
    eng32.solve()
    eng32.set_profiling(False)
    prof32 = {}
    for cls, name in ((3, "k_primal32"), (4, "k_dual32")):
        n_l, ms = eng32.kernel_times(cls)
        if n_l:
            prof32[name] = {"launches": n_l, "avg_us": ms / n_l * 1e3, "bytes_per_launch": eng32.kernel_bytes(cls),
                            "gbs": eng32.kernel_bytes(cls) / (ms / n_l / 1e3) / 1e9}
    eng32.close()
    nnz, m, n = base.nnz, base.num_rows, base.num_cols
    ref_model = 24.0 * nnz + 80.0 * (m + n) * K  # the reference's effective-bandwidth model, per iteration
    fused_bytes = sum(p["bytes_per_launch"] for p in prof.values())
    fused_s = sum(p["avg_us"] for p in prof.values()) / 1e6
    peak, peak_kind = measured_peak()
    # e2e: the public batch call from host arrays (set-up, uploads, loop, downloads)
    e2e = []
    h2d = d2h = 0
    for s_ in range(args.warmup + args.steps):
        flush.zero_()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        rb = pdhg.solvePdhgBatch(base, cases, opts)
        t1 = time.perf_counter()
        if s_ >= args.warmup:
            e2e.append(t1 - t0)
            h2d, d2h = rb[0].stats.bytesUploaded, rb[0].stats.bytesDownloaded
    t_e2e = statistics.mean(e2e)
    # the same cases one at a time (plain FP64 single-LP engine): per-iteration time of one case
    single = pdhg.solvePdhg(fam.instance(params[0]), opts)
    t_single = single.stats.kernelSeconds / max(1, single.iterations)
    dominant = max(prof, key=lambda k: prof[k]["avg_us"])
    achieved = prof[dominant]["gbs"]
    line = {"metric": SWEEP_METRIC, "value": fused_bytes / fused_s / 1e9, "unit": "GB/s", "n_gpus": 1,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": t_dev * 1e3, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded)",
            "workload": "sweep",
            "config": {"workload": f"refinery LP {m} rows x {n} cols, {nnz} nnz (rows/cols rescaled 10^U(-3,3)), "
                                   f"{K} cases with the 6 crude prices on a seeded grid over 40-120, one shared-A "
                                   f"batch, {iters} iterations per step",
                       "l2": "512 MiB L2 flush before each step; the batch's vectors (~2 GB) exceed L2"},
            "ms_per_iteration": t_dev / iters * 1e3,
            "iterations_per_step": iters,
            "status": {"optimal": int(sum(r.status == "Optimal" for r in rs)),
                       "max_relative_kkt": float(max(r.relativeKkt for r in rs))},
            "kernels": prof,
            "kernels_fp32": prof32,
            "reference_model_gbs": ref_model / (t_dev / iters) / 1e9,
            "tuned": {"streamed_vectors_primal": bool(st.streaming_at), "streamed_vectors_dual": bool(st.streaming_a),
                      "cases_per_thread_primal": int(st.cases_per_thread_at),
                      "cases_per_thread_dual": int(st.cases_per_thread_a),
                      "warp_rows_primal": bool(st.warp_rows_at), "warp_rows_dual": bool(st.warp_rows_a),
                      "tile_rows_primal": int(st.tile_rows_at), "tile_rows_dual": int(st.tile_rows_a)},
            "e2e": {"value": t_e2e, "unit": "s per batch call (host arrays)", "h2d_bytes_per_step": h2d,
                    "d2h_bytes_per_step": d2h},
            "single_case_ms_per_iteration": t_single * 1e3,
            "speedup_vs_cases_one_at_a_time": t_single * K / (t_dev / iters),
            "roofline": {"bound": "hbm", "kernel": dominant, "achieved": achieved, "peak": peak, "unit": "GB/s",
                         "frac": achieved / peak, "peak_kind": peak_kind, "traffic": None},
            "gpu_launches": int(st.kernel_launches),
            "clocks": clk.summary()}
    print(json.dumps(line))
    return 0


def sweep_family(K: int, size: str = "large"):
    """The crude-price sweep of a refinery family (by default the large one:
    5,064 x 11,376, 57,178 nonzeros, unit row and column scales): K cases whose
    6 crude prices are permutations of a seeded grid over 40-120 $/bbl,
    demands at their mid scale.  Returns (family, K x 16 parameters)."""
    import numpy as np

    from pramana_b200 import warmstart as W
    fam = W.RefineryFamily(seed=5, **FAMILY_SIZES[size])
    rng = np.random.default_rng(9)
    levels = np.linspace(40.0, 120.0, K)
    prices = np.stack([rng.permutation(levels) for _ in range(fam.crudes)], axis=1)
    return fam, np.hstack([prices, np.ones((K, fam.num_params - fam.crudes))])


SWEEP_TOL_METRIC = "time to certified rel KKT 1e-6 (s) of a 256-case crude-price sweep of the refinery LP"


def run_sweep_tol(args, rank, world):
    """--workload sweep-tol: the crude-price sweep of the refinery LP solved to
    rel KKT 1e-6, every case certified (KKT recomputed in FP64 and the
    reference's family rule on the outward-rounded bound over implied column
    bounds).  Forms: the shared-A batch engine (k-interleaved vectors, per-case
    restarts) and the multi-LP CTA form (one thread block per case, the one
    operator in L2), each in plain FP64 and in the mixed form (FP32 iterates,
    FP64 termination, re-measure and polish).  Baseline: plain FP64 single-LP
    solves of a sample of the cases, one at a time, scaled to all cases.
    Each form: one short untimed solve (module load), then --steps timed
    batches; value = the fastest form's mean wall time per batch plus its
    certification."""
    import numpy as np
    import torch

    from pramana_b200 import _lib, pdhg
    from pramana_b200 import warmstart as W

    if world > 1 and rank != 0:
        return 0
    torch.cuda.set_device(0)
    K = args.cases
    fam, params = sweep_family(K, args.family_size)
    base = fam.base
    cases = [fam.case(p) for p in params]
    lps = [fam.instance(p) for p in params]
    with open(os.path.join(ROOT, "tests", "golden", "answers.json")) as f:
        ans = json.load(f)["sweep"]
    sample = ans["sample"] if ans["cases"] == K and args.family_size == "large" else []
    exact = dict(zip(sample, ans["exact"]))
    forms = {}
    with ClockSampler(0) as clk:
        for name, prec, engine in (("batch_fp64", 0, "batch"), ("batch_mixed", 1, "batch"),
                                   ("cta_fp64", 0, "cta"), ("cta_mixed", 1, "cta")):
            if args.sweep_forms and name not in args.sweep_forms.split(","):
                continue
            kw = dict(tolerance=TOL, maxIterations=args.family_max_iters, precision=prec)
            if engine == "cta":
                kw["multiForm"] = _lib.MULTI_CTA
            opts = pdhg.PdhgOptions(**kw)
            short = pdhg.PdhgOptions(**{**kw, "maxIterations": 128})
            walls, loops = [], []
            for step in range(args.steps + 1):
                o = short if step == 0 else opts
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                if engine == "batch":
                    rs = pdhg.solvePdhgBatch(base, cases, o)
                else:
                    rs = pdhg.solvePdhgMulti(lps, o)
                wall = time.perf_counter() - t0
                if step > 0:
                    walls.append(wall)
                    loops.append(rs[0].stats.kernelSeconds)
            X = np.array([r.x for r in rs])
            Y = np.array([r.rowDual for r in rs])
            t1 = time.perf_counter()
            cert = W.certify_family(fam, params, X, Y, kkt_tol=TOL)
            cert_s = time.perf_counter() - t1
            obj = np.array([r.objective for r in rs])
            err = [abs(obj[i] - e) / (1 + abs(e)) for i, e in exact.items()]
            its = np.array([r.iterations for r in rs])
            forms[name] = {"seconds_per_batch": statistics.mean(walls), "loop_seconds": statistics.mean(loops),
                           "certify_seconds": cert_s, "optimal": int(sum(r.status == "Optimal" for r in rs)),
                           "certified": int(cert["certified"].sum()),
                           "certification_failures": int((~cert["certified"]).sum()),
                           "max_relative_kkt_fp64": float(cert["kkt"][:, 3].max()),
                           "iterations_mean": float(its.mean()), "iterations_max": int(its.max()),
                           "fp32_iterations": int(rs[0].stats.fp32Iterations),
                           "max_objective_rel_err_vs_exact_sample": float(max(err)) if err else None}
    # baseline: plain FP64 single-LP solves, one case at a time
    plain = pdhg.PdhgOptions(tolerance=TOL, maxIterations=args.family_max_iters, precision=0)
    pick = [int(i) for i in np.linspace(0, K - 1, args.per_instance_sample).round()]
    per, its1 = [], []
    pdhg.solvePdhg(lps[0], pdhg.PdhgOptions(tolerance=TOL, maxIterations=128))
    for i in pick:
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        r = pdhg.solvePdhg(lps[i], plain)
        per.append(time.perf_counter() - t0)
        its1.append(r.iterations)
    seq = statistics.mean(per) * K
    best = min(forms, key=lambda k: forms[k]["seconds_per_batch"] + forms[k]["certify_seconds"])
    value = forms[best]["seconds_per_batch"] + forms[best]["certify_seconds"]
    line = {"metric": SWEEP_TOL_METRIC, "value": value, "unit": "s", "n_gpus": 1, "steps": args.steps,
            "warmup": 1, "ms_per_step": value * 1e3, "higher_is_better": False, "scaling": "weak",
            "vs_baseline": None, "dtype": f"{best}: " + ("f32 iterates, f64 checks and polish" if "mixed" in best
                                                        else "f64"),
            "data": "synthetic (seeded)", "workload": "sweep-tol",
            "config": {"workload": f"refinery LP ({args.family_size}) {base.num_rows} rows x {base.num_cols} cols, "
                                   f"{base.nnz} nnz ({FAMILY_SIZES[args.family_size]}), {K} cases "
                                   f"with the 6 crude prices on a seeded grid over 40-120, to rel KKT {TOL:g}, "
                                   "every case certified",
                       "step": "one batch call from host arrays plus certify_family on its answers"},
            "chosen_form": best, "forms": forms,
            "sequential_fp64": {"cases_timed": len(pick), "seconds_per_case": statistics.mean(per),
                                "iterations_mean": float(np.mean(its1)), "seconds_all_cases_scaled": seq},
            "speedup_vs_sequential_fp64": seq / value,
            "exact_sample": {"cases": sample, "source": "the reference's dual simplex (tests/golden/answers.json)"},
            "clocks": clk.summary()}
    print(json.dumps(line))
    return 0


MULTI_METRIC = "time-to-1e-6 rel KKT (s) of a batch of uneven LPs in one multi-LP run & its HBM GB/s"


def run_multi(args, rank, world):
    """--workload multi: independent LPs of uneven size (config-2 generator,
    nnz log-uniform) in one multi-LP run per GPU; under torchrun the LPs are
    sharded across the GPUs, balanced by nonzeros, with no communication until
    the results are gathered.  With --profile-iters, a fixed iteration count for
    the per-iteration bandwidth only."""
    import torch

    from pramana_b200 import _lib
    from pramana_b200 import generators as G
    from pramana_b200 import pdhg
    from pramana_b200.shard import gather, max_over_ranks, partition

    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local_rank if world > 1 else 0)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))
    dev_id = torch.cuda.current_device()
    sizes = G.uneven_family_sizes(args.instances, 1e4, args.nnz_hi, seed=4)
    mine = partition(sizes, world)[rank] if world > 1 else list(range(args.instances))
    lps = G.uneven_family(args.instances, 1e4, args.nnz_hi, seed=4, only=mine)
    fixed = args.profile_iters > 0
    po = pdhg.PdhgOptions(tolerance=1e-30 if fixed else TOL, maxIterations=args.profile_iters if fixed else 1000000,
                          spmvSchedule=["auto", "binned", "tiled", "tuned"].index(args.schedule), device=dev_id)
    flush = torch.empty(512 * 1024 * 1024, dtype=torch.uint8, device=f"cuda:{dev_id}")

    def barrier():
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()

    runs = []
    for s in range(args.warmup + args.steps):
        flush.zero_()
        barrier()
        st = pdhg.PdhgStats()
        t0 = time.perf_counter()
        rs = pdhg.solvePdhgMulti(lps, po, batchStats=st) if lps else []
        wall = time.perf_counter() - t0
        barrier()
        if s >= args.warmup:
            raw = pdhg.solvePdhgMulti.last_stats if lps else _lib.B2pStats()
            runs.append((st.kernelSeconds if lps else 0.0, wall, st.iterations, rs, raw.kernel_launches,
                         raw.bytes_uploaded, raw.bytes_downloaded, raw.lanes_per_row_a, raw.lanes_per_row_at,
                         raw.schedule_a, raw.schedule_at,
                         {"setup_s": raw.setup_seconds, "host_preparation_s": raw.prepare_seconds,
                          "uploads_schedules_autotune_s": raw.upload_seconds, "autotune_s": raw.autotune_seconds,
                          "graphs_s": raw.graph_seconds, "loop_s": raw.solve_seconds}))
    dev = statistics.mean(r[0] for r in runs)
    wall = statistics.mean(r[1] for r in runs)
    rs = runs[-1][3]

    # work actually done: each LP's bytes per iteration times its own iteration count
    # (terminated LPs drop out of the schedule)
    def lp_bytes(lp, fused_model):
        base = 24 * lp.nnz + 4 * (lp.num_rows + lp.num_cols + 2) + 16 * (lp.num_rows + lp.num_cols)
        if fused_model:
            base += -8 * (lp.num_rows + lp.num_cols) + 56 * lp.num_cols + 80 * lp.num_rows
        return base

    local = {i: {"status": r.status, "iterations": r.iterations, "alg": lp_bytes(lp, False) * r.iterations,
                 "fused": lp_bytes(lp, True) * r.iterations, "nnz": lp.nnz, "m": lp.num_rows, "n": lp.num_cols}
             for i, lp, r in zip(mine, lps, rs)}
    if dist is not None:
        dev, wall = max_over_ranks([dev, wall], device=f"cuda:{dev_id}")
        merged = gather(local)
    else:
        merged = local
    seq = None
    if rank == 0 and world == 1 and not fixed and args.per_instance_sample > 0:
        # sequential plain FP64 single-LP solves of a sample, extrapolated by nonzeros
        import numpy as np
        pick = np.random.default_rng(0).choice(len(lps), size=min(args.per_instance_sample, len(lps)), replace=False)
        t_s, nnz_s = 0.0, 0
        for i in pick:
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            pdhg.solvePdhg(lps[i], pdhg.PdhgOptions(tolerance=TOL, precision=0))
            t_s += time.perf_counter() - t0
            nnz_s += lps[i].nnz
        total_nnz = sum(v["nnz"] for v in merged.values())
        seq = {"members_timed": len(pick), "seconds_timed": t_s,
               "seconds_extrapolated": t_s * total_nnz / max(1, nnz_s),
               "extrapolation": "wall time of one-at-a-time solves x (batch nnz / sample nnz)"}
    if rank == 0:
        peak, peak_kind = measured_peak()
        nnz = sum(v["nnz"] for v in merged.values())
        m = sum(v["m"] for v in merged.values())
        n = sum(v["n"] for v in merged.values())
        done_alg = sum(v["alg"] for v in merged.values())
        done_fused = sum(v["fused"] for v in merged.values())
        its = max(v["iterations"] for v in merged.values())
        line = {"metric": MULTI_METRIC, "value": dev, "unit": "s", "n_gpus": world, "steps": args.steps,
                "warmup": args.warmup, "ms_per_step": dev * 1e3, "higher_is_better": False,
                "scaling": "strong" if world > 1 else "weak", "vs_baseline": None, "dtype": "f64",
                "data": "synthetic (seeded generator)", "workload": "multi",
                "config": {"workload": f"{args.instances} config-2-generator LPs, nnz log-uniform [1e4, {args.nnz_hi:g}], "
                                       f"seeds 4..{3 + args.instances}: {m} rows, {n} cols, {nnz} nnz in total",
                           "to": "fixed iterations" if fixed else f"rel KKT {TOL:g} per LP",
                           "parallelism": f"LPs sharded over {world} GPUs by nonzeros" if world > 1 else "single GPU",
                           "lanes_per_row": [runs[-1][7], runs[-1][8]], "schedule_requested": args.schedule,
                           "schedule_used": [runs[-1][9], runs[-1][10]],
                           "l2": "flushed before each step; the operators (24 B/nnz per iteration) exceed L2"},
                "iterations": its, "optimal": sum(v["status"] == "Optimal" for v in merged.values()),
                "e2e": {"value": wall, "unit": "s", "h2d_bytes_per_step": int(runs[-1][5]),
                        "d2h_bytes_per_step": int(runs[-1][6])},
                "setup": runs[-1][11],
                "gpu_launches": runs[-1][4],
                "sequential_fp64": seq,
                "speedup_vs_sequential": (seq["seconds_extrapolated"] / wall) if seq else None,
                "roofline": {"bound": "hbm", "kernel": "fused primal + dual kernels (+ checks every 64)",
                             "achieved": done_alg / dev / 1e9, "peak": peak * world, "unit": "GB/s",
                             "frac": done_alg / dev / 1e9 / (peak * world), "peak_source": peak_kind,
                             "algorithmic_bytes": done_alg, "fused_model_bytes": done_fused,
                             "fused_model_frac": done_fused / dev / 1e9 / (peak * world),
                             "unit_of_work": "the whole loop: every LP's SpMV bytes x its own iterations / device "
                                             "time (max over GPUs); peak = per-GPU peak x GPUs"}}
        print(json.dumps(line))
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()
    return 0


GEMM_SHAPES = ((1024, 512, 512), (1024, 128, 512), (512, 512, 1024), (1024, 512, 16), (4096, 512, 512),
               (8192, 8192, 8192))


def measured_bf16_peak():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(p) as f:
            d = json.load(f)
        return float(d["bf16_tflops"]), "measured"
    except (OSError, KeyError, ValueError):
        return 1590.0, "fallback"


def gemm_ctas(m, n, sms):
    """CTAs of k_gemm_group: the widest of its tiles that still give every SM one."""
    counts = [-(-m // 128) * -(-n // bn) for bn in (256, 128, 64)]
    return next((c for c in counts[:2] if c >= sms), counts[2])


def run_gemm(args, rank, world):
    """--workload gemm: the warm-start network's tcgen05 BF16 GEMM (its TMA form,
    k_gemm_group: both operands here are K-contiguous) timed with CUDA events
    (b2p_mlp_gemm_bf16_time) at the network's shapes -- batch 1,024 through
    512-wide hidden layers, the output layer, a weight gradient (K = batch),
    the input layer -- and two larger ones, as TFLOP/s of 2 M N K against the
    bf16 tensor peak."""
    import ctypes as C

    import torch

    from pramana_b200 import _lib
    if world > 1 and rank != 0:
        return 0
    torch.cuda.set_device(0)
    lib = _lib.load()
    peak, kind = measured_bf16_peak()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(0)
    rows = []
    for m, n, k in GEMM_SHAPES:
        a = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
        bt = torch.randn(n, k, device="cuda", generator=g).to(torch.bfloat16)  # B(k, n) = bt[n, k]
        c = torch.empty(m, n, device="cuda", dtype=torch.float32)
        ms = C.c_double(0)
        reps = max(3, min(200, int(2e11 // (2 * m * n * k))))
        _lib.check(lib.b2p_mlp_gemm_bf16_time(m, n, k, a.data_ptr(), k, 1, bt.data_ptr(), 1, k, c.data_ptr(), n,
                                              reps, C.byref(ms)))
        ref = a.float() @ bt.float().t()
        err = float((c - ref).abs().max() / ref.abs().max())
        tflops = 2.0 * m * n * k / (ms.value * 1e-3) / 1e12
        rows.append({"M": m, "N": n, "K": k, "us_per_launch": ms.value * 1e3, "tflops": tflops,
                     "frac_of_peak": tflops / peak, "ctas": gemm_ctas(m, n, sms), "reps": reps,
                     "max_rel_err_vs_fp32_matmul": err})
    line = {"metric": "tcgen05 BF16 GEMM TFLOP/s at the warm-start network's shapes", "workload": "gemm",
            "unit": "TFLOP/s", "value": max(r["tflops"] for r in rows), "higher_is_better": True,
            "peak": peak, "peak_source": kind, "kernel": "k_gemm_group (TMA copies into 128B-swizzled stages, producer and MMA warps; the widest of 128x256, 128x128 and 128x64 tiles that fill every SM)",
            "shapes": rows}
    print(json.dumps(line))
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--reference-backend", choices=["cpu", "gpu"], default="cpu",
                    help="reference arm: its CPU PDHG (the contract's arm) or its own GPU backend on this GPU")
    ap.add_argument("--cpu-sample-iters", type=int, default=CPU_SAMPLE_ITERS)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--workload", choices=["lp", "family", "multi", "sweep", "router", "plan", "families",
                                           "calibrate", "gemm", "sweep-tol", "c3"], default="lp")
    ap.add_argument("--plan", default="plan_60x156", help="plan: which refinery plan of the published runs")
    ap.add_argument("--plan-tol", type=float, default=1e-4, help="plan: relative KKT tolerance (1e-4 or 1e-6)")
    ap.add_argument("--c3-max-iters", type=int, default=3000000, help="c3: iteration limit per solve")
    ap.add_argument("--router-limit", type=float, default=3.0, help="router: time limit per engine and LP (s)")
    ap.add_argument("--router-out", default="router_calibration",
                    help="router: folder for the fitted model and the per-LP timings")
    ap.add_argument("--cases", type=int, default=256, help="sweep: cases in the shared-A batch")
    ap.add_argument("--sweep-iters", type=int, default=640, help="sweep: PDHG iterations per step")
    ap.add_argument("--instances", type=int, default=256, help="multi: LPs in the batch")
    ap.add_argument("--nnz-hi", type=float, default=5e5, help="multi: largest nonzero count (log-uniform from 1e4)")
    ap.add_argument("--schedule", choices=["auto", "binned", "tiled", "tuned"], default="auto",
                    help="multi: SpMV schedule of the multi-LP kernels")
    ap.add_argument("--train", type=int, default=32768, help="family: training members")
    ap.add_argument("--family-size", choices=sorted(FAMILY_SIZES), default=None,
                    help="family / sweep-tol: refinery LP size (small 164 x 324, medium 1,692 x 3,528, large "
                         "5,064 x 11,376; default medium for family, large for sweep-tol)")
    ap.add_argument("--precision", choices=["fp64", "mixed"], default="mixed",
                    help="family: arithmetic of the batched solves (the per-instance baseline is plain FP64)")
    ap.add_argument("--family-max-iters", type=int, default=None,
                    help="family / sweep-tol: iteration limit per member (default 400,000 for family; the "
                         "reference's 1,000,000 for sweep-tol)")
    ap.add_argument("--warm-max-iters", type=int, default=None,
                    help="family: iteration limit of the warm attempts (default: --family-max-iters); a member "
                         "past it falls back to a cold solve")
    ap.add_argument("--cold-fallback-only", dest="continue_failed", action="store_false",
                    help="family: a warm-started member that fails re-solves cold at once (default: it continues "
                         "from its final point and primal weight first, then cold)")
    ap.add_argument("--family-weights", choices=["default", "nearest"], default="default",
                    help="family (engine multi): starting primal weight of the warm strategies -- the default "
                         "||c|| / ||b||, or the geometric mean of the 4 nearest training members' final weights")
    ap.add_argument("--sweep-forms", default="", help="sweep-tol: comma-separated subset of the forms to run")
    ap.add_argument("--batch", type=int, default=1024, help="family: members per batched solve")
    ap.add_argument("--engine", choices=["multi", "batch"], default="multi",
                    help="family: multi-LP engine (one block per member) or the shared-A batch engine")
    ap.add_argument("--epochs", type=int, default=200, help="family: MLP training epochs")
    ap.add_argument("--per-instance-sample", type=int, default=16,
                    help="family: members solved one at a time for the per-instance FP64 baseline")
    ap.add_argument("--profile-iters", type=int, default=0,
                    help="small case for ncu: stop every solve after this many iterations, skip e2e and the CPU "
                         "baseline; the printed line is not a benchmark result")
    args = ap.parse_args()
    if args.family_size is None:
        args.family_size = "large" if args.workload == "sweep-tol" else "medium"
    if args.family_max_iters is None:
        args.family_max_iters = 1000000 if args.workload == "sweep-tol" else 400000
    if args.warmup < 3:
        ap.error("--warmup must be >= 3")
    if args.steps < 1:
        ap.error("--steps must be >= 1")

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        return run_reference(args, rank, world)
    if args.workload == "family":
        return run_family(args, rank, world)
    if args.workload == "multi":
        return run_multi(args, rank, world)
    if args.workload == "sweep":
        return run_sweep(args, rank, world)
    if args.workload == "router":
        return run_router(args, rank, world)
    if args.workload == "plan":
        return run_plan(args, rank, world)
    if args.workload == "families":
        return run_families(args, rank, world)
    if args.workload == "calibrate":
        return run_calibrate(args, rank, world)
    if args.workload == "gemm":
        return run_gemm(args, rank, world)
    if args.workload == "c3":
        return run_c3(args, rank, world)
    if args.workload == "sweep-tol":
        return run_sweep_tol(args, rank, world)

    import torch
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        torch.cuda.set_device(local_rank)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    else:
        torch.cuda.set_device(0)
    dev = torch.cuda.current_device()

    from pramana_b200 import generators as G
    from pramana_b200 import pdhg

    lp = G.config2(SEED)
    po_plain = pdhg.PdhgOptions(tolerance=TOL, device=dev, precision=0)
    po = pdhg.PdhgOptions(tolerance=TOL, device=dev, precision=1)  # the chosen form: mixed precision
    if args.profile_iters > 0:
        po.maxIterations = po_plain.maxIterations = args.profile_iters
    flush = torch.empty(512 * 1024 * 1024, dtype=torch.uint8, device=f"cuda:{dev}")

    def barrier():
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()

    def timed_solves(eng, steps, sampler=None):
        """K solves from the cold start; device time of each loop (CUDA events on the engine's stream)."""
        out = []
        for _ in range(steps):
            flush.zero_()
            torch.cuda.synchronize()
            r = eng.solve()[0]
            st = eng.last_stats
            assert r.status == "Optimal" or args.profile_iters > 0, r.status
            out.append((st.kernel_seconds, st.kernel_launches, r, st.fp32_iterations))
        return out

    # ---- value: device-timed loop of the chosen (mixed) form, problem resident in HBM ----
    eng = pdhg.Engine(lp, po)
    timed_solves(eng, args.warmup)
    barrier()
    with ClockSampler(dev) as clk:
        res = timed_solves(eng, args.steps)
        barrier()
    t_dev = statistics.mean(x[0] for x in res)
    launches = sum(x[1] for x in res)
    r_mixed, fp32_iters = res[-1][2], res[-1][3]
    iters = r_mixed.iterations
    eng.close()

    # ---- the plain FP64 form on the same LP, for the comparison the metric asks for ----
    eng = pdhg.Engine(lp, po_plain)
    timed_solves(eng, args.warmup)
    barrier()
    res_plain = timed_solves(eng, args.steps)
    barrier()
    t_plain = statistics.mean(x[0] for x in res_plain)
    r_plain = res_plain[-1][2]

    # ---- roofline of the dominant kernel: a profiled plain solve (events around every launch) ----
    eng.set_profiling(True)
    flush.zero_()
    torch.cuda.synchronize()
    eng.solve()
    eng.set_profiling(False)
    prof = []
    for cls, name in ((0, "k_primal_binned"), (1, "k_dual_binned"), (2, "k_resident")):
        n_l, ms = eng.kernel_times(cls)
        if n_l > 0:
            prof.append((ms, n_l, name, eng.kernel_bytes(cls)))
    prof.sort(reverse=True)
    ms, n_l, kname, kbytes = prof[0]
    # per launch for the per-iteration kernels; per iteration for the resident interval kernel
    avg_s = ms / 1e3 / max(1, n_l)
    achieved = kbytes / avg_s / 1e9
    peak, peak_kind = measured_peak()
    spmv_total_bytes = sum(p[3] * p[1] for p in prof)
    spmv_total_s = sum(p[0] for p in prof) / 1e3
    form = {1: "fused", 2: "resident"}.get(eng.last_stats.kernel_mode, "?")
    eng.close()

    if args.profile_iters > 0:
        print(json.dumps({"profile_run": True, "iterations": iters, "device_s_per_solve": t_dev,
                          "dominant_kernel": kname, "avg_launch_us": avg_s * 1e6}))
        return 0

    # ---- e2e: public C ABI from host arrays, chosen form ----
    e2e_times, h2d, d2h = [], 0, 0
    for s in range(args.warmup + args.steps):
        flush.zero_()
        barrier()
        t0 = time.perf_counter()
        r = pdhg.solvePdhg(lp, po)
        t1 = time.perf_counter()
        if s >= args.warmup:
            e2e_times.append(t1 - t0)
            h2d, d2h = r.stats.bytesUploaded, r.stats.bytesDownloaded
    t_e2e = statistics.mean(e2e_times)

    # ---- e2e of the plain FP64 form through the same call ----
    e2e_plain = []
    for s in range(args.warmup + args.steps):
        flush.zero_()
        barrier()
        t0 = time.perf_counter()
        r = pdhg.solvePdhg(lp, po_plain)
        t1 = time.perf_counter()
        if s >= args.warmup:
            e2e_plain.append(t1 - t0)
    t_e2e_plain = statistics.mean(e2e_plain)

    if dist is not None:
        tt = torch.tensor([t_dev, t_e2e, t_plain, t_e2e_plain], dtype=torch.float64, device=f"cuda:{dev}")
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        t_dev, t_e2e, t_plain, t_e2e_plain = tt.tolist()

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        from oracle import oracle as O
        if O.available("ref"):
            threads = os.cpu_count() or 1
            loop, wall, rr, _ = cpu_reference_solve(lp, threads)
            cpu = {"value": loop, "unit": "s", "cores": threads, "kind": "reference",
                   "sample": f"one full solve of the same LP to rel KKT {TOL:g} ({rr.iterations} iterations, "
                             f"{wall:.1f} s wall), loop time"}

    if rank == 0:
        line = {"metric": METRIC, "value": t_dev, "unit": "s", "n_gpus": world, "steps": args.steps,
                "warmup": args.warmup, "ms_per_step": t_dev * 1e3, "higher_is_better": False, "scaling": "weak",
                "vs_baseline": None, "dtype": "f32 iterates, f64 checks and polish",
                "data": "synthetic (seeded generator)",
                "config": workload_config(lp, world),
                "run": {"iterations": iters, "fp32_iterations": fp32_iters, "kernel_form": form,
                        "chosen_form": "mixed precision"},
                "forms": {
                    "mixed": {"value": t_dev, "iterations": iters, "fp32_iterations": fp32_iters,
                              "relative_kkt_fp64": r_mixed.relativeKkt,
                              "objective_rel_diff_vs_fp64": abs(r_mixed.objective - r_plain.objective)
                              / (1 + abs(r_plain.objective)),
                              **answer_errors(r_mixed.objective)},
                    "plain_fp64": {"value": t_plain, "iterations": r_plain.iterations,
                                   "relative_kkt": r_plain.relativeKkt,
                                   "e2e": {"value": t_e2e_plain, "unit": "s", "h2d_bytes_per_step": h2d,
                                           "d2h_bytes_per_step": d2h}}},
                "e2e": {"value": t_e2e, "unit": "s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h},
                "gpu_launches": launches,
                "spmv_gbs": spmv_total_bytes / spmv_total_s / 1e9,
                "roofline": {"bound": "hbm", "kernel": kname, "achieved": achieved, "peak": peak, "unit": "GB/s",
                             "frac": achieved / peak, "peak_source": peak_kind,
                             "traffic": ncu_traffic(kname), "algorithmic_bytes_per_launch": kbytes,
                             "avg_launch_us": avg_s * 1e6, "launches_profiled": n_l,
                             "unit_of_work": "one PDHG iteration" if kname == "k_resident" else "one launch"},
                "clocks": clk.summary(),
                "cpu_baseline": cpu}
        print(json.dumps(line))
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
