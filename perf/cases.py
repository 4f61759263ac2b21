"""Performance cases: what a user of the engine has it do, through its public entry points.

The cases cover the PDHG engine (one LP, a family of cases over one A, many LPs in one call), the certification
that follows a batch, and the warm-start network (its training, its prediction, its GEMM).  Every PDHG case runs a
fixed number of iterations, the way the repository's own sweep and calibration workloads do: the tolerance is out
of reach, so a pass is the same amount of work whatever the inputs are.  All data is synthetic, made from the seed.
"""
import dataclasses
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "optimized-gpu-accelerator_b200"))

from pramana_b200 import _lib, generators, pdhg, warmstart  # noqa: E402
from pramana_b200.mlp import MlpNetwork, TrainOptions, gemm_bf16, he_uniform  # noqa: E402
from pramana_b200.model import Model  # noqa: E402

# Plain FP64 and the mixed form (FP32 iterates, FP64 checks).
PRECISIONS = {"fp64": _lib.PRECISION_FP64, "mixed": _lib.PRECISION_MIXED}

# The three sizes of the refinery-planning family: 164 x 324, 1,692 x 3,528 and 5,064 x 11,376.
REFINERIES = {
    "small": dict(periods=2, regions=1, units=4, streams=4, properties=2, scale_exponent=0.0),
    "medium": dict(periods=6, regions=2, units=6, streams=6, properties=3, pools=12, scale_exponent=0.0),
    "large": dict(periods=12, regions=2, units=8, streams=8, properties=4, pools=12, scale_exponent=0.0),
}
SIZES = {"small": (164, 324, 1072), "medium": (1692, 3528, 14982), "large": (5064, 11376, 57178)}  # rows, columns, nonzeros

CERTIFICATE = ("accepted", "used_implied_bounds", "primal_objective", "safe_dual_bound", "max_primal_violation",
               "max_dual_violation")

WIDTHS = (16, 512, 512, 512, 128)  # the warm-start network of the refinery family


def listed():
    return [
        # The smallest LP of the repository's benchmarks, one call from host arrays: set-up and launches count.
        {"name": "lp_small_call", "kind": "lp", "matrix": "random", "rows": 1000, "precision": "fp64",
         "entry": "call", "iterations": 1280},
        # The benchmark LP (40,000 x 80,000, 1% of the rows hold 10% of the nonzeros) prepared once and solved again.
        {"name": "lp_skew_prepared", "kind": "lp", "matrix": "skew", "rows": 40000, "precision": "fp64",
         "entry": "prepared", "iterations": 2560},
        # The same LP in the mixed form, from host arrays to host arrays: the benchmark's end-to-end call.
        {"name": "lp_skew_mixed_call", "kind": "lp", "matrix": "skew", "rows": 40000, "precision": "mixed",
         "entry": "call", "iterations": 2560},
        # A large transportation-like LP of the per-iteration calibration, whose operators exceed shared memory.
        {"name": "lp_transport_prepared", "kind": "lp", "matrix": "transport", "rows": 256000, "precision": "fp64",
         "entry": "prepared", "iterations": 512},
        # The crude-price sweep of the large refinery: 256 cases over one A, prepared once.
        {"name": "sweep_256", "kind": "batch", "refinery": "large", "cases": 256, "precision": "fp64",
         "entry": "prepared", "iterations": 640},
        # A published-size family study with an odd number of cases: solve from host arrays, then certify the answers.
        {"name": "plan_batch_certified", "kind": "batch", "refinery": "medium", "cases": 61, "precision": "fp64",
         "entry": "call", "iterations": 640},
        # A held-out batch of the small family: 1,024 little LPs in one call, one thread block each.
        {"name": "family_small_1024", "kind": "family", "refinery": "small", "members": 1024, "precision": "fp64",
         "iterations": 5120},
        # Members of the medium family, whose operators exceed a block's shared memory.
        {"name": "family_medium_296", "kind": "family", "refinery": "medium", "members": 296, "precision": "fp64",
         "iterations": 5120},
        # LPs of uneven size in one call, nonzeros spread log-uniformly, as the uneven batch workload has them.
        {"name": "uneven_multi", "kind": "uneven", "lps": 24, "nnz_lo": 10000, "nnz_hi": 200000, "precision": "fp64",
         "iterations": 2560},
        # Training the warm-start network from its initial weights: forward, backward and Adam.
        {"name": "network_train", "kind": "train", "samples": 8192, "batch": 512, "epochs": 4},
        # Predicting starting points for a handful of members: the smallest call.
        {"name": "network_predict", "kind": "predict", "rows": 100},
        # The tensor-core GEMM at the benchmark's largest shape.
        {"name": "gemm_8192", "kind": "gemm", "m": 8192, "n": 8192, "k": 8192, "b_layout": "nk"},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lp", "lp", "lp", "batch", "batch", "family", "family", "uneven", "train", "predict", "gemm"])
    precision = rng.choice(["fp64", "fp64", "mixed"])
    if kind == "lp":
        matrix = rng.choice(["random", "skew", "transport"])
        return {"kind": kind, "matrix": matrix, "precision": precision,
                "rows": _spread(rng, 300, 200000 if matrix == "transport" else 40000),
                "entry": rng.choice(["call", "prepared"]), "iterations": _spread(rng, 300, 1000)}
    if kind == "batch":
        refinery = rng.choice(["small", "medium", "large"])
        return {"kind": kind, "refinery": refinery, "precision": precision,
                "cases": _spread(rng, 2, {"small": 200, "medium": 200, "large": 250}[refinery]),
                "entry": rng.choice(["call", "prepared"]), "iterations": _spread(rng, 200, 640)}
    if kind == "family":
        refinery = rng.choice(["small", "medium"])
        return {"kind": kind, "refinery": refinery, "precision": precision,
                "members": _spread(rng, 2, {"small": 1000, "medium": 290}[refinery]),
                "iterations": _spread(rng, 500, 1280 if precision == "mixed" else 5000)}
    if kind == "uneven":
        return {"kind": kind, "lps": rng.randint(3, 23), "nnz_lo": 10000, "nnz_hi": 200000, "precision": precision,
                "iterations": _spread(rng, 300, 2500)}
    if kind == "train":
        batch = _spread(rng, 100, 512)
        return {"kind": kind, "samples": batch * rng.randint(2, 12) + rng.randint(0, 99), "batch": batch,
                "epochs": rng.randint(1, 3)}
    if kind == "predict":
        return {"kind": kind, "rows": _spread(rng, 1, 2000)}
    step = rng.choice([1, 8])  # row strides that are multiples of 16 bytes, and any
    return {"kind": kind, "m": _spread(rng, 100, 6000), "n": step * _spread(rng, 72 // step, 5600 // step),
            "k": step * _spread(rng, 72 // step, 5600 // step), "b_layout": rng.choice(["nk", "kn"])}


# ---- inputs ----------------------------------------------------------------------------------------------------


def _transport_lp(m, seed):
    """min c'x, A x >= 1, 0 <= x <= 10 with four entries 0.5 + U(0, 1) a column at random rows, c = U(0, 1) - 0.3."""
    rng = np.random.default_rng(seed)
    n = 2 * m
    rows = np.sort(rng.integers(0, m, size=(n, 4)), axis=1)
    keep = np.ones((n, 4), dtype=bool)
    keep[:, 1:] = rows[:, 1:] != rows[:, :-1]  # an entry that repeats a row of its column is dropped
    start = np.concatenate([[0], np.cumsum(keep.sum(axis=1))])
    value = 0.5 + rng.random((n, 4))
    return Model(num_rows=m, num_cols=n, start=start, index=rows[keep], value=value[keep],
                 col_cost=rng.random(n) - 0.3, col_lower=np.zeros(n), col_upper=np.full(n, 10.0),
                 row_lower=np.ones(m), row_upper=np.full(m, np.inf))


_matrices = {}  # a prepared LP keeps its matrix from seed to seed: its costs and sides are new


def _lp(case, seed):
    """A new LP for a call from host arrays; for a prepared one, new costs and sides over one matrix."""
    m, prepared = case["rows"], case["entry"] == "prepared"
    at = (case["matrix"], m)
    if prepared and at in _matrices:
        lp = _matrices[at]
    elif case["matrix"] == "transport":
        lp = _transport_lp(m, 2 if prepared else seed)
    else:
        lp = generators.scaled_random_lp(m, 2 if prepared else seed, skew=case["matrix"] == "skew")
    if not prepared:
        return lp
    _matrices.clear()
    _matrices[at] = lp
    rng = np.random.default_rng(seed)
    if case["matrix"] == "transport":
        return dataclasses.replace(lp, col_cost=rng.random(2 * m) - 0.3)
    # sides and costs from a primal and a dual point, as the generator makes them
    cols = np.repeat(np.arange(lp.num_cols), np.diff(lp.start))
    side = np.bincount(lp.index, lp.value * rng.uniform(0.0, 10.0, size=lp.num_cols)[cols], minlength=m)
    equal = np.isfinite(lp.row_lower)
    cost = np.bincount(cols, lp.value * rng.standard_normal(m)[lp.index], minlength=lp.num_cols)
    return dataclasses.replace(lp, row_lower=np.where(equal, side, -np.inf),
                               row_upper=np.where(equal, side, side + rng.random(m)),
                               col_cost=cost + rng.random(lp.num_cols))


_families = {}  # a refinery's structure is the same for every seed: only prices and demands differ


def _family(name):
    if name not in _families:
        _families[name] = warmstart.RefineryFamily(seed=5, **REFINERIES[name])
    return _families[name]


def _uneven(case, seed):
    lo, hi, count = case["nnz_lo"], case["nnz_hi"], case["lps"]
    sizes = [lo * (hi / lo) ** ((i + 0.5) / count) / 12.8 for i in range(count)]
    return [generators.scaled_random_lp(int(round(m)), seed * 1000 + i, skew=True) for i, m in enumerate(sizes)]


def _options(case):
    return pdhg.PdhgOptions(tolerance=1e-9, maxIterations=case["iterations"], precision=PRECISIONS[case["precision"]])


def _network_data(rows, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1.0, 1.0, size=(rows, WIDTHS[0])).astype(np.float32)
    mix = rng.standard_normal((WIDTHS[0], WIDTHS[-1])).astype(np.float32)
    return x, np.tanh(0.3 * (x @ mix)).astype(np.float32)


def _gemm_data(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    m, n, k = case["m"], case["n"], case["k"]
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(*((n, k) if case["b_layout"] == "nk" else (k, n)), device="cuda", generator=g).to(torch.bfloat16)
    return a, b


def prepare(case, seed):
    kind, s = case["kind"], {"kind": case["kind"]}
    if kind == "lp":
        s["lp"], s["options"] = _lp(case, seed), _options(case)
        if case["entry"] == "prepared":
            s["engine"] = pdhg.Engine(s["lp"], s["options"])
    elif kind == "batch":
        fam = _family(case["refinery"])
        s["lp"], s["options"] = fam.base, _options(case)
        s["cases"] = [fam.case(p) for p in fam.sample(case["cases"], seed)]
        if case["entry"] == "prepared":
            s["engine"] = pdhg.Engine(s["lp"], s["options"], s["cases"])
    elif kind == "family":
        fam = _family(case["refinery"])
        s["lps"], s["options"] = [fam.instance(p) for p in fam.sample(case["members"], seed)], _options(case)
    elif kind == "uneven":
        s["lps"], s["options"] = _uneven(case, seed), _options(case)
    elif kind == "train":
        s["x"], s["target"] = _network_data(case["samples"], seed)
        s["net"] = MlpNetwork(WIDTHS, max_batch=max(512, case["batch"]), seed=None)
        s["weights"] = he_uniform(WIDTHS, seed)
        s["options"] = TrainOptions(epochs=case["epochs"], batch=case["batch"], seed=seed)
    elif kind == "predict":
        s["x"], _ = _network_data(case["rows"], seed)
        s["net"] = MlpNetwork(WIDTHS, max_batch=1024, seed=seed)
    else:
        s["a"], s["b"] = _gemm_data(case, seed)
        s["m"], s["n"], s["k"] = case["m"], case["n"], case["k"]
        s["b_strides"] = (1, case["k"]) if case["b_layout"] == "nk" else (case["n"], 1)
        s["c"] = torch.empty(case["m"], case["n"], device="cuda", dtype=torch.float32)
    return s


# ---- one pass --------------------------------------------------------------------------------------------------


def _answers(results):
    return {"x": np.concatenate([r.x for r in results]), "y": np.concatenate([r.rowDual for r in results]),
            "objective": np.array([r.objective for r in results]),
            "dual_objective": np.array([r.dualObjective for r in results]),
            "relative_kkt": np.array([r.relativeKkt for r in results]),
            "iterations": np.array([r.iterations for r in results]),
            "optimal": np.array([r.status == "Optimal" for r in results])}


def run(state):
    kind = state["kind"]
    if "engine" in state:
        return _answers(state["engine"].solve())
    if kind == "lp":
        return _answers([pdhg.solvePdhg(state["lp"], state["options"])])
    if kind == "batch":
        out = _answers(pdhg.solvePdhgBatch(state["lp"], state["cases"], state["options"]))
        verdicts = pdhg.certifyLp(state["lp"], out["x"], out["y"], state["cases"])
        out["certificates"] = {f: np.array([v[f] for v in verdicts]) for f in CERTIFICATE}
        return out
    if kind in ("family", "uneven"):
        return _answers(pdhg.solvePdhgMulti(state["lps"], state["options"]))
    if kind == "train":
        net = state["net"]
        net.set_params(state["weights"])
        losses = net.train(state["x"], state["target"], state["options"])
        return {"losses": losses, "weights": net.get_params()}
    if kind == "predict":
        return state["net"].forward(state["x"])
    gemm_bf16(state["a"], state["b"], out_f32=state["c"], b_strides=state["b_strides"], m=state["m"], n=state["n"],
              k=state["k"])
    return state["c"]


# ---- the work that a pass cannot do without --------------------------------------------------------------------


def _pdhg_work(m, n, nnz, cases, operators, iterations):
    """Bytes in and out once (the matrices, the costs, bounds and sides, the answers), operations of the iterations."""
    moved = operators * (12 * nnz + 4 * (n + 1)) + 8 * cases * (4 * n + 3 * m)
    return moved, iterations * cases * (4 * nnz + 10 * n + 17 * m)


def work(case):
    kind = case["kind"]
    if kind == "lp":
        m, per_column = case["rows"], {"random": 5.0, "skew": 6.4, "transport": 4.0}[case["matrix"]]
        moved, ops = _pdhg_work(m, 2 * m, 2 * m * per_column, 1, 1, case["iterations"])
    elif kind in ("batch", "family"):
        count = case["cases"] if kind == "batch" else case["members"]
        moved, ops = _pdhg_work(*SIZES[case["refinery"]], count, 1, case["iterations"])
    elif kind == "uneven":
        nnz = (case["nnz_hi"] - case["nnz_lo"]) / math.log(case["nnz_hi"] / case["nnz_lo"])
        moved, ops = _pdhg_work(nnz / 12.8, nnz / 6.4, nnz, case["lps"], case["lps"], case["iterations"])
    elif kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        moved, ops = 2 * (m * k + k * n) + 4 * m * n, 2 * m * n * k
    else:
        weights = sum(a * b for a, b in zip(WIDTHS[:-1], WIDTHS[1:]))
        if kind == "predict":
            moved, ops = 4 * case["rows"] * (WIDTHS[0] + WIDTHS[-1]) + 2 * weights, 2 * case["rows"] * weights
        else:
            steps = case["epochs"] * (case["samples"] // case["batch"])
            moved = 4 * case["samples"] * (WIDTHS[0] + WIDTHS[-1]) + 8 * weights
            ops = steps * (case["batch"] * (6 * weights - 2 * WIDTHS[0] * WIDTHS[1]) + 15 * weights)
    return {"bytes": float(moved), "flops": float(ops)}


# ---- the same results in 64 bits -------------------------------------------------------------------------------


def _power_of_two(v):
    return torch.pow(2.0, torch.round(torch.log2(v)))


def _finite(v):
    return v.abs() < 1e20


def _norm(v, ok=None):
    return (v if ok is None else torch.where(ok, v, torch.zeros_like(v))).square().sum(dim=0).sqrt()


def _rhs_norm(lo, up):
    other = _finite(up) & (up != lo)
    return (_norm(lo, _finite(lo)).square() + _norm(up, other).square()).sqrt()


def _pdhg64(lp, cost, lower, upper, row_lower, row_upper, own_scale, iterations, check_every=64):
    """Restarted reflected-Halpern PDHG of k cases over lp's matrix (cost, bounds: n x k and m x k): Ruiz and
    Pock-Chambolle scaling, objective and bounds rescaled (by each case's own norms, or by the first one's), step
    0.998 / ||A||, restart and primal weight tested every check_every iterations."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = lambda v: torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float64, device=dev)  # noqa: E731
    m, n = lp.num_rows, lp.num_cols
    rows = torch.as_tensor(lp.index, dtype=torch.int64, device=dev)
    cols = torch.repeat_interleave(torch.arange(n, device=dev), torch.as_tensor(np.diff(lp.start), device=dev))
    val = f64(lp.value)
    r, s = torch.ones(m, dtype=torch.float64, device=dev), torch.ones(n, dtype=torch.float64, device=dev)
    for step in range(11):
        a = val.abs() * s[cols] * r[rows]
        how = "amax" if step < 10 else "sum"
        ra = torch.zeros_like(r).scatter_reduce(0, rows, a, how)
        ca = torch.zeros_like(s).scatter_reduce(0, cols, a, how)
        r, s = torch.where(ra > 0, r / ra.sqrt(), r), torch.where(ca > 0, s / ca.sqrt(), s)
    r, s = _power_of_two(r), _power_of_two(s)
    val = val * r[rows] * s[cols]
    A = torch.sparse_coo_tensor(torch.stack([rows, cols]), val, (m, n)).coalesce().to_sparse_csr()
    AT = torch.sparse_coo_tensor(torch.stack([cols, rows]), val, (n, m)).coalesce().to_sparse_csr()
    r, s = r[:, None], s[:, None]
    cost, lower, upper, row_lower, row_upper = map(f64, (cost, lower, upper, row_lower, row_upper))
    cnorm, rnorm = _norm(cost), _rhs_norm(row_lower, row_upper)
    if own_scale:
        gamma, beta = 1 + _norm(cost * s), 1 + _rhs_norm(row_lower * r, row_upper * r)
    else:
        base = [f64(v)[:, None] for v in (lp.col_cost, lp.row_lower, lp.row_upper)]
        gamma, beta = 1 + _norm(base[0] * s), 1 + _rhs_norm(base[1] * r, base[2] * r)
    c = cost * s / gamma
    lo, up = torch.where(_finite(lower), lower / s / beta, lower), torch.where(_finite(upper), upper / s / beta, upper)
    rl = torch.where(_finite(row_lower), row_lower * r / beta, row_lower)
    ru = torch.where(_finite(row_upper), row_upper * r / beta, row_upper)
    cn, bn = _norm(c), _rhs_norm(rl, ru)
    omega = torch.where((cn > 1e-10) & (bn > 1e-10), cn / bn, torch.ones_like(cn))
    z = torch.full((n, 1), 1 / math.sqrt(n), dtype=torch.float64, device=dev)
    for _ in range(40):
        z = AT @ (A @ z)
        top = _norm(z)
        z = z / top
    eta = 0.998 / (1.01 * top.sqrt())
    tau, sigma = eta / omega, eta * omega
    x = torch.minimum(torch.maximum(torch.zeros_like(lo), lo), up)
    y, ax = torch.zeros_like(rl), A @ x
    x0, y0, ax0 = x, y, ax
    last, ref = torch.full_like(omega, math.inf), torch.full_like(omega, math.inf)
    since, age = torch.zeros_like(omega), torch.zeros_like(omega)
    move = lambda w, dx, dy: (w * dx + dy / w).sqrt()  # noqa: E731
    square = lambda v: v.square().sum(dim=0)  # noqa: E731
    for it in range(iterations):
        xp = torch.minimum(torch.maximum(x - tau * (c - AT @ y), lo), up)
        axp = A @ xp
        v = y - sigma * (2 * axp - ax)
        yp = v + sigma * torch.minimum(torch.maximum(-v / sigma, rl), ru)
        check = (it + 1) % check_every == 0
        if check:
            dx, dy = square(x - xp), square(y - yp)
            since = since + check_every
            fp = move(omega, dx, dy)
            ref = torch.where(torch.isinf(ref), fp, ref)
            again = (fp <= 0.2 * ref) | ((fp <= 0.8 * ref) & (fp > last)) | (since >= math.floor(0.36 * (it + 1)))
            last = fp
            gone_x, gone_y = square(xp - x0).sqrt(), square(yp - y0).sqrt()
            moved = again & (gone_x > 1e-10) & (gone_y > 1e-10)
            omega = torch.where(moved, (gone_y / gone_x * omega).sqrt(), omega)
            ref = torch.where(again, move(omega, dx, dy), ref)
            last = torch.where(again, torch.full_like(last, math.inf), last)
            since = torch.where(again, torch.zeros_like(since), since)
        lam = (age + 1) / (age + 2)
        halpern = lambda z, zp, z0: lam * (2 * zp - z) + (1 - lam) * z0  # noqa: E731, B023
        x, y, ax, age = halpern(x, xp, x0), halpern(y, yp, y0), halpern(ax, axp, ax0), age + 1
        if check:
            tau, sigma = eta / omega, eta * omega
            x, x0 = torch.where(again, xp, x), torch.where(again, xp, x0)
            y, y0 = torch.where(again, yp, y), torch.where(again, yp, y0)
            ax, ax0 = torch.where(again, axp, ax), torch.where(again, axp, ax0)
            age = torch.where(again, torch.zeros_like(age), age)
    # the answer and its relative KKT error, in the LP's own space
    x, y = xp * s * beta, yp * r * gamma
    act, d = axp * beta / r, cost - (AT @ yp) * gamma / s
    zero = torch.zeros_like
    has = [_finite(row_lower), _finite(row_upper), _finite(lower), _finite(upper)]
    off = torch.where(has[0], (row_lower - act).clamp(min=0), zero(act))
    off = off + torch.where(has[1], (act - row_upper).clamp(min=0), zero(act))
    wrong = torch.where(has[2], zero(d), d.clamp(min=0)) + torch.where(has[3], zero(d), (-d).clamp(min=0))
    primal = (cost * x).sum(dim=0)
    dual = torch.where((y > 0) & has[0], y * row_lower, zero(y)).sum(dim=0)
    dual = dual + torch.where((y < 0) & has[1], y * row_upper, zero(y)).sum(dim=0)
    dual = dual + torch.where((d > 0) & has[2], d * lower, zero(d)).sum(dim=0)
    dual = dual + torch.where((d < 0) & has[3], d * upper, zero(d)).sum(dim=0)
    gap = (primal - dual).abs() / (1 + primal.abs() + dual.abs())
    kkt = torch.maximum(torch.maximum(_norm(off) / (1 + rnorm), _norm(wrong) / (1 + cnorm)), gap)
    host = lambda v: v.cpu().numpy()  # noqa: E731
    return {"x": host(x.T.reshape(-1)), "y": host(y.T.reshape(-1)), "objective": host(primal) + lp.obj_offset,
            "dual_objective": host(dual) + lp.obj_offset, "relative_kkt": host(kkt)}


def _exact_members(models, iterations, own_scale):
    """Models over one matrix, together."""
    stack = [np.stack([getattr(p, f) for p in models], axis=1)
             for f in ("col_cost", "col_lower", "col_upper", "row_lower", "row_upper")]
    return _pdhg64(models[0], *stack, own_scale, iterations)


def exact(case, seed):
    kind = case["kind"]
    if kind == "gemm":
        a, b = _gemm_data(case, seed)
        return a.double() @ (b.double().T if case["b_layout"] == "nk" else b.double())
    if kind == "predict":
        h, _ = _network_data(case["rows"], seed)
        weights, at = he_uniform(WIDTHS, seed).astype(np.float64), 0
        h = h.astype(np.float64)
        for i, (a, b) in enumerate(zip(WIDTHS[:-1], WIDTHS[1:])):
            h = h @ weights[at:at + a * b].reshape(b, a).T + weights[at + a * b:at + a * b + b]
            at += a * b + b
            h = np.maximum(h, 0.0) if i + 2 < len(WIDTHS) else h
        return h
    if kind == "train":
        return None  # minibatches are drawn inside the call: no value outside it
    none = {"iterations": None, "optimal": None}
    if kind == "lp":
        return _exact_members([_lp(case, seed)], case["iterations"], True) | none
    if kind == "uneven":
        each = [_exact_members([lp], case["iterations"], True) for lp in _uneven(case, seed)]
        return {f: np.concatenate([e[f] for e in each]) for f in each[0]} | none
    fam = _family(case["refinery"])
    count = case["cases"] if kind == "batch" else case["members"]
    out = _exact_members([fam.instance(p) for p in fam.sample(count, seed)], case["iterations"], kind == "family")
    if kind == "batch" and case["entry"] == "call":
        out["certificates"] = {f: None for f in CERTIFICATE}
    return out | none
