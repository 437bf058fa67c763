"""What a user of this framework has it do, as cases to time: whole solves through
`pdot.optimize`, `pdot.Solver` and `pdot.optimize_batched`, the device-level passes of
include/pdot.h that stand beside a solve, and the learned warm start's network.

Solves run a fixed number of iterations (an unreachable tolerance and an iteration
limit), so that a pass is the same work on every input; each ends with the evaluation
that a converged solve ends with. Points, marginals and distributions are those of
`pdot/instances.py`; every input is made from the seed alone.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "pdot.jl_b200"))

import pdot  # noqa: E402
from pdot import _abi, instances, learned, multiscale  # noqa: E402

F64, F32 = torch.float64, torch.float32
UNREACHABLE = 1e-14  # relative tolerance that no case meets within its iterations


def listed():
    return [
        # A small problem with odd sizes (the size of a test or an assignment between two
        # short lists), solved from host arrays: latency and set-up are everything.
        {"name": "solve_tiny", "kind": "solve", "m": 127, "n": 93, "dim": 2, "cost": "f64", "iterations": 256},
        # The 1000 x 1000 configuration on a problem that stays on the GPU between solves.
        {"name": "solve_1000", "kind": "resident", "m": 1000, "n": 1000, "dim": 2, "cost": "f64", "iterations": 256},
        # The 10000 x 10000 configuration (points in three dimensions), host to host
        # through page-locked arrays.
        {"name": "solve_10000", "kind": "solve", "m": 10000, "n": 10000, "dim": 3, "cost": "f64", "iterations": 128},
        # One fused FP64 primal pass of the benchmark instance (20000 x 15000) on device
        # buffers: the building block that a caller with a loop of its own uses.
        {"name": "pass_20000", "kind": "pass", "m": 20000, "n": 15000},
        # Mixed precision on the benchmark's point cloud, cost from coordinates.
        {"name": "points_20000", "kind": "solve", "m": 20000, "n": 15000, "dim": 2, "cost": "sqeuclid", "iterations": 256},
        # The same from a warm start's duals, with the plan recovered from them.
        {"name": "points_warm", "kind": "solve", "m": 8000, "n": 6000, "dim": 2, "cost": "sqeuclid", "iterations": 128,
         "rounds": 100},
        # 512 uneven instances of the batched configuration (m, n log-uniform in 64..2048, L1
        # cost in the plane), duals wanted, with the tile balance that the tuner picks.
        {"name": "batched_512", "kind": "batched", "count": 512, "low": 64, "high": 2048, "cost": "l1", "iterations": 128},
        # 24 histogram pairs on the 32 x 32 grid, each a warm start raced against a cold one.
        {"name": "grid_race", "kind": "race", "count": 24, "side": 32, "iterations": 128, "rounds": 100},
        # 32 training steps of the warm start's network, then its weights.
        {"name": "train_256", "kind": "train", "batch": 256, "steps": 32},
        # Rounding a nearly feasible plan onto its marginals.
        {"name": "rounding_10000", "kind": "rounding", "m": 10000, "n": 10000},
        # The squared-Euclidean cost of two point sets, normalised, built where it is used.
        {"name": "cost_10000", "kind": "cost", "m": 10000, "n": 10000, "dim": 3},
        # Coarse duals extended to two point sets, with the cost's normaliser.
        {"name": "extend_20000", "kind": "extend", "m": 20000, "n": 15000, "dim": 2, "centres": 6000},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "resident", "mixed", "mixed", "warm", "pass", "batched", "race", "train",
                       "predict", "rounding", "cost", "extend"])
    if kind == "solve":  # the FP64 drop-in from host arrays
        return {"kind": "solve", "m": _log(rng, 16, 6000), "n": _log(rng, 16, 6000), "dim": rng.choice([1, 2, 3]),
                "cost": "f64", "iterations": rng.choice([32, 128, 256])}
    if kind == "resident":
        return {"kind": "resident", "m": _log(rng, 64, 6000), "n": _log(rng, 64, 6000), "dim": rng.choice([2, 3]),
                "cost": rng.choice(["f64", "f64", "sqeuclid", "l1"]), "iterations": 256}
    if kind == "mixed":  # mixed precision: each cost source, even and odd sizes
        return {"kind": "solve", "m": _log(rng, 200, 16000), "n": _log(rng, 200, 12000), "dim": rng.choice([1, 2, 3, 4]),
                "cost": rng.choice(["sqeuclid", "l1", "f32", "bf16"]), "iterations": rng.choice([128, 256])}
    if kind == "warm":
        return {"kind": "solve", "m": _log(rng, 200, 8000), "n": _log(rng, 200, 6000), "dim": rng.choice([2, 3]),
                "cost": rng.choice(["sqeuclid", "l1", "f32", "f64"]), "iterations": 128, "rounds": rng.choice([20, 100])}
    if kind == "pass":
        return {"kind": "pass", "m": _log(rng, 100, 20000), "n": _log(rng, 100, 15000)}
    if kind == "batched":
        return {"kind": "batched", "count": _log(rng, 8, 512), "low": 64, "high": rng.choice([512, 1024, 2048]),
                "cost": rng.choice(["l1", "sqeuclid", "f32"]), "iterations": 128}
    if kind == "race":
        return {"kind": "race", "count": rng.randint(4, 24), "side": rng.choice([24, 32]), "iterations": 128,
                "rounds": rng.choice([20, 100])}
    if kind == "train":
        return {"kind": "train", "batch": rng.randint(32, 512), "steps": rng.randint(4, 24)}
    if kind == "predict":
        return {"kind": "predict", "rows": _log(rng, 1, 2000)}
    if kind == "rounding":
        return {"kind": "rounding", "m": _log(rng, 100, 12000), "n": _log(rng, 100, 12000)}
    if kind == "cost":
        return {"kind": "cost", "m": _log(rng, 100, 20000), "n": _log(rng, 100, 15000), "dim": rng.choice([1, 2, 3])}
    return {"kind": "extend", "m": _log(rng, 500, 20000), "n": _log(rng, 500, 15000), "dim": rng.choice([1, 2, 3]),
            "centres": _log(rng, 100, 12000)}


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(g, *shape, low=0.0, high=1.0):
    return torch.rand(*shape, generator=g, device="cuda", dtype=F64) * (high - low) + low


def _marginal(g, k):
    w = _uniform(g, k, low=0.1, high=1.0)
    return w / w.sum()


def _points(g, k, dim, mixture):
    """U[0,1]^dim, or a mixture of 8 Gaussians (sigma 0.05), in FP32 values."""
    if not mixture:
        return _uniform(g, k, dim).to(F32)
    means = _uniform(g, 8, dim)
    pick = torch.randint(0, 8, (k,), generator=g, device="cuda")
    return (means[pick] + 0.05 * torch.randn(k, dim, generator=g, device="cuda", dtype=F64)).to(F32)


def _distances(x, y, l1=False):
    """Pairwise distances in FP64 as an (n, m) tensor: row j is column j of the m x n matrix."""
    x, y = x.to(F64), y.to(F64)
    D = torch.zeros(y.shape[0], x.shape[0], dtype=F64, device=x.device)
    for k in range(x.shape[1]):
        t = y[:, k : k + 1] - x[None, :, k]
        D += t.abs_() if l1 else t.square_()
    return D


def _cost(x, y, l1=False):
    D = _distances(x, y, l1)
    return D.div_(D.max())


def _problem(case, seed):
    """Points, marginals and, for a warm start, duals of the kind that a coarse solve leaves."""
    g = _generator(seed)
    m, n = case["m"], case["n"]
    x = _points(g, m, case["dim"], case["cost"] != "f64")
    y = _points(g, n, case["dim"], case["cost"] != "f64")
    a, b = _marginal(g, m), _marginal(g, n)
    duals = None
    if "rounds" in case:
        l1 = case["cost"] == "l1"
        cx, cy = x[:: max(1, m // 200)], y[:: max(1, n // 200)]
        C = _cost(cx, cy, l1).T
        f, h, eps = torch.zeros(C.shape[0], dtype=F64, device="cuda"), torch.zeros(C.shape[1], dtype=F64, device="cuda"), 0.02
        for _ in range(50):
            f = -eps * torch.logsumexp((h[None, :] - C) / eps, 1)
            h = -eps * torch.logsumexp((f[:, None] - C) / eps, 0)
        s = 1.0 / _distances(cx, cy, l1).max()
        u = (s * _distances(cy, x, l1) - h[None, :]).amin(1)
        v = (s * _distances(cx, y, l1) - f[None, :]).amin(1)
        duals = u.cpu().numpy(), v.cpu().numpy()
    return x, y, a, b, duals


EPS = 3e-4  # of the recovered plans, learned.RECOVER_PLAN
WARM_WEIGHT = 1e3  # initial primal weight of the warm starts: near ||duals|| / ||plan||


def _parameters(case):
    return pdot.default_parameters(UNREACHABLE, verbosity=0, iteration_limit=case["iterations"])


def _host(t, pinned):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=pinned)
    out.copy_(t)
    return out.numpy()


def _prepare_solve(case, seed):
    x, y, a, b, duals = _problem(case, seed)
    m, n = case["m"], case["n"]
    pinned = m * n >= 1 << 22  # large problems live in page-locked arrays, as the benchmark's do
    kw = {"precision": "f64"}
    C = None
    if case["cost"] == "f64":
        C = _host(_cost(x, y), pinned).T
    else:
        kw = {"precision": "f32", "cost": case["cost"]}
        if case["cost"] in ("sqeuclid", "l1"):
            kw["points"] = x.cpu().numpy(), y.cpu().numpy()
        else:
            C = _host(_cost(x, y), pinned).T
    if duals is not None:
        kw.update(warm_start=duals, recover_plan=(EPS, case["rounds"]), warm_primal_weight=WARM_WEIGHT)
    if pinned:
        kw["out"] = (torch.empty(n, m, dtype=F64, pin_memory=True).numpy().T, np.empty(m), np.empty(n))
    return {"params": _parameters(case), "problem": pdot.OptimalTransportProblem(C, a.cpu().numpy(), b.cpu().numpy()),
            "kw": kw}


def _prepare_resident(case, seed):
    x, y, a, b, _ = _problem(case, seed)
    kw, C = {}, None
    if case["cost"] == "f64":
        C = _cost(x, y)
    else:
        kw = {"precision": "f32", "cost": case["cost"], "points": (x.data_ptr(), y.data_ptr(), case["dim"])}
    torch.cuda.synchronize()
    solver = pdot.Solver(_parameters(case), device_problem=(case["m"], case["n"], C.data_ptr() if C is not None else 0,
                                                            a.data_ptr(), b.data_ptr()), **kw)
    return {"solver": solver, "keep": (x, y, a, b, C)}


def _plan(g, a, b, width=0.3):
    """A plan whose row and column sums miss the marginals by some per cent, most entries zero, as
    PDHG's averages are: (n, m)."""
    m, n = a.shape[0], b.shape[0]
    X = _uniform(g, n, m)
    X.sub_(1.0 - width).clamp_(min=0.0)
    X.mul_(a[None, :] / X.sum(0, keepdim=True).clamp(min=1e-300))
    return X.mul_(b[:, None] / X.sum(1, keepdim=True).clamp(min=1e-300) * _uniform(g, n, 1, low=0.9, high=1.1))


def _prepare_pass(case, seed):
    g = _generator(seed)
    m, n = case["m"], case["n"]
    x, y = _points(g, m, 2, True), _points(g, n, 2, True)
    a, b = _marginal(g, m), _marginal(g, n)
    X = _plan(g, a, b)
    Xa = X * _uniform(g, n, 1)
    s = {"m": m, "n": n, "C": _cost(x, y), "X": X, "Xa": Xa, "u": 0.1 * _uniform(g, m), "v": 0.1 * _uniform(g, n)}
    s["dr"], s["dc"], s["dq"] = (torch.empty(k, dtype=F64, device="cuda") for k in (m, n, 1))
    lib = _abi.load()
    s["bytes"] = lib.pdot_primal_pass_workspace_bytes(m, n)
    s["work"] = torch.empty(s["bytes"], dtype=torch.uint8, device="cuda")
    return s


PASS_STEP, PASS_NEW, PASS_SCALE = 1e-7, 0.25, 0.8


def _shapes(case):
    """Shapes of a batch: they belong to the case, only the values come from the seed."""
    rng = np.random.default_rng(0)
    lo, hi = math.log(case["low"]), math.log(case["high"])
    return [(int(round(math.exp(rng.uniform(lo, hi)))), int(round(math.exp(rng.uniform(lo, hi)))))
            for _ in range(case["count"])]


def _prepare_batched(case, seed):
    shapes = _shapes(case)
    rng = np.random.default_rng(seed)
    problems, points = [], []
    for m, n in shapes:
        x, y = rng.uniform(0, 1, (m, 2)).astype(np.float32), rng.uniform(0, 1, (n, 2)).astype(np.float32)
        C = None
        if case["cost"] == "f32":
            C = _cost(torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda(), True).cpu().numpy().T
        problems.append(pdot.OptimalTransportProblem(C, rng.dirichlet(np.ones(m)), rng.dirichlet(np.ones(n))))
        points.append((x, y))
    kw = {"cost": case["cost"], "return_primal": False, "unit_cost": 8.0}
    if case["cost"] != "f32":
        kw["points"] = points
    return {"params": _parameters(case), "problems": problems, "points": points, "kw": kw}


def _grid(side):
    r = np.arange(side, dtype=np.float32)
    return np.stack([np.tile(r, side), np.repeat(r, side)], axis=1)


def _prepare_race(case, seed):
    """Histograms of 1 to 5 Gaussians; the warm duals are an entropic solve's, near the optimum as
    a network's prediction is."""
    k, side = case["count"], case["side"]
    rng = np.random.default_rng(seed)
    h = np.stack([instances.grid_histogram(rng, side) for _ in range(2 * k)])
    A, B = torch.from_numpy(h[:k]).cuda(), torch.from_numpy(h[k:]).cuda()
    r = torch.arange(side, dtype=F64, device="cuda")
    eps = 0.005
    K1 = torch.exp(-((r[:, None] - r[None, :]) ** 2) / (2.0 * (side - 1) ** 2) / eps)
    smooth = lambda w: (K1 @ w.view(-1, side, side) @ K1).reshape(-1, side * side)  # noqa: E731
    q = torch.ones_like(B)
    for _ in range(100):
        p = A / smooth(q)
        q = B / smooth(p)
    u, v = (eps * p.log()).cpu().numpy(), (eps * q.log()).cpu().numpy()
    pts = _grid(side)
    problems = [pdot.OptimalTransportProblem(None, h[i], h[k + i]) for i in range(k)]
    kw = {"cost": "sqeuclid", "points": [(pts, pts)] * (2 * k), "return_primal": False,
          "warm_starts": [(u[i], v[i]) for i in range(k)] + [None] * k, "recover_plan": (EPS, case["rounds"]),
          "race_groups": list(range(k)) * 2, "warm_restart": "zero"}
    return {"params": _parameters(case), "problems": problems * 2, "points": kw["points"], "kw": kw}


def _network(seed, rows):
    """A network (2048 -> 1024 -> 1024 -> 2048) and its parameters."""
    width, hidden = 2 * learned.BINS, 1024
    g = _generator(seed)
    parts = []
    for fan, out in ((width, hidden), (hidden, hidden), (hidden, width)):
        bound = 1.0 / math.sqrt(fan)
        parts += [_uniform(g, out * fan, low=-bound, high=bound), _uniform(g, out, low=-bound, high=bound)]
    theta = torch.cat(parts).to(F32)
    net = learned.MLP(width, hidden, width, max_batch=rows, seed=0)
    net.set_parameters(theta.cpu().numpy())
    return net, theta, g


def _histograms(g, rows):
    h = torch.exp(1.5 * torch.randn(rows, 2, learned.BINS, generator=g, device="cuda", dtype=F64))
    return (h / h.sum(2, keepdim=True)).view(rows, 2 * learned.BINS)


def _prepare_train(case, seed):
    net, theta, g = _network(seed, case["batch"])
    rows = case["batch"] * case["steps"]
    return {"net": net, "theta": theta, "batch": case["batch"], "steps": case["steps"], "hist": _histograms(g, rows),
            "target": torch.randn(rows, 2 * learned.BINS, generator=g, device="cuda", dtype=F32)}


RATE, DECAY = 1e-4, 1e-4


def _rate(k, steps):
    return RATE * 0.5 * (1.0 + math.cos(math.pi * k / steps))


def _prepare_predict(case, seed):
    net, theta, g = _network(seed, 512)
    return {"net": net, "theta": theta, "hist": _histograms(g, case["rows"]).cpu().numpy()}


def _prepare_rounding(case, seed):
    g = _generator(seed)
    a, b = _marginal(g, case["m"]), _marginal(g, case["n"])
    return {"m": case["m"], "n": case["n"], "a": a, "b": b, "X": _plan(g, a, b)}


def _prepare_cost(case, seed):
    g = _generator(seed)
    m, n, d = case["m"], case["n"], case["dim"]
    return {"m": m, "n": n, "dim": d, "x": _uniform(g, m, d), "y": _uniform(g, n, d),
            "C": torch.empty(n, m, dtype=F64, device="cuda")}


def _prepare_extend(case, seed):
    g = _generator(seed)
    x, y = _points(g, case["m"], case["dim"], True), _points(g, case["n"], case["dim"], True)
    host = lambda t: t.to(F64).cpu().numpy()  # noqa: E731
    cx, cy = _points(g, case["centres"], case["dim"], True), _points(g, case["centres"], case["dim"], True)
    return {"x": x, "y": y, "cx": host(cx), "cy": host(cy), "du": host(0.1 * _uniform(g, case["centres"])),
            "dv": host(0.1 * _uniform(g, case["centres"])), "scale": 0.5}


def prepare(case, seed):
    return {**globals()["_prepare_" + case["kind"]](case, seed), "kind": case["kind"]}


# ------------------------------------------------------------------ passes
def _solution(out):
    return {"plan": out.primal_solution, "source_dual": out.dual_source_solution,
            "target_dual": out.dual_target_solution, "iterations": out.iteration_count}


def _run_solve(s):
    return _solution(pdot.optimize(s["params"], s["problem"], **s["kw"]))


def _run_resident(s):
    s["solver"].reset()
    return _solution(s["solver"].finish())


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _run_pass(s):
    lib = _abi.load()
    p = {k: t.data_ptr() for k, t in s.items() if isinstance(t, torch.Tensor)}
    _abi.check(lib, lib.pdot_primal_pass_f64(s["m"], s["n"], p["C"], p["X"], p["Xa"], p["u"], p["v"], PASS_STEP, PASS_NEW,
                                             PASS_SCALE, 0, p["dr"], p["dc"], p["dq"], p["work"], s["bytes"], _stream()),
               "pdot_primal_pass_f64")
    return {"plan": s["X"], "average": s["Xa"], "rows": s["dr"], "columns": s["dc"], "square": s["dq"]}


def _run_batched(s):
    outs, _ = pdot.optimize_batched(s["params"], s["problems"], **s["kw"])
    return {"source_dual": np.concatenate([o.dual_source_solution for o in outs]),
            "target_dual": np.concatenate([o.dual_target_solution for o in outs]),
            "iterations": np.array([o.iteration_count for o in outs])}


_run_race = _run_batched


def _run_train(s):
    net, batch = s["net"], s["batch"]
    for k in range(s["steps"]):
        net.set_input(s["hist"][k * batch :].data_ptr(), batch)
        net.train_step(s["target"][k * batch :].data_ptr(), _rate(k, s["steps"]), DECAY, k % 16 == 0)
    return {"parameters": net.get_parameters()}


def _run_predict(s):
    return {"duals": learned.forward_rows(s["net"], s["hist"])}


def _run_rounding(s):
    lib = _abi.load()
    _abi.check(lib, lib.pdot_rounding_f64(s["m"], s["n"], s["a"].data_ptr(), s["b"].data_ptr(), s["X"].data_ptr(),
                                          _stream()), "pdot_rounding_f64")
    return {"plan": s["X"]}


def _run_cost(s):
    lib = _abi.load()
    _abi.check(lib, lib.pdot_sqeuclid_cost_f64(s["m"], s["n"], s["dim"], s["x"].data_ptr(), s["y"].data_ptr(), 1,
                                               s["C"].data_ptr(), _stream()), "pdot_sqeuclid_cost_f64")
    return {"cost": s["C"]}


def _run_extend(s):
    return {"largest": multiscale.max_sq_distance(s["x"], s["y"]),
            "source_dual": multiscale.c_transform(s["x"], s["cy"], s["dv"], s["scale"]),
            "target_dual": multiscale.c_transform(s["y"], s["cx"], s["du"], s["scale"])}


def run(state):
    return globals()["_run_" + state["kind"]](state)


# ------------------------------------------------------------------ least work
def work(case):
    """Bytes: inputs and outputs once and, for a solve, what every iteration has to update (the plan
    and its average) and read (a stored cost), which no call can keep in registers; the recovery of a
    plan, the c-transforms and the network are arithmetic."""
    kind, n2 = case["kind"], case.get("m", 0) * case.get("n", 0)
    if kind in ("solve", "resident"):
        entry, per = {"f64": (8, 40), "f32": (8, 20), "bf16": (8, 18)}.get(case["cost"], (0, 16))
        return {"bytes": n2 * (entry + 8 + per * case["iterations"]),
                "flops": n2 * (12.0 * case["iterations"] + 2 * 12.0 * case.get("rounds", 0))}
    if kind == "pass":
        return {"bytes": 40 * n2, "flops": 12.0 * n2}
    if kind in ("batched", "race"):
        if kind == "race":
            entries = 2 * case["count"] * case["side"] ** 4
            extra = case["count"] * case["side"] ** 4 * 2 * 12.0 * case["rounds"]
        else:
            entries, extra = sum(m * n for m, n in _shapes(case)), 0.0
        per = 20 if case.get("cost") == "f32" else 16
        return {"bytes": entries * per * case["iterations"], "flops": entries * 12.0 * case["iterations"] + extra}
    if kind in ("train", "predict"):
        weights = 1024 * (2048 + 1024 + 2048)
        if kind == "train":
            rows = case["batch"] * case["steps"]
            return {"bytes": case["steps"] * weights * 28 + rows * 2048 * 12, "flops": 6.0 * weights * rows}
        return {"bytes": weights * 2 + case["rows"] * 2048 * 12, "flops": 2.0 * weights * case["rows"]}
    if kind == "rounding":
        return {"bytes": 16 * n2, "flops": 8.0 * n2}
    if kind == "cost":
        return {"bytes": 8 * n2, "flops": 3.0 * case["dim"] * n2}
    pairs = case["m"] * case["n"] + case["centres"] * (case["m"] + case["n"])
    return {"bytes": 4 * case["dim"] * (case["m"] + case["n"]) + 8 * (case["m"] + case["n"]), "flops": 3.0 * case["dim"] * pairs}


# ------------------------------------------------------------------ the same in 64 bits
def _point(C, a, b, X, u, v, zero):
    """The sums of an evaluated point: objectives, residual and variable norms."""
    G = torch.zeros_like(C) if zero else C - u[None, :] - v[:, None]
    pobj, dobj = (C * X).sum(), a @ u + b @ v
    rp = ((a - X.sum(0)).square().sum() + (b - X.sum(1)).square().sum()).sqrt()
    return [float(t) for t in (rp, G.clamp_(max=0.0).norm(), (pobj - dobj).abs(), X.norm(), (u @ u + v @ v).sqrt())]


def _weighted(p, w):
    return math.sqrt(w * p[0] ** 2 + p[1] ** 2 / w + p[2] ** 2)


def _pdhg(C, a, b, iterations, start=None, at_zero=False, omega=1.0, freq=128):
    """Restarted adaptive PDHG on the (n, m) cost for a fixed number of iterations, from zero or a
    (plan, duals) start: the returned average and duals."""
    zero = start is None
    X = torch.zeros_like(C) if zero else start[0].clone()
    u = torch.zeros_like(a) if zero else start[1].clone()
    v = torch.zeros_like(b) if zero else start[2].clone()
    tau, S, count, trials, ratio_last = 1.0, 0.0, 0, 0, 1.0
    last = [float((a @ a + b @ b).sqrt()), 0.0, 0.0, 0.0, 0.0]
    if not zero and not at_zero:
        last = _point(C, a, b, X, u, v, False)
    r, c = X.sum(0), X.sum(1)
    Xa, ua, va, ra, ca = X.clone(), u.clone(), v.clone(), r.clone(), c.clone()
    for it in range(1, iterations + 2):
        if it <= 10 or (it - 1) % freq == 0 or it == iterations + 1:
            if it > iterations:
                return (Xa, ua, va) if count else (X, u, v)
            if count:
                cur, avg = _point(C, a, b, X, u, v, zero), _point(C, a, b, Xa, ua, va, zero)
                kc, ka = _weighted(cur, omega), _weighted(avg, omega)
                cand, kl = min(kc, ka), _weighted(last, omega)
                go = count >= 0.36 * (it - 1)
                if not go:
                    ratio = cand / kl
                    go = ratio < 0.9 and (ratio < 0.1 or ratio > ratio_last)
                    ratio_last = ratio
                if go:
                    moved_p, moved_d = math.sqrt(omega / tau) * last[3] / math.sqrt(omega), math.sqrt(1 / (tau * omega)) * last[4] * math.sqrt(omega)
                    last = avg if kc >= ka else cur
                    if kc >= ka:
                        X, u, v, r, c = Xa.clone(), ua.clone(), va.clone(), ra.clone(), ca.clone()
                    S, count = 0.0, 0
                    if moved_p > 2.3e-16 and moved_d > 2.3e-16:
                        omega = math.exp(0.5 * math.log(moved_d / moved_p) + 0.5 * math.log(omega))
        D = torch.zeros_like(C) if zero else (C - u[None, :]).sub_(v[:, None]).mul_(-tau / omega)
        D.add_(X).clamp_(min=0.0).sub_(X)
        X.add_(D)
        rn, cn = r + D.sum(0), c + D.sum(1)
        un, vn = u + tau * omega * (a - 2 * rn + r), v + tau * omega * (b - 2 * cn + c)
        du, dv = un - u, vn - v
        inter = abs(float((rn - r) @ du + (cn - c) @ dv))
        move = 0.5 * omega * float(D.norm()) ** 2 + 0.5 / omega * float(du @ du + dv @ dv)
        limit, weight, ok = (move / inter if inter > 0 else math.inf), tau, False
        while not ok:
            trials += 1
            ok = tau <= limit
            tau = min((1 - 1 / (trials + 1) ** 2) * limit, (1 + 1 / (trials + 1)) * tau)
        nw, aw = (1.0, 1.0) if S == 0 else (weight / S, S / (S + weight))
        u, v, r, c, zero = un, vn, rn, cn, False
        for avg_t, t in ((Xa, X), (ua, u), (va, v), (ra, r), (ca, c)):
            if S == 0:
                avg_t.copy_(t)
            else:
                avg_t.add_(t, alpha=nw).mul_(aw)
        S, count = S + weight, count + 1


def _recovered(C, a, b, u, v, rounds, eps=EPS):
    f, h = u, v
    for _ in range(rounds):
        f = eps * (a.log() - torch.logsumexp((h[:, None] - C) / eps, 0))
        h = eps * (b.log() - torch.logsumexp((f[None, :] - C) / eps, 1))
    return torch.exp((f[None, :] + h[:, None] - C) / eps)


def _exact_solve(case, seed):
    """None for cold solves with an FP32 plan, or of more than 128 iterations, or on long and narrow
    problems: their restarts and adaptive steps amplify one rounding of the iterates by 1e6 and more, so
    that the outputs have no value in 64 bits to be compared with."""
    comparable = case["cost"] == "f64" and case["iterations"] <= 128
    if "rounds" not in case and (not comparable or not 1 / 16 <= case["m"] / case["n"] <= 16):
        return None
    x, y, a, b, duals = _problem(case, seed)
    C = _cost(x, y, case["cost"] == "l1")
    start = None
    if duals is not None:
        u, v = (torch.from_numpy(t).cuda() for t in duals)
        start = (_recovered(C, a, b, u, v, case["rounds"]), u, v)
    X, u, v = _pdhg(C, a, b, case["iterations"], start, omega=1.0 if start is None else WARM_WEIGHT)
    return {"plan": X.cpu().numpy().T if comparable else None, "source_dual": u.cpu().numpy(), "target_dual": v.cpu().numpy(),
            "iterations": case["iterations"]}


_exact_resident = _exact_solve


def _exact_pass(case, seed):
    s = _prepare_pass(case, seed)
    D = (s["C"] - s["u"][None, :] - s["v"][:, None]).mul_(-PASS_STEP).add_(s["X"]).clamp_(min=0.0).sub_(s["X"])
    X = s["X"] + D
    return {"plan": X, "average": (s["Xa"] + X * PASS_NEW) * PASS_SCALE, "rows": D.sum(0), "columns": D.sum(1),
            "square": D.square().sum().view(1)}


def _exact_batched(case, seed):
    s = globals()["_prepare_" + case["kind"]](case, seed)
    if len(s["problems"]) > 64:  # one after another, they would take too long
        return None
    U, V = [], []
    for i, p in enumerate(s["problems"]):
        x, y = (torch.from_numpy(t).cuda() for t in s["points"][i])
        C = _cost(x, y, case.get("cost") in ("l1", "f32"))
        a, b = torch.from_numpy(p.source_distribution).cuda(), torch.from_numpy(p.target_distribution).cuda()
        w, start = (s["kw"].get("warm_starts") or [None] * (i + 1))[i], None
        if w is not None:
            u, v = torch.from_numpy(w[0]).cuda(), torch.from_numpy(w[1]).cuda()
            start = (_recovered(C, a, b, u, v, case["rounds"]), u, v)
        _, u, v = _pdhg(C, a, b, case["iterations"], start, at_zero=True)
        U.append(u.cpu().numpy())
        V.append(v.cpu().numpy())
    return {"source_dual": np.concatenate(U), "target_dual": np.concatenate(V),
            "iterations": np.full(len(U), case["iterations"])}


_exact_race = _exact_batched


def _layers(theta):
    shapes, out, at = ((1024, 2048), (1024,), (1024, 1024), (1024,), (2048, 1024), (2048,)), [], 0
    for sh in shapes:
        k = math.prod(sh)
        out.append(theta[at : at + k].to(F64).view(sh).clone())
        at += k
    return out


def _forward(p, hist):
    z = (hist.clamp(min=1e-30).log() + learned.FEATURE_SHIFT) * learned.FEATURE_SCALE
    for k in (0, 2):
        z = torch.nn.functional.gelu(z @ p[k].T + p[k + 1])
    return z @ p[4].T + p[5]


def _exact_train(case, seed):
    s = _prepare_train(case, seed)
    p = [t.requires_grad_() for t in _layers(s["theta"])]
    m, v = [torch.zeros_like(t) for t in p], [torch.zeros_like(t) for t in p]
    for k in range(case["steps"]):
        rows = slice(k * case["batch"], (k + 1) * case["batch"])
        grads = torch.autograd.grad((_forward(p, s["hist"][rows]) - s["target"][rows].to(F64)).square().mean(), p)
        with torch.no_grad():
            for t, g, mt, vt in zip(p, grads, m, v):
                mt.mul_(0.9).add_(g, alpha=0.1)
                vt.mul_(0.999).add_(g.square(), alpha=0.001)
                step = (mt / (1 - 0.9 ** (k + 1))) / ((vt / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
                t.sub_(_rate(k, case["steps"]) * (step + (DECAY * t if t.dim() == 2 else 0.0)))
    return {"parameters": torch.cat([t.detach().view(-1) for t in p])}


def _exact_predict(case, seed):
    s = _prepare_predict(case, seed)
    return {"duals": _forward(_layers(s["theta"]), torch.from_numpy(s["hist"]).cuda())}


def _exact_rounding(case, seed):
    s = _prepare_rounding(case, seed)
    X = s["X"] * (s["a"] / s["X"].sum(0)).nan_to_num(nan=0.0).clamp(max=1.0)[None, :]
    X = X * (s["b"] / X.sum(1)).nan_to_num(nan=0.0).clamp(max=1.0)[:, None]
    er, ec = s["a"] - X.sum(0), s["b"] - X.sum(1)
    norm = er.abs().sum()
    return {"plan": X + ec[:, None] * (er / norm if norm > 0 else er)[None, :]}


def _exact_cost(case, seed):
    s = _prepare_cost(case, seed)
    return {"cost": _cost(s["x"], s["y"])}


def _exact_extend(case, seed):
    s = _prepare_extend(case, seed)
    back = lambda p, c, d: torch.cat([  # noqa: E731
        (s["scale"] * _distances(torch.from_numpy(c).cuda(), q) - torch.from_numpy(d).cuda()[None, :]).amin(1)
        for q in p.split(2000)])
    return {"largest": float(_distances(s["x"], s["y"]).max()), "source_dual": back(s["x"], s["cy"], s["dv"]),
            "target_dual": back(s["y"], s["cx"], s["du"])}


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)
