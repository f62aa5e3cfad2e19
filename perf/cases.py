"""What the framework is used for, as cases that can be timed and compared.

A pass is one solve through the public Python API: a QUBO roof-dual LP (PRAQ)
or a joint replenishment LP (PRIA), on an instance that is resident on the GPU
or on host arrays, alone or in a batch.  Each function below takes a case, a
dict of plain values; `listed` names twelve, `draw` makes more of the same
ranges.  Inputs are seeded synthetic instances of the shapes and distributions
of the package's generators.
"""

from __future__ import annotations

import math
import types

import numpy as np
import torch

from reformulation_b200 import batch as rb_batch
from reformulation_b200 import praq, pria
from reformulation_b200.instances import QuboInstance, jrp_demand

# Tolerances as the package's benchmark and tests use them: 1e-4 for FP32
# iterates ("mixed"), 1e-6 for FP64.
TOLERANCE = {"mixed": 1e-4, "fp64": 1e-6}
CAP = 4000   # iterations: a bound, not reached by the listed cases


def listed():
    return [
        # The smallest call: a QUBO of 200 variables on host arrays, one-shot
        # (set-up, solve, tear-down), as a branch-and-bound node bounds itself.
        {"name": "qubo_200_oneshot", "kind": "qubo_oneshot", "n": 200, "m": 1000, "precision": "fp64"},
        # A few thousand variables, resident: the size of most public QUBO sets.
        {"name": "qubo_3k", "kind": "qubo", "n": 3001, "m": 24007, "precision": "mixed"},
        # The middle of the range in FP64, odd sizes, average degree 30.
        {"name": "qubo_20k_fp64", "kind": "qubo", "n": 20011, "m": 300007, "precision": "fp64"},
        # A re-solve from an earlier solution's neighbourhood (the warm-start
        # call), edges in no order, returning the dual as well.
        {"name": "qubo_30k_warm", "kind": "qubo_warm", "n": 30000, "m": 199999, "precision": "fp64"},
        # The benchmark's headline: n = 1e5, m = 1e6, resident, FP32 iterates.
        {"name": "qubo_100k", "kind": "qubo", "n": 100000, "m": 1000000, "precision": "mixed"},
        # The same from host arrays in FP64: upload, layout and solve.
        {"name": "qubo_100k_oneshot", "kind": "qubo_oneshot", "n": 100000, "m": 1000000, "precision": "fp64"},
        # The largest rung of the QUBO ladder: working set far above L2.
        {"name": "qubo_2m", "kind": "qubo", "n": 2000000, "m": 20000000, "precision": "mixed"},
        # A small JRP, resident, with its solution: latency.
        {"name": "jrp_10x25", "kind": "jrp", "items": 10, "periods": 25, "precision": "fp64", "solution": True},
        # An ordinary JRP from host arrays with its solution (FP32 interface).
        {"name": "jrp_40x120_oneshot", "kind": "jrp_oneshot", "items": 40, "periods": 120, "precision": "mixed"},
        # A year of days (odd, so padded) in FP64; bounds, as the backend returns.
        {"name": "jrp_60x365_fp64", "kind": "jrp", "items": 60, "periods": 365, "precision": "fp64", "solution": False},
        # The benchmark's JRP: 100 items, 500 periods, FP32 iterates.
        {"name": "jrp_100x500", "kind": "jrp", "items": 100, "periods": 500, "precision": "mixed", "solution": False},
        # A set of QUBOs and JRPs of uneven size in one batched engine.
        {"name": "batch_16q_8j", "kind": "batch", "qubos": 16, "jrps": 8, "n_low": 500, "n_high": 30000,
         "items_high": 60, "periods_high": 250, "precision": "mixed"},
    ]


def draw(rng):
    def log_uniform(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    precision = rng.choice(["mixed", "fp64"])
    kind = rng.choice(["qubo", "qubo", "qubo_oneshot", "qubo_warm", "jrp", "jrp", "jrp_oneshot", "batch"])
    if kind.startswith("qubo"):
        n = log_uniform(200, 1000000)
        m = max(1, min(int(n * rng.uniform(2.0, 10.0)), n * (n - 1) // 4))
        return {"kind": kind, "n": n, "m": m, "precision": precision}
    if kind == "batch":
        return {"kind": kind, "qubos": rng.randint(2, 16), "jrps": rng.randint(1, 8), "n_low": 300,
                "n_high": log_uniform(1000, 30000), "items_high": rng.randint(10, 60),
                "periods_high": rng.randint(60, 250), "precision": "mixed"}
    periods = log_uniform(10, 700)
    items = min(log_uniform(3, 200), max(3, 25_000_000 // (periods * (periods + 1))))
    if kind == "jrp_oneshot":
        items = min(items, max(3, 4_000_000 // (periods * (periods + 1))))
        return {"kind": kind, "items": items, "periods": periods, "precision": precision}
    return {"kind": kind, "items": items, "periods": periods, "precision": precision,
            "solution": items * periods * periods < 1_000_000}


# ---- instances -----------------------------------------------------------------

def _qubo(seed, n, m, ordered=True):
    """m distinct pairs i < j uniform over all pairs, in row order (or, not
    `ordered`, in a random one); weights nonzero integers in [-100, 100]."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device=dev).manual_seed(int(seed))
    code = torch.empty(0, dtype=torch.int64, device=dev)
    while code.numel() < m:
        k = int((m - code.numel()) * 1.1) + 64
        a = torch.randint(0, n, (k,), generator=g, device=dev)
        b = torch.randint(0, n, (k,), generator=g, device=dev)
        lo, hi = torch.minimum(a, b), torch.maximum(a, b)
        code = torch.unique(torch.cat([code, (lo * n + hi)[lo != hi]]))
    keep = torch.randperm(code.numel(), generator=g, device=dev)[:m]
    code = code[keep.sort().values if ordered else keep]
    vals = torch.randint(-100, 100, (m,), generator=g, device=dev)
    vals = vals + (vals >= 0)
    diag = torch.randint(-100, 101, (n,), generator=g, device=dev)
    return QuboInstance(f"qubo-n{n}-m{m}", "perf", n, diag.double().cpu().numpy(),
                        (code // n).cpu().numpy(), (code % n).cpu().numpy(), vals.double().cpu().numpy())


def _warm_point(inst, seed):
    rng = np.random.default_rng(seed + 77)
    return rng.uniform(0.0, 1.0, inst.n), rng.normal(0.0, 20.0, (inst.vals.size, 2))


def _batch_instances(case, seed):
    """QUBO sizes log-uniform with average degree 4 to 16, JRP sizes
    log-uniform: the shape of the package's batch workload.  The sizes are the
    case's, the data the seed's."""
    sizes = np.random.default_rng(11)

    def log_uniform(a, b):
        return int(round(math.exp(sizes.uniform(math.log(a), math.log(b)))))

    qubos, jrps = [], []
    for k in range(case["qubos"]):
        n = log_uniform(case["n_low"], case["n_high"])
        qubos.append(_qubo(seed * 1000 + k, n, int(n * sizes.uniform(2.0, 8.0))))
    for k in range(case["jrps"]):
        jrps.append(jrp_demand(seed * 1000 + 500 + k, log_uniform(10, max(11, case["items_high"])),
                               log_uniform(30, max(31, case["periods_high"]))))
    return qubos, jrps


def _praq_parameters(case):
    return praq.Library().parameters(tolerance=TOLERANCE[case["precision"]], max_iter=CAP,
                                     use_float32=int(case["precision"] == "mixed"))


def _pria_parameters(case):
    return pria.Library().parameters(CAP, TOLERANCE[case["precision"]])


# ---- the passes ----------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = types.SimpleNamespace(case=case)
    if kind.startswith("qubo"):
        s.inst = _qubo(seed, case["n"], case["m"], ordered=kind != "qubo_warm")
        s.params = _praq_parameters(case)
        if kind == "qubo":
            s.solver = praq.DeviceSolver(s.inst, s.params)
        elif kind == "qubo_oneshot":
            s.library = praq.Library()
        else:
            s.warm = _warm_point(s.inst, seed)
    elif kind.startswith("jrp"):
        s.inst = jrp_demand(seed, case["items"], case["periods"])
        s.params = _pria_parameters(case)
        if kind == "jrp":
            s.solver = pria.DeviceSolver(s.inst, s.params, case["precision"])
        else:
            s.library = pria.Library()
    else:
        qubos, jrps = _batch_instances(case, seed)
        s.batch = rb_batch.Batch(case["precision"])
        s.qubos = [s.batch.add_qubo(q, _praq_parameters(case)) for q in qubos]
        s.jrps = [s.batch.add_jrp(j, _pria_parameters(case)) for j in jrps]
        s.batch.start()
    return s


def _qubo_result(r):
    return {"lower": r.lower, "upper": r.upper, "iterations": r.iterations, "status": r.status, "x": r.x}


def _jrp_result(r):
    out = {"upper": r.primal_objective, "lower": r.dual_objective, "iterations": r.iterations}
    if r.x is not None:
        out |= {"x": r.x, "y": r.y, "z": r.z}
    return out


def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "qubo":
        state.solver.run()
        return _qubo_result(state.solver.result())
    if kind == "qubo_oneshot":
        return _qubo_result(state.library.solve(state.inst, state.params))
    if kind == "qubo_warm":
        x, y, iterations = praq.solve_warm_start(state.inst, state.params, state.warm)
        return {"x": x, "y": y, "iterations": iterations}
    if kind == "jrp":
        state.solver.run()
        out = _jrp_result(state.solver.result(want_solution=case["solution"]))
        if case["solution"] and case["precision"] == "mixed":
            # FP32 iterates come back widened; they are kept as they are
            out |= {k: out[k].astype(np.float32) for k in "xyz"}
        return out
    if kind == "jrp_oneshot":
        return _jrp_result(state.library.solve(state.inst, state.params, precision=case["precision"],
                                               want_solution=True))
    state.batch.restart()
    state.batch.run()
    out = {"qubo%d" % k: _qubo_result(state.batch.result_qubo(i)) for k, i in enumerate(state.qubos)}
    # up to 64 outputs: the QUBOs' points and the JRPs' bounds whole, the
    # scalars of one kind side by side
    x = {"x%d" % k: r["x"] for k, r in enumerate(out.values())}
    jrp = [state.batch.result_jrp(i) for i in state.jrps]
    return x | {
        "qubo_bounds": np.array([[r["lower"], r["upper"]] for r in out.values()], np.float32),
        "qubo_iterations": np.array([r["iterations"] for r in out.values()]),
        "jrp_bounds": np.array([[r.dual_objective, r.primal_objective] for r in jrp], np.float32),
        "jrp_iterations": np.array([r.iterations for r in jrp])}


# ---- what a pass cannot do without -----------------------------------------------

def _iterations(case):
    """Typical iterations to the case's tolerance (they vary with the data)."""
    if case["kind"].startswith("qubo"):
        return 64 if case["precision"] == "mixed" else 112
    return 96 if case["precision"] == "mixed" else 144


def _qubo_work(n, m, real, iterations):
    # per iteration: an edge's ends, weight, dual and anchor read, dual
    # written; a node's diagonal, degree, point and anchor read, point written
    return {"bytes": iterations * (m * (8 + 4 * real) + n * (6 * real + 4)),
            "flops": iterations * (12 * m + 14 * n)}


def _jrp_work(items, periods, real, iterations):
    entries = items * periods * (periods + 1) // 2
    # per iteration and entry: h, and x, y, z with their anchors read; x, y, z
    # written; three projections of about four rounds each
    return {"bytes": iterations * entries * 10 * real, "flops": iterations * entries * 45}


def work(case):
    real = 4 if case["precision"] == "mixed" else 8
    its = _iterations(case)
    if case["kind"].startswith("qubo"):
        return _qubo_work(case["n"], case["m"], real, its)
    if case["kind"].startswith("jrp"):
        return _jrp_work(case["items"], case["periods"], real, its)
    sizes = np.random.default_rng(11)
    total = {"bytes": 0, "flops": 0}
    parts = []
    for _ in range(case["qubos"]):
        n = math.exp(sizes.uniform(math.log(case["n_low"]), math.log(case["n_high"])))
        parts.append(_qubo_work(int(n), int(n * sizes.uniform(2.0, 8.0)), real, 64))
    for _ in range(case["jrps"]):
        items = math.exp(sizes.uniform(math.log(10), math.log(max(11, case["items_high"]))))
        periods = math.exp(sizes.uniform(math.log(30), math.log(max(31, case["periods_high"]))))
        parts.append(_jrp_work(int(items), int(periods), real, 96))
    for p in parts:
        total = {k: total[k] + p[k] for k in total}
    return total


# ---- the same in 64 bits, in plain torch -------------------------------------------

class _Restarts:
    """The restart and weight-update rules both LPs share (scalars only)."""

    def __init__(self, p, tolerance):
        self.p, self.tolerance = p, tolerance
        self.omega, self.theta = p.omega, p.theta_initial
        self.iteration = self.since = 0
        self.check_error = math.inf
        self.fp_error = math.nan

    def stop(self, lower, upper):
        gap = (upper - lower) / (1.0 + abs(upper) + abs(lower))
        return not (self.iteration < CAP and not gap <= self.tolerance)

    def after_block(self, error, primal_drift, dual_drift):
        """Whether to restart at this check; moves omega and theta with it."""
        p = self.p
        restart = (error <= p.beta_sufficient * self.fp_error
                   or (error <= p.beta_necessary * self.fp_error and error > self.check_error)
                   or self.since >= p.beta_artificial * self.iteration)
        if not restart:
            self.check_error = error
            return False
        if primal_drift > 1e-16 and dual_drift > 1e-16:
            self.omega = math.exp(self.theta * (math.log(dual_drift) - math.log(primal_drift))
                                  + (1.0 - self.theta) * math.log(self.omega))
            self.theta = p.theta_target + p.theta_decay * (self.theta - p.theta_target)
        return True

    def restarted(self, error):
        self.fp_error, self.check_error, self.since = error, math.inf, 0


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _exact_qubo(inst, p, tolerance, warm=None):
    dev = _device()
    eta = 0.999
    i = torch.from_numpy(np.ascontiguousarray(inst.rows)).to(dev)
    j = torch.from_numpy(np.ascontiguousarray(inst.cols)).to(dev)
    signed = 2.0 * torch.from_numpy(inst.vals).to(dev)
    diag = torch.from_numpy(inst.diag).to(dev)
    scale = math.sqrt(float((signed * signed).sum() + (diag * diag).sum())) or 1.0
    signed, diag = signed / scale, diag / scale
    w, cover = signed.abs(), signed > 0
    one = torch.ones_like(w)
    deg = torch.zeros_like(diag).index_add_(0, i, one).index_add_(0, j, one).clamp_(min=1.0)
    low, high = torch.where(cover, -w, 0.0 * w), torch.where(cover, 0.0 * w, w)

    def other(u):   # the second coordinate of a pair
        return torch.where(cover, u, w - u)

    def scatter(u):
        return torch.zeros_like(diag).index_add_(0, i, u).index_add_(0, j, other(u))

    def step(x, u, omega):
        x2 = (x - eta / omega * ((diag - scatter(u)) / deg)).clamp_(0.0, 1.0)
        r = 2.0 * x2 - x
        d = torch.where(cover, 1.0 - r[i] - r[j], r[j] - r[i])
        return x2, torch.minimum(torch.maximum(u + 0.5 * eta * omega * d, low), high)

    def norm(x, x2, u, u2, omega):
        dx, du = x - x2, u - u2
        cross = (torch.where(cover, dx[i] + dx[j], dx[i] - dx[j]) * du).sum()
        v = omega / eta * (deg * dx * dx).sum() + 2.0 * (du * du).sum() / (eta * omega) + 2.0 * cross
        return math.sqrt(max(float(v), 0.0))

    def bounds(x, u):
        upper = (diag * x).sum() + torch.where(cover, w * (x[i] + x[j] - 1.0).clamp(min=0.0),
                                               -w * torch.minimum(x[i], x[j])).sum()
        lower = (diag - scatter(u)).clamp(max=0.0).sum() + torch.where(cover, u, 0.0 * u).sum()
        return float(lower) * scale, float(upper) * scale

    x, u = torch.full_like(diag, 0.5), -0.5 * signed
    if warm is not None:
        x = torch.from_numpy(warm[0]).to(dev).clamp(0.0, 1.0)
        y = torch.from_numpy(warm[1]).to(dev) / scale
        a, b = y[:, 0], y[:, 1]
        u = torch.where(cover, 0.5 * (a + b), a + 0.5 * (w - a - b))
        u = torch.minimum(torch.maximum(u, low), high)
    s = _Restarts(p, tolerance)
    x0, u0 = x, u
    lower, upper = bounds(x, u)
    x2, u2 = step(x, u, s.omega)
    s.fp_error = norm(x, x2, u, u2, s.omega)
    if s.stop(lower, upper):
        x2, u2 = x, u
    else:
        while True:
            for _ in range(int(p.op_steps)):
                k = s.since + 1.0
                x = k / (k + 1.0) * (2.0 * x2 - x) + x0 / (k + 1.0)
                u = k / (k + 1.0) * (2.0 * u2 - u) + u0 / (k + 1.0)
                x2, u2 = step(x, u, s.omega)
                s.since += 1
                s.iteration += 1
            error = norm(x, x2, u, u2, s.omega)
            lower, upper = bounds(x2, u2)
            if s.stop(lower, upper):
                break
            if s.after_block(error, math.sqrt(float((deg * (x - x0) ** 2).sum())),
                             math.sqrt(float(2.0 * ((u - u0) ** 2).sum()))):
                x, u = x2, u2
                x0, u0 = x, u
                x2, u2 = step(x, u, s.omega)
                s.restarted(norm(x, x2, u, u2, s.omega))
    y = torch.stack([u2, other(u2)], 1) * scale
    return lower, upper, s.iteration, x2.cpu().numpy(), y.cpu().numpy()


def _exact_jrp(inst, p, tolerance):
    dev = _device()
    n, t = inst.items, inst.periods
    tp = t + t % 2
    h = torch.zeros((n, tp, tp), dtype=torch.float64, device=dev)
    h[:, :t, :t] = torch.from_numpy(inst.holding_costs).to(dev)
    on = torch.ones((tp, tp), dtype=torch.bool, device=dev).triu()
    h = torch.where(on, h, 0.0 * h)
    k = torch.from_numpy(inst.order_costs).to(dev)
    k0 = float(inst.joint_order_cost)
    scale = math.sqrt(float((h * h).sum() + (k * k).sum()) + k0 * k0) or 1.0
    h, k, k0 = h / scale, k / scale, k0 / scale
    onf = on.double()

    def project(v, dims, target):
        """Onto {v >= 0, sum over dims = target}: the threshold's fixed point."""
        count = onf.expand_as(v).sum(dims, keepdim=True)
        th = ((v * onf).sum(dims, keepdim=True) - target) / count
        while True:
            active = ((v > th) & on).double()
            fewer = active.sum(dims, keepdim=True)
            better = (fewer < count) & (fewer > 0)   # counts only fall: it ends
            if not bool(better.any()):
                return (v - th).clamp(min=0.0) * onf
            th = torch.where(better, ((v * active).sum(dims, keepdim=True) - target) / fewer.clamp(min=1.0), th)
            count = torch.where(better, fewer, count)

    def step(x, y, z, omega):
        tau, sigma = p.eta / omega, p.eta * omega
        x2 = project(x - tau * (h + y + z), (1,), 1.0)
        r = sigma * (2.0 * x2 - x)
        return x2, project(y + r, (2,), k[:, None, None]), project(z + r, (0, 2), k0)

    def norm(a, b, omega):
        dx, dy, dz = (u - v for u, v in zip(a, b))
        v = (omega / p.eta * (dx * dx).sum() + ((dy * dy).sum() + (dz * dz).sum()) / (p.eta * omega)
             - 2.0 * (dx * (dy + dz)).sum())
        return math.sqrt(max(float(v), 0.0))

    def upper_of(x):
        return float((k[:, None] * x.amax(2)).sum() + k0 * x.amax((0, 2)).sum() + (h * x).sum()) * scale

    def lower_of(y, z):
        return float(torch.where(on, h + y + z, torch.inf).amin(1).sum()) * scale

    ar = torch.arange(tp, dtype=torch.float64, device=dev)
    x = (1.0 / (ar + 1.0))[None, None, :] * onf.expand(n, tp, tp)
    y = k[:, None, None] / (tp - ar)[None, :, None] * onf
    z = k0 / (n * (tp - ar))[None, :, None] * onf.expand(n, tp, tp)
    s = _Restarts(p, tolerance)
    a, a0 = (x, y, z), (x, y, z)
    lower, upper = lower_of(y, z), upper_of(x)
    b = step(*a, s.omega)
    s.fp_error = norm(a, b, s.omega)
    if s.stop(lower, upper):
        b = a
    else:
        while True:
            for _ in range(int(p.op_steps)):
                c = s.since + 1.0
                a = tuple(c / (c + 1.0) * (2.0 * v - u) + u0 / (c + 1.0) for u, v, u0 in zip(a, b, a0))
                b = step(*a, s.omega)
                s.since += 1
                s.iteration += 1
            error = norm(a, b, s.omega)
            lower, upper = lower_of(b[1], b[2]), upper_of(b[0])
            if s.stop(lower, upper):
                break
            if s.after_block(error, math.sqrt(float(((a[0] - a0[0]) ** 2).sum())),
                             math.sqrt(float(((a[1] - a0[1]) ** 2).sum() + ((a[2] - a0[2]) ** 2).sum()))):
                a = a0 = b
                b = step(*a, s.omega)
                s.restarted(norm(a, b, s.omega))
    x, y, z = b
    part = torch.zeros_like(x)
    part[:, :t, :t] = x[:, :t, :t]
    y = torch.where(k[:, None, None] > 0, y / k[:, None, None], 0.0 * y)
    z = z / k0 if k0 > 0 else 0.0 * z
    return lower, upper_of(part), s.iteration, *(v[:, :t, :t].cpu().numpy() for v in (x, y, z))


def exact(case, seed):
    kind = case["kind"]
    tolerance = TOLERANCE[case["precision"]]
    if kind.startswith("qubo"):
        inst = _qubo(seed, case["n"], case["m"], ordered=kind != "qubo_warm")
        warm = _warm_point(inst, seed) if kind == "qubo_warm" else None
        lower, upper, _, x, y = _exact_qubo(inst, _praq_parameters(case), tolerance, warm)
        if kind == "qubo_warm":
            return {"x": x, "y": y, "iterations": None}
        return {"lower": lower, "upper": upper, "iterations": None, "status": None, "x": x}
    if kind.startswith("jrp"):
        inst = jrp_demand(seed, case["items"], case["periods"])
        lower, upper, _, x, y, z = _exact_jrp(inst, _pria_parameters(case), tolerance)
        out = {"upper": upper, "lower": lower, "iterations": None}
        if kind == "jrp_oneshot" or case["solution"]:
            out |= {"x": x, "y": y, "z": z}
        return out
    qubos, jrps = _batch_instances(case, seed)
    q = [_exact_qubo(i, _praq_parameters(case), tolerance) for i in qubos]
    j = [_exact_jrp(i, _pria_parameters(case), tolerance) for i in jrps]
    return {"x%d" % k: r[3] for k, r in enumerate(q)} | {
        "qubo_bounds": np.array([r[:2] for r in q]), "qubo_iterations": None,
        "jrp_bounds": np.array([r[:2] for r in j]), "jrp_iterations": None}
