"""Timed workloads of the game-value solvers, through their public Python API.

Each case is one pass of real use: a capture-tube solve in float32 or in the
exact arithmetic, an 8D contact or square-arena solve, semi-Lagrangian value
iteration and its policy backup, a batch of uneven solves, and the learned
surrogate's training, bulk inference and online queries.  `prepare` makes what
a program holds before the call (solver handles, page-locked result buffers,
networks, inputs), `run` is one pass, `work` the bytes and operations the pass
cannot do without, and `exact` the same outputs in 64-bit arithmetic, in plain
torch.
"""

import math
from pathlib import Path
import sys

import numpy as np
import torch

_ROOT = Path(__file__).resolve().parents[1] / "pursuit-evasion-core_b200"
if str(_ROOT) not in sys.path:
    sys.path.insert(0, str(_ROOT))

# reversible_free_a3: (speed_min, speed_max, max_curvature) of the two cars
PURSUER = (-1.0, 2.0, 1.0)
EVADER = (-0.5, 1.0, 2.0)
EXACT_CELL_STAGES = 1.2e10  # above this `exact` would take too long


# ---------------------------------------------------------------------------
# the cases
def _tube(name, precision, grid, steps):
    positions, headings, p_speeds, e_speeds, extent = grid
    return {"name": name, "family": "tube", "precision": precision,
            "positions": positions, "headings": headings, "p_speeds": p_speeds,
            "e_speeds": e_speeds, "extent": extent, "steps": steps}


def _world(name, fast, game, boundary, grid, steps):
    positions, headings, p_speeds, e_speeds, extent = grid
    return {"name": name, "family": "world", "fast": fast, "game": game,
            "boundary": boundary, "positions": positions, "headings": headings,
            "p_speeds": p_speeds, "e_speeds": e_speeds, "extent": extent, "steps": steps}


def _semilag(name, mode, policy, grid, steps):
    positions, headings, p_speeds, e_speeds, extent = grid
    return {"name": name, "family": "semilag", "mode": mode, "policy": policy,
            "positions": positions, "headings": headings, "p_speeds": p_speeds,
            "e_speeds": e_speeds, "extent": extent, "steps": steps}


def _learned(name, use, grid, rows, steps):
    positions, headings, p_speeds, e_speeds, extent = grid
    return {"name": name, "family": "learned", "use": use, "positions": positions,
            "headings": headings, "p_speeds": p_speeds, "e_speeds": e_speeds,
            "extent": extent, "rows": rows, "steps": steps}


def listed():
    return [
        # the smoke-test solve of the README grid: launches and latency count
        _tube("tube32_smoke", "float32", (17, 12, 7, 7, 4.0), 16),
        # the headline 89M-cell table, float32 arithmetic: its first frames
        _tube("tube32_full", "float32", (65, 48, 21, 21, 8.0), 60),
        # the default (reference-exact) arithmetic on the coarse table that
        # warm starts are trained on
        _tube("tube64_coarse", "float64", (33, 24, 11, 11, 8.0), 60),
        # the headline table in the exact arithmetic
        _tube("tube64_full", "float64", (65, 48, 21, 21, 8.0), 12),
        # the default 8D solve: square arena with the pursuer's avoid floor
        _world("world_square", False, "square", "linear", (9, 8, 7, 7, 3.5), 10),
        # the 58M-cell rectangle-contact game on the fast stage
        _world("world_contact_fast", True, "contact", "linear", (11, 9, 7, 7, 3.0), 15),
        # minimum-time value iteration on the headline grid from a warm start
        _semilag("semilag_value", "min_time", False, (65, 48, 21, 21, 8.0), 12),
        # scheme="semi_lagrangian" on the coarse grid: tube backups with
        # arrival times, the policy recorded with the last one
        _semilag("semilag_policy", "tube", True, (33, 24, 11, 11, 8.0), 24),
        # uneven solves in one persistent launch, the default arithmetic
        {"name": "batch", "family": "batch", "precision": "float64", "set": 5, "count": 4,
         "min_steps": 20, "max_steps": 60},
        # surrogate training on node samples of a table
        _learned("learned_train", "train", (33, 24, 11, 11, 8.0), 8192, 256),
        # the surrogate's prediction on every node of a grid (warm start)
        _learned("learned_nodes", "nodes", (41, 30, 13, 13, 8.0), 131072, 1),
        # an online query of a few hundred states: the smallest call
        _learned("learned_query", "query", (65, 48, 21, 21, 8.0), 1000, 1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid5(rng, cells):
    """A relative grid of about `cells` states, odd sizes among them."""
    while True:
        g = (rng.randint(13, 65), rng.randint(8, 48), rng.randint(5, 21), rng.randint(5, 21))
        n = g[0] ** 2 * g[1] * g[2] * g[3]
        if 0.7 * cells < n < 1.4 * cells:
            return g + (rng.choice([4.0, 6.0, 8.0]),)


def _grid8(rng, cells):
    while True:
        g = (rng.randint(5, 11), rng.randint(4, 10), rng.randint(3, 7), rng.randint(3, 7))
        n = g[0] ** 4 * g[1] ** 2 * g[2] * g[3]
        if 0.6 * cells < n < 1.6 * cells:
            return g + (rng.choice([3.0, 3.25, 3.5]),)


def draw(rng):
    family = rng.choice(["tube32", "tube64", "world", "semilag", "batch", "learned"])
    if family in ("tube32", "tube64"):
        cells = _log(rng, 1.0e5, 5.0e7)
        steps = max(2, min(60, int((1.6e9 if family == "tube32" else 4.0e8) / cells)))
        c = _tube("", "float32" if family == "tube32" else "float64", _grid5(rng, cells), steps)
    elif family == "world":
        cells = _log(rng, 1.0e6, 4.0e7)
        fast = rng.random() < 0.5
        c = _world("", fast, rng.choice(["square", "contact"]),
                   rng.choice(["linear", "legacy_signed"]), _grid8(rng, cells),
                   max(2, min(24, int(1.6e8 / cells))))
    elif family == "semilag":
        if rng.random() < 0.5:
            cells = _log(rng, 2.0e6, 5.0e7)
            c = _semilag("", "min_time", False, _grid5(rng, cells),
                         max(3, min(24, int(3.0e8 / cells))))
        else:
            cells = _log(rng, 5.0e5, 5.0e6)
            c = _semilag("", "tube", True, _grid5(rng, cells), rng.randint(6, 24))
    elif family == "batch":
        c = {"family": "batch", "precision": rng.choice(["float64", "float32"]),
             "set": rng.randint(0, 10 ** 6), "count": rng.randint(2, 6),
             "min_steps": rng.randint(4, 12), "max_steps": rng.randint(16, 32)}
    else:
        use = rng.choice(["train", "nodes", "query"])
        grid = _grid5(rng, _log(rng, 5.0e5, 8.0e6))
        rows = {"train": 2048 * rng.randint(1, 4), "nodes": 1 << rng.randint(13, 17),
                "query": _log(rng, 1, 8192)}[use]
        c = _learned("", use, grid, rows, rng.randint(32, 128) if use == "train" else 1)
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# shared pieces of prepare / exact
def _physics(seed):
    """Accelerations and capture radius of one problem (the ranges of the
    batched workload)."""
    rng = np.random.default_rng(seed)
    return (float(rng.uniform(1.5, 4.0)), float(rng.uniform(1.5, 4.0)),
            float(rng.uniform(0.3, 0.8)))


def _config(physics):
    from pursuit_evasion_b200.reversible.model import ReversibleConfig, VehicleLimits

    acc_p, acc_e, radius = physics
    return ReversibleConfig(
        name="reversible_free",
        pursuer=VehicleLimits(PURSUER[0], PURSUER[1], acc_p, PURSUER[2]),
        evader=VehicleLimits(EVADER[0], EVADER[1], acc_e, EVADER[2]),
        capture_radius=radius)


def _pinned(count):
    """A page-locked float32 result buffer."""
    return torch.empty(count, dtype=torch.float32, pin_memory=True).numpy()


def _footprints(seed):
    rng = np.random.default_rng([seed, 8])
    return tuple((float(rng.uniform(0.4, 0.9)), float(rng.uniform(0.25, 0.5)))
                 for _ in range(2))


def _shape5(c):
    return (c["p_speeds"], c["e_speeds"], c["headings"], c["positions"], c["positions"])


def _relative_grid(c):
    from pursuit_evasion_b200.reversible.free_dp import RelativeGrid

    return RelativeGrid(c["positions"], c["headings"], c["p_speeds"], c["e_speeds"],
                        c["extent"])


def _axes5(c, device, dtype):
    """Broadcastable vP, vE, psi, y, x."""
    def axis(lo, hi, n, k, periodic=False):
        a = torch.arange(n, device=device, dtype=torch.float64)
        a = lo + a * ((hi - lo) / (n if periodic else n - 1))
        shape = [1] * 5
        shape[k] = n
        return a.to(dtype).reshape(shape)
    w = c["extent"]
    return (axis(PURSUER[0], PURSUER[1], c["p_speeds"], 0),
            axis(EVADER[0], EVADER[1], c["e_speeds"], 1),
            axis(-math.pi, math.pi, c["headings"], 2, True),
            axis(-w, w, c["positions"], 3), axis(-w, w, c["positions"], 4))


def _table(c, seed, dtype=torch.float32):
    """A smooth capture-time-like field 1 - exp(-T) over the relative grid."""
    _, _, radius = _physics(seed)
    rng = np.random.default_rng([seed, 5])
    k = rng.uniform(0.1, 0.4, size=4).tolist()
    vp, ve, psi, y, x = _axes5(c, "cuda", dtype)
    d = torch.clamp(torch.hypot(x, y) - radius, min=0.0)
    rate = 1.2 + k[0] * torch.cos(psi) + k[1] * vp - k[2] * ve
    lead = 1.0 + k[3] * x / (1.0 + torch.hypot(x, y))
    return 1.0 - torch.exp(-(d * lead) / torch.clamp(rate, min=0.4))


def _states(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand(c["rows"], 5, generator=g, device="cuda")
    w = c["extent"]
    lo = torch.tensor([-w, -w, -math.pi, PURSUER[0], EVADER[0]], device="cuda")
    hi = torch.tensor([w, w, math.pi, PURSUER[1], EVADER[1]], device="cuda")
    return (lo + u * (hi - lo)).contiguous()


def _batch_solves(c, seed):
    """Grid sizes and step counts from the case, physics from the seed."""
    rng = np.random.default_rng(c["set"])
    out = []
    for k in range(c["count"]):
        grid = dict(positions=int(rng.integers(17, 50)), headings=int(rng.integers(12, 37)),
                    p_speeds=int(rng.integers(7, 16)), e_speeds=int(rng.integers(7, 16)),
                    extent=4.0)
        steps = int(rng.integers(c["min_steps"], c["max_steps"] + 1))
        out.append((grid, steps, _physics([seed, k])))
    return out


# ---------------------------------------------------------------------------
def prepare(case, seed):
    c, s = case, {"case": case}
    family = c["family"]
    if family == "tube":
        from pursuit_evasion_b200.reversible.relative_solver import RelativeSolver

        solver = RelativeSolver(_config(_physics(seed)), _relative_grid(c),
                                local_precision=c["precision"])
        s["solver"] = solver
        s["goals"] = _goals(solver.cfl_dt_limit, c["steps"], 4)
        s["field"] = _pinned(solver.cells)
        if c["precision"] == "float64":
            s["arrival"] = _pinned(solver.cells)
    elif family == "world":
        from pursuit_evasion_b200.reversible.world_dp import WorldGrid, WorldSolver

        grid = WorldGrid(c["positions"], c["headings"], c["p_speeds"], c["e_speeds"],
                         c["extent"])
        solver = WorldSolver(_config(_physics(seed)), grid, speed_boundary=c["boundary"],
                             avoid=c["game"] == "square", fast=c["fast"])
        s["solver"] = solver
        s["goals"] = _goals(solver.dt_limit, c["steps"], 2)
        s["bodies"] = _footprints(seed)
        s["field"] = _pinned(solver.cells)
        if not c["fast"]:
            s["arrival"] = _pinned(solver.cells)
    elif family == "semilag":
        from pursuit_evasion_b200.reversible.semilag import SemiLagrangianSolver

        s["solver"] = SemiLagrangianSolver(_config(_physics(seed)), _relative_grid(c),
                                           mode=c["mode"])
        if c["mode"] == "min_time":
            s["initial"] = _table(c, seed)
            s["value"] = torch.empty_like(s["initial"])
    elif family == "batch":
        from pursuit_evasion_b200.batch import BatchSolve, BatchSolver
        from pursuit_evasion_b200.reversible.free_dp import RelativeGrid
        from pursuit_evasion_b200.reversible.relative_solver import cfl_limit

        solves = []
        for grid, steps, physics in _batch_solves(c, seed):
            config, grid = _config(physics), RelativeGrid(**grid)
            solves.append(BatchSolve(config, grid, steps * cfl_limit(config, grid)))
        s["solver"] = BatchSolver(solves, local_precision=c["precision"])
    else:
        from pursuit_evasion_b200.learned.mlp import ValueMLP
        from pursuit_evasion_b200.learned.train import RelativeNodeSampler

        config, grid = _config(_physics(seed)), _relative_grid(c)
        rows = max(128, (c["rows"] + 127) // 128 * 128)
        s["net"] = ValueMLP(6, seed=seed % 2 ** 31, max_batch=rows)
        s["config"] = config
        if c["use"] == "train":
            s["sampler"] = RelativeNodeSampler(config, grid, _table(c, seed).reshape(-1))
            s["seed"] = seed
        elif c["use"] == "nodes":
            s["sampler"] = RelativeNodeSampler(config, grid)
            s["out"] = torch.empty(grid.states, device="cuda")
        else:
            s["states"] = _states(c, seed)
    torch.cuda.synchronize()
    return s


def _goals(limit, steps, frames):
    """`frames` output times that end after `steps` steps of the CFL limit."""
    counts = sorted({max(1, round(steps * (k + 1) / frames)) for k in range(frames)})
    return [limit * n for n in counts]


def run(state):
    c = state["case"]
    family = c["family"]
    if family == "tube":
        s = state["solver"]
        s.initialize()
        for goal in state["goals"]:
            s.advance(goal)
        out = {"field": s.field(state["field"])}
        if "arrival" in state:
            out["arrival"] = s.arrival(state["arrival"])
        return out
    if family == "world":
        s = state["solver"]
        if c["game"] == "contact":
            s.init_contact(*state["bodies"])
        else:
            s.init_square()
        for goal in state["goals"]:
            s.advance(goal)
        out = {"field": s.field(state["field"])}
        if "arrival" in state:
            out["arrival"] = s.arrival(state["arrival"])
        return out
    if family == "semilag":
        s = state["solver"]
        if c["mode"] == "min_time":
            s.initialize_device(state["initial"].data_ptr())
            s.iterate(c["steps"], tol=1e-7, check_every=5)
            s.value_to_device(state["value"].data_ptr())
            return {"value": state["value"]}
        s.initialize()
        s.track_arrival()
        for _ in range(c["steps"] - 1):
            s.backup()
        s.backup(with_policy=c["policy"])
        out = {"value": s.value(), "arrival": s.arrival()}
        if c["policy"]:
            out["policy_p"], out["policy_e"] = s.policy()
        return out
    if family == "batch":
        s = state["solver"]
        s.initialize()
        s.run()
        s.synchronize()
        return [s.field(i) for i in range(len(s))]
    from pursuit_evasion_b200.learned.train import predict_nodes, predict_states, train

    net = state["net"]
    if c["use"] == "train":
        losses, _ = train(net, state["sampler"], samples=c["rows"] * c["steps"] // 2, epochs=2,
                          batch=c["rows"], seed=state["seed"])
        return {"losses": losses, "weights": net.w, "biases": net.b,
                "head": [net.w_out, net.b_out]}
    if c["use"] == "nodes":
        return predict_nodes(net, state["sampler"], state["out"], chunk=c["rows"])
    return predict_states(net, state["config"], c["extent"], state["states"])


# ---------------------------------------------------------------------------
def work(case):
    c = case
    if c["family"] == "batch":
        stages = sum(2 * steps * math.prod((g["p_speeds"], g["e_speeds"], g["headings"],
                                            g["positions"], g["positions"]))
                     for g, steps, _ in _batch_solves(c, 0))
        return {"bytes": 10 * stages, "flops": 110 * stages}
    if c["family"] == "learned":
        macs = 6 * 256 + 3 * 256 * 256 + 256  # per row
        weights = 4 * macs
        if c["use"] == "train":
            rows = c["rows"] * (c["steps"] // 2) * 2
            # a sampled value and index per row; the weights, their gradients
            # and both moments once per step
            return {"bytes": 12 * rows + 6 * weights * c["steps"], "flops": 6 * macs * rows}
        rows = math.prod(_shape5(c)) if c["use"] == "nodes" else c["rows"]
        per_row = 4 if c["use"] == "nodes" else 24
        return {"bytes": per_row * rows + weights, "flops": 2 * macs * rows}
    if c["family"] == "world":
        cells = (c["positions"] ** 4 * c["headings"] ** 2 * c["p_speeds"] * c["e_speeds"])
        return {"bytes": 20 * cells * c["steps"], "flops": 2 * 170 * cells * c["steps"]}
    cells = math.prod(_shape5(c))
    if c["family"] == "semilag":
        # about 13 interpolated action pairs of 37 operations per backup
        return {"bytes": 8 * cells * c["steps"], "flops": 13 * 37 * cells * c["steps"]}
    return {"bytes": 20 * cells * c["steps"], "flops": 2 * 110 * cells * c["steps"]}


# ---------------------------------------------------------------------------
# the same in 64-bit arithmetic
def _slopes(v, dim, h, end):
    """(left, right) ENO2 slopes.  `end`: "wrap", "inward" (one-sided at the
    end nodes) or "ghost" (values pushed away from zero beyond the ends)."""
    n = v.shape[dim]
    at = lambda k: v.narrow(dim, k, 1)  # noqa: E731
    if end == "wrap":
        e = torch.cat([v.narrow(dim, n - 2, 2), v, v.narrow(dim, 0, 2)], dim)
    elif end == "ghost":
        a, da = at(0), (at(1) - at(0)).abs() * torch.sign(at(0))
        b, db = at(n - 1), (at(n - 1) - at(n - 2)).abs() * torch.sign(at(n - 1))
        e = torch.cat([a + 2 * da, a + da, v, b + db, b + 2 * db], dim)
    else:
        e = torch.cat([at(0), at(0), v, at(n - 1), at(n - 1)], dim)
    d1 = (e.narrow(dim, 1, n + 3) - e.narrow(dim, 0, n + 3)) / h  # edges -3/2 .. n+1/2
    d2 = (d1.narrow(dim, 1, n + 2) - d1.narrow(dim, 0, n + 2)) / h  # nodes -1 .. n
    del e
    if end == "inward":
        d2.narrow(dim, 1, 1).copy_(d2.narrow(dim, 2, 1))
        d2.narrow(dim, n, 1).copy_(d2.narrow(dim, n - 1, 1))
    a, b = d2.narrow(dim, 0, n + 1), d2.narrow(dim, 1, n + 1)
    pick = torch.where(a.abs() < b.abs(), a, b) * (0.5 * h)
    d1 = d1.narrow(dim, 1, n + 1)
    lo = (d1 + pick).narrow(dim, 0, n).contiguous()
    hi = (d1 - pick).narrow(dim, 1, n).contiguous()
    if end == "inward":
        lo.narrow(dim, 0, 1).copy_(d1.narrow(dim, 1, 1))
        hi.narrow(dim, 0, 1).copy_(d1.narrow(dim, 1, 1))
        lo.narrow(dim, n - 1, 1).copy_(d1.narrow(dim, n - 1, 1))
        hi.narrow(dim, n - 1, 1).copy_(d1.narrow(dim, n - 1, 1))
    return lo, hi


def _speed_term(g, dim, acc, minimise):
    """min (max) over the acceleration of a * gradient; none outward at a bound."""
    n = g.shape[dim]
    shape = [1] * g.dim()
    shape[dim] = n
    lo = torch.full((n,), -acc, device=g.device, dtype=g.dtype)
    hi = torch.full((n,), acc, device=g.device, dtype=g.dtype)
    lo[0] = 0
    hi[n - 1] = 0
    a, b = lo.reshape(shape) * g, hi.reshape(shape) * g
    return torch.minimum(a, b) if minimise else torch.maximum(a, b)


def _exact_tube(c, physics, steps):
    acc_p, acc_e, radius = physics
    vp, ve, psi, y, x = _axes5(c, "cuda", torch.float64)
    n, w = c["positions"], c["extent"]
    h = [(PURSUER[1] - PURSUER[0]) / (c["p_speeds"] - 1),
         (EVADER[1] - EVADER[0]) / (c["e_speeds"] - 1), 2 * math.pi / c["headings"],
         2 * w / (n - 1), 2 * w / (n - 1)]
    top_p, top_e = max(map(abs, PURSUER[:2])), max(map(abs, EVADER[:2]))
    turn = top_p * PURSUER[2] * w
    dt = 0.8 / ((top_p + top_e + turn) / h[4] + (top_e + turn) / h[3]
                + (top_p * PURSUER[2] + top_e * EVADER[2]) / h[2] + acc_p / h[0]
                + acc_e / h[1])
    wp, we = vp.abs() * PURSUER[2], ve.abs() * EVADER[2]
    bx, by = ve * torch.cos(psi) - vp, ve * torch.sin(psi)

    def rate(v):
        grad, total = {}, 0
        alpha = {0: acc_p, 1: acc_e, 2: wp + we, 3: by.abs() + wp * x.abs(),
                 4: bx.abs() + wp * y.abs()}
        for k in range(5):
            lo, hi = _slopes(v, k, h[k], "wrap" if k == 2 else "inward")
            total = total + 0.5 * alpha[k] * (hi - lo)
            g = 0.5 * (lo + hi)
            if k < 2:
                total = total + _speed_term(g, k, acc_p if k == 0 else acc_e, k == 0)
            else:
                grad[k] = g
        total = total + bx * grad[4] + by * grad[3]
        total = total - wp * (y * grad[4] - x * grad[3] - grad[2]).abs() + we * grad[2].abs()
        return torch.clamp(total, max=0.0)

    v = (torch.hypot(x, y) - radius).expand(_shape5(c)).contiguous()
    for _ in range(steps):
        mid = v + dt * rate(v)
        v = 0.5 * (v + mid + dt * rate(mid))
    return v


def _exact_world(c, physics, bodies):
    acc_p, acc_e, radius = physics
    n, nh, w = c["positions"], c["headings"], c["extent"]
    shape = (n, n, nh, c["p_speeds"], n, n, nh, c["e_speeds"])

    def axis(k, lo, step):
        a = lo + step * torch.arange(shape[k], device="cuda", dtype=torch.float64)
        return a.reshape([shape[k] if j == k else 1 for j in range(8)])

    dx, dh = 2 * w / (n - 1), 2 * math.pi / nh
    hv = [(PURSUER[1] - PURSUER[0]) / (shape[3] - 1), (EVADER[1] - EVADER[0]) / (shape[7] - 1)]
    h = [dx, dx, dh, hv[0], dx, dx, dh, hv[1]]
    low = [-w, -w, -math.pi, PURSUER[0], -w, -w, -math.pi, EVADER[0]]
    q = [axis(k, low[k], h[k]) for k in range(8)]
    top_p, top_e = max(map(abs, PURSUER[:2])), max(map(abs, EVADER[:2]))
    dt = 0.8 / (2 * (top_p + top_e) / dx + (top_p * PURSUER[2] + top_e * EVADER[2]) / dh
                + acc_p / hv[0] + acc_e / hv[1])
    avoid = None
    if c["game"] == "square":
        arena = 3.0
        avoid = torch.maximum(q[0].abs(), q[1].abs()) - arena + 1e-6
        target = torch.minimum(arena - torch.maximum(q[4].abs(), q[5].abs()),
                               torch.hypot(q[0] - q[4], q[1] - q[5]) - radius)
        v = torch.maximum(target, avoid)
    else:
        turn = q[6] - q[2]
        ca, sa = torch.cos(turn).abs(), torch.sin(turn).abs()
        d0, d1 = q[4] - q[0], q[5] - q[1]
        v = None
        for heading, own, other in ((q[2], *bodies), (q[6], *bodies[::-1])):
            cs, sn = torch.cos(heading), torch.sin(heading)
            gx = (d0 * cs + d1 * sn).abs() - own[0] / 2 - (other[0] * ca + other[1] * sa) / 2
            gy = (d1 * cs - d0 * sn).abs() - own[1] / 2 - (other[0] * sa + other[1] * ca) / 2
            gap = torch.maximum(gx, gy)
            v = gap if v is None else torch.maximum(v, gap)
    v = v.expand(shape).contiguous()
    wp, we = q[3].abs() * PURSUER[2], q[7].abs() * EVADER[2]
    flow = {0: q[3] * torch.cos(q[2]), 1: q[3] * torch.sin(q[2]),
            4: q[7] * torch.cos(q[6]), 5: q[7] * torch.sin(q[6])}
    speed_end = "inward" if c["boundary"] == "linear" else "ghost"

    def rate(v):
        total = torch.zeros_like(v)
        for k in range(8):
            end = "wrap" if k in (2, 6) else speed_end if k in (3, 7) else "ghost"
            lo, hi = _slopes(v, k, h[k], end)
            g = 0.5 * (lo + hi)
            alpha = {2: wp, 3: acc_p, 6: we, 7: acc_e}.get(k)
            total += 0.5 * (flow[k].abs() if alpha is None else alpha) * (hi - lo)
            if k in flow:
                total += flow[k] * g
            elif k == 2:
                total -= wp * g.abs()
            elif k == 6:
                total += we * g.abs()
            else:
                total += _speed_term(g, k, acc_p if k == 3 else acc_e, k == 3)
        return total

    for _ in range(c["steps"]):
        mid = v + dt * rate(v)
        new = torch.minimum(0.5 * (v + mid + dt * rate(mid)), v)
        v = new if avoid is None else torch.maximum(new, avoid)
    return v


def _arc(v, a, k, dt, lo, hi):
    """Final speed, turn and the displacement of a held command, car frame."""
    target = hi if a >= 0 else lo
    active = min(dt, max(0.0, (target - v) / a)) if a else dt
    end = min(max(v + a * dt, lo), hi)
    dist = v * active + 0.5 * a * active * active + end * (dt - active)
    turn = k * dist
    chord = dist if abs(turn) < 1e-12 else dist * math.sin(0.5 * turn) / (0.5 * turn)
    return end, turn, chord


def _exact_semilag_tube(c, physics):
    acc_p, acc_e, radius = physics
    n, w, nh = c["positions"], c["extent"], c["headings"]
    dx, dh = 2 * w / (n - 1), 2 * math.pi / nh
    hv = [(PURSUER[1] - PURSUER[0]) / (c["p_speeds"] - 1),
          (EVADER[1] - EVADER[0]) / (c["e_speeds"] - 1)]
    top_p, top_e = max(map(abs, PURSUER[:2])), max(map(abs, EVADER[:2]))
    turn = top_p * PURSUER[2] * w
    dt = 1.0 / max((top_p + top_e + turn) / dx, (top_p * PURSUER[2] + top_e * EVADER[2]) / dh,
                   acc_p / hv[0], acc_e / hv[1])
    psi, y, x = (t.reshape(t.shape[2:]) for t in _axes5(c, "cuda", torch.float64)[2:])
    v = (torch.hypot(x, y) - radius).expand(_shape5(c)).contiguous()
    commands = [(a, k) for a in (-1, 0, 1) for k in (-1, 0, 1)]
    ne = c["e_speeds"]

    def locate(speed, lo, step, count):
        f = (speed - lo) / step
        j = min(max(int(math.floor(f)), 0), count - 2)
        return j, f - j

    def column(values, dtype=torch.float64):
        return torch.tensor(values, device="cuda", dtype=dtype).reshape(-1, 1, 1, 1)

    # per evader command, over its speed levels: node and weight of the final
    # speed, turn, displacement, and the cell's storage offset
    replies = []
    for ea, ek in commands:
        arcs = [_arc(EVADER[0] + ie * hv[1], ea * acc_e, ek * EVADER[2], dt, *EVADER[:2])
                for ie in range(ne)]
        at = [locate(a[0], EVADER[0], hv[1], ne) for a in arcs]
        turns, chords = column([a[1] for a in arcs]), column([a[2] for a in arcs])
        replies.append((column([j for j, _ in at], torch.long).reshape(-1),
                        column([f for _, f in at]), turns,
                        chords * torch.cos(psi + 0.5 * turns),
                        chords * torch.sin(psi + 0.5 * turns)))
    heads = torch.arange(nh, device="cuda").reshape(1, -1, 1, 1)
    slab = torch.arange(ne, device="cuda").reshape(-1, 1, 1, 1) * nh

    def backup(v):
        out = torch.empty_like(v)
        for iv in range(c["p_speeds"]):
            best = v[iv]
            for pa, pk in commands:
                pv, pturn, pchord = _arc(PURSUER[0] + iv * hv[0], pa * acc_p, pk * PURSUER[2],
                                         dt, *PURSUER[:2])
                j, f = locate(pv, PURSUER[0], hv[0], c["p_speeds"])
                row = torch.lerp(v[j], v[j + 1], f)
                worst = None
                for je, we, eturn, ex, ey in replies:
                    field = torch.lerp(row[je], row[je + 1], we).reshape(-1)
                    dxp = x + ex - pchord * math.cos(0.5 * pturn)
                    dyp = y + ey - pchord * math.sin(0.5 * pturn)
                    fx = (math.cos(pturn) * dxp + math.sin(pturn) * dyp + w) / dx
                    fy = (math.cos(pturn) * dyp - math.sin(pturn) * dxp + w) / dx
                    jx = torch.clamp(torch.floor(fx), 0, n - 2)
                    jy = torch.clamp(torch.floor(fy), 0, n - 2)
                    at, wx, wy = (jy * n + jx).long(), fx - jx, fy - jy
                    shift = (eturn - pturn) / dh
                    base = torch.floor(shift)
                    value = 0.0
                    for b, wb in ((0, 1 - (shift - base)), (1, shift - base)):
                        k = at + (slab + (heads + base.long() + b) % nh) * (n * n)
                        top = torch.lerp(field[k], field[k + 1], wx)
                        low = torch.lerp(field[k + n], field[k + n + 1], wx)
                        value = value + wb * torch.lerp(top, low, wy)
                    worst = value if worst is None else torch.maximum(worst, value)
                best = torch.minimum(best, worst)
            out[iv] = best
        return out

    for _ in range(c["steps"]):
        v = backup(v)
    return v


def _exact_net(seed):
    """The surrogate's initial weights, in 64 bits."""
    gen = torch.Generator().manual_seed(seed % 2 ** 31)
    weights, biases, width = [], [], 128
    for layer in range(4):
        bound = 1.0 / math.sqrt(6 if layer == 0 else 256)
        w = (torch.rand(256, width, generator=gen) * 2 - 1) * bound
        weights.append(w[:, :6] if layer == 0 else w)
        biases.append((torch.rand(256, generator=gen) * 2 - 1) * bound)
        width = 256
    weights.append((torch.rand(256, generator=gen) * 2 - 1) / math.sqrt(256))
    return [[t.double().cuda() for t in ts] for ts in (weights, biases)]


def _exact_forward(net, x, y, psi, vp, ve, extent):
    weights, biases = net
    unit = lambda v, car: 2 * (v - car[0]) / (car[1] - car[0]) - 1  # noqa: E731
    a = torch.stack([x / extent, y / extent, torch.cos(psi), torch.sin(psi),
                     unit(vp, PURSUER), unit(ve, EVADER)], -1)
    for w, b in zip(weights, biases):
        a = torch.nn.functional.silu(a @ w.T + b)
    return a @ weights[4]


def exact(case, seed):
    c = case
    if c["family"] == "tube":
        if 2 * c["steps"] * math.prod(_shape5(c)) > EXACT_CELL_STAGES:
            return None
        v = _exact_tube(c, _physics(seed), c["steps"])
        out = {"field": v}
        if c["precision"] == "float64":
            out["arrival"] = None
        return out
    if c["family"] == "world":
        cells = (c["positions"] ** 4 * c["headings"] ** 2 * c["p_speeds"] * c["e_speeds"])
        if 2 * c["steps"] * cells > EXACT_CELL_STAGES:
            return None
        out = {"field": _exact_world(c, _physics(seed), _footprints(seed))}
        if not c["fast"]:
            out["arrival"] = None
        return out
    if c["family"] == "semilag":
        # 81 interpolated successors per cell and backup
        if (c["mode"] != "tube" or math.prod(_shape5(c)) * c["steps"] > 8e7
                or 81 * c["p_speeds"] * c["steps"] > 3e4):
            return None
        out = {"value": _exact_semilag_tube(c, _physics(seed)), "arrival": None}
        if c["policy"]:
            out["policy_p"] = out["policy_e"] = None
        return out
    if c["family"] == "batch":
        solves = _batch_solves(c, seed)
        if sum(2 * steps * math.prod(_shape5(g)) for g, steps, _ in solves) > EXACT_CELL_STAGES:
            return None
        return [_exact_tube(g, physics, steps) for g, steps, physics in solves]
    if c["use"] == "train":
        return None  # a whole training run: thousands of updates follow one another
    net = _exact_net(seed)
    if c["use"] == "query":
        x, y, psi, vp, ve = _states(c, seed).double().unbind(-1)
        return _exact_forward(net, x, y, psi, vp, ve, c["extent"])
    vp, ve, psi, y, x = (t.expand(_shape5(c)).reshape(-1)
                         for t in _axes5(c, "cuda", torch.float64))
    out = torch.empty_like(x)
    for k in range(0, len(x), 1 << 20):
        p = slice(k, k + (1 << 20))
        out[p] = _exact_forward(net, x[p], y[p], psi[p], vp[p], ve[p], c["extent"])
    return out
