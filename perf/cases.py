"""Workloads of the grid symbolic-control library, through its public entry points.

A case names what a program does (`kind`) and the grid it does it on:

  solve     a held problem is solved again and its results are read
  query     a new K-invariance query against a held abstraction: set-up, solve, read
  run       the whole one-shot call (abstraction, query, solve, read)
  batch     many independent instances in one pipelined call
  serve     queries submitted to a held server, and every result waited for
  simulate  closed-loop trajectories under a held problem's controller
  noalloc   the fixpoint over an abstraction the caller holds in device memory

Two model families, both with theta wrapped: `unicycle` (the benchmark
family: one Euler step, quadric safe set, elliptical candidate set) and
`hyperbolic` (the published demo's constraint, 32 Euler substeps, rectangular
candidate set, optionally obstacles).  The seed moves the query (disturbance
bound, safe set, candidate set, obstacles), as successive queries of one
program differ.  Results go to page-locked host memory, as in the benchmark.
"""
from __future__ import annotations

import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "gpu-inner-outer_b200"))

import gsc_b200 as G  # noqa: E402
import gsc_cases as C  # noqa: E402

METHODS = {"auto": G.METHOD_AUTO, "stored": G.METHOD_STORED, "fused": G.METHOD_FUSED}
ARRAYS = (("valid_mask", 1), ("candidate_mask", 1), ("reachable_mask", 1), ("controller", 4), ("reach_step", 4))
# The three grids a server of the benchmark keeps resident, as (n0, n1, n2, n3, ma, mw).
SERVED = ((20, 20, 16, 10, 5, 5), (65, 65, 38, 25, 10, 10), (32, 32, 24, 16, 8, 8))


def _case(name, kind, family, n, m, **more):
    c = {"name": name, "kind": kind, "family": family, "n0": n[0], "n1": n[1], "n2": n[2], "n3": n[3],
         "ma": m[0], "mw": m[1], "eta": 0.0, "obstacles": 0, "method": "auto", "graph": False, "count": 1,
         "steps": 0, "max_iterations": 256}
    c.update(more)
    return c


def listed():
    return [
        # The smallest call: a controller re-synthesised online on a coarse grid.
        _case("small_solve", "solve", "unicycle", (20, 20, 16, 10), (5, 5)),
        # The published demo run, as the reference's one call makes it (eta 0.1 in every dimension).
        _case("demo_run", "run", "hyperbolic", (70, 70, 63, 13), (10, 10), eta=0.1, max_iterations=100),
        # The benchmark's headline grid, re-solved as one CUDA graph.
        _case("scale_solve", "solve", "unicycle", (65, 65, 38, 25), (10, 10), graph=True),
        # The largest grid of the configurations.
        _case("large_solve", "solve", "unicycle", (128, 128, 72, 48), (12, 12), graph=True),
        # A new query on a grid of odd sizes.
        _case("odd_query", "query", "unicycle", (47, 83, 29, 17), (7, 9)),
        # A cluttered map: obstacles make validity differ from safety.
        _case("obstacle_query", "query", "hyperbolic", (45, 41, 30, 9), (8, 7), obstacles=5, max_iterations=100),
        # The reference's own method, asked for by name.
        _case("stored_solve", "solve", "hyperbolic", (48, 40, 31, 12), (8, 8), method="stored", max_iterations=100),
        # More x cells than the bit-sliced rows take: 16-bit stored boxes.
        _case("wide_query", "query", "hyperbolic", (300, 24, 20, 8), (5, 5), max_iterations=100),
        # A sweep over many small models.
        _case("batch_run", "batch", "unicycle", (16, 16, 16, 16), (5, 5), count=32),
        # A burst of queries to a server with three resident models.
        _case("serve_burst", "serve", "unicycle", SERVED[1][:4], SERVED[1][4:], count=15),
        # Monte-Carlo check of a controller.
        _case("simulate", "simulate", "hyperbolic", (35, 35, 32, 7), (5, 5), count=12000, steps=30,
              max_iterations=100),
        # A solve inside a process that owns all device memory.
        _case("noalloc_solve", "noalloc", "hyperbolic", (41, 39, 33, 8), (5, 5), max_iterations=100),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        kind = rng.choice(["solve", "solve", "query", "query", "run", "run", "batch", "serve", "simulate", "noalloc"])
        family = rng.choice(["unicycle", "unicycle", "hyperbolic"])
        method = rng.choice(["auto", "auto", "auto", "stored"]) if kind in ("solve", "query", "run") else "auto"
        hi = (128, 128, 72, 48)
        if method == "stored" or kind in ("noalloc", "simulate"):
            hi = (48, 48, 32, 16)
        n = [_log_int(rng, lo, h) for lo, h in zip((16, 16, 12, 6), hi)]
        if method == "stored" and rng.random() < 0.3:
            n[0] = rng.randint(257, 400)   # rows of 16-bit stored boxes
            n[1:] = [_log_int(rng, 10, 24), _log_int(rng, 8, 20), _log_int(rng, 4, 8)]
            family = "hyperbolic"
        m = [_log_int(rng, 3, 12), _log_int(rng, 3, 12)]
        c = _case("", kind, family, n, m, method=method, graph=rng.random() < 0.5,
                  max_iterations=rng.choice([8, 64, 256]))
        del c["name"]
        if family == "hyperbolic":
            c["obstacles"] = rng.choice([0, 0, rng.randint(1, 8)])
        if kind == "batch":
            c.update(family="unicycle", obstacles=0, count=rng.randint(3, 40), max_iterations=256)
        if kind == "serve":
            c.update(family="unicycle", obstacles=0, count=rng.randint(3, 15))
        if kind == "simulate":
            c.update(family="hyperbolic", obstacles=0, count=_log_int(rng, 200, 100000), steps=rng.randint(5, 40))
        pairs = math.prod(n) * m[0] * m[1]
        limit = {"batch": 1e12, "serve": 1e9, "simulate": 4e7, "noalloc": 2e7}.get(kind, 8e9)
        if pairs > (6e7 if method == "stored" else limit) or pairs < 2e5:
            continue
        if list(C.grid_shape(_model(c))[0]) != n:
            continue   # width / (width / n) rounded up to n + 1
        return c


def _model(case):
    """The grid, inputs and dynamics of a case, with the family's own query."""
    n, m = [case["n%d" % d] for d in range(4)], (case["ma"], case["mw"])
    if case["family"] == "unicycle":
        return C.unicycle_grid_case(tuple(n), m, max_iterations=case["max_iterations"])
    c = C.hyperbolic_demo_case()
    width = [u - lb for lb, u in zip(c["state_lb"], c["state_ub"])]
    c["state_eta"] = [case["eta"] or w / k for w, k in zip(width, n)]
    c["input_eta"] = [(u - lb) / k for lb, u, k in zip(c["input_lb"], c["input_ub"], m)]
    c["max_iterations"] = case["max_iterations"]
    return c


def _query(case, rng):
    """The case's model with a query drawn near the family's own."""
    c = _model(case)
    if case["family"] == "unicycle":
        c["disturbance_half_width"] = [rng.uniform(0.009, 0.011)] * 4
        c["constraint_params"] = [1.0, rng.uniform(0.97, 1.03), rng.uniform(0.95, 1.05), rng.uniform(1.75, 1.85)]
        c["candidate_ellipse"] = [rng.uniform(-0.05, 0.05), rng.uniform(-0.05, 0.05), 1.0, 1.0,
                                  rng.uniform(0.45, 0.55)]
        return c
    c["disturbance_half_width"] = [rng.uniform(0.045, 0.05)] * 4
    c["constraint_params"] = [rng.uniform(3.8, 4.2), 4.0, rng.uniform(15.0, 17.0), 0.0]
    half = rng.uniform(0.75, 0.85)
    c["candidate_lb"][:2] = [-half, -half]
    c["candidate_ub"][:2] = [half, half]
    for _ in range(case["obstacles"]):
        at = rng.uniform(0.0, 2.0 * math.pi)
        x, y, w = 1.7 * math.cos(at), 1.7 * math.sin(at), rng.uniform(0.1, 0.3)
        c["obstacles"].append([x - w, y - w, -C.PI, -0.1, x + w, y + w, C.PI, 1.2])
    return c


_held = {}


def _context():
    if "ctx" not in _held:
        _held["ctx"] = G.Context(0)
    return _held["ctx"]


def _results(sizes):
    """Page-locked result arrays of problems with these many states: one
    buffer per array kind, and each problem's views into them."""
    total = sum(sizes)
    flat = {}
    for k, size in ARRAYS:
        buf = torch.empty(total * size, dtype=torch.uint8, pin_memory=True)
        flat[k] = buf.numpy() if size == 1 else buf.numpy().view(np.uint32)
    views, at = [], 0
    for s in sizes:
        views.append({k: flat[k][at:at + s] for k, _ in ARRAYS})
        at += s
    return flat, views


def _states(c):
    return math.prod(C.grid_shape(c)[0])


def _instances(case, seed):
    """The models and queries of a batch."""
    if case["kind"] == "batch":
        models = [C.random_instance(case["count"], i) for i in range(case["count"])]
        return [C.random_query(c, seed, i, 64, 256) for i, c in enumerate(models)]
    out = []
    for i in range(case["count"]):
        out.append((i % 3, C.random_query(_served(i % 3), seed, i)))
    return out


def _served(k):
    return C.unicycle_grid_case(SERVED[k][:4], SERVED[k][4:])


def _summary(results):
    return np.array([[r["iterations"], r["converged"], r["reachable_states"], r["certified_candidates"],
                      r["candidate_count"], r["valid_count"]] for r in results], dtype=np.int64)


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "batch":
        cases = _instances(case, seed)
        flat, outs = _results([_states(c) for c in cases])
        return {"kind": kind, "ctx": _context(), "cases": cases, "flat": flat, "outs": outs}
    if kind == "serve":
        if "srv" not in _held:
            ctx = _context()
            _held["srv"] = (G.Server(ctx, memory_budget=24 << 30),
                            [G.Abstraction(ctx, _served(k)) for k in range(3)])
        queries = _instances(case, seed)
        flat, outs = _results([_states(q) for _, q in queries])
        srv, models = _held["srv"]
        return {"kind": kind, "srv": srv, "models": models, "queries": queries, "flat": flat, "outs": outs}
    c = _query(case, rng)
    state = {"kind": kind, "ctx": _context(), "case": c, "method": METHODS[case["method"]], "graph": case["graph"]}
    if kind in ("solve", "query", "run"):
        state["flat"], (state["out"],) = _results([_states(c)])
        if kind != "run":
            state["abs"] = G.Abstraction(state["ctx"], c)
        if kind == "solve":
            state["problem"] = G.Problem(state["ctx"], state["abs"], c, state["method"])
        return state
    state["abs"] = G.Abstraction(state["ctx"], c)
    p = G.Problem(state["ctx"], state["abs"], c, G.METHOD_AUTO)
    if kind == "simulate":
        p.solve()
        gen = np.random.default_rng(seed)
        lo = [-0.8, -0.8, -math.pi, 0.0]
        hi = [0.8, 0.8, math.pi, 1.0]
        state.update(problem=p, x0=gen.uniform(lo, hi, size=(case["count"], 4)), steps=case["steps"], seed=seed)
        return state
    # noalloc: the abstraction, masks and outputs in the caller's device memory.
    mn, mx, ok = p.export_abstraction()
    r = p.read()
    p.close()
    dev = torch.device("cuda", 0)
    state.update(shape=r["shape"], inputs=r["inputs"], max_iterations=c["max_iterations"])
    state["in"] = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).to(dev)
                   for a in (mn, mx, ok, r["valid_mask"], r["candidate_mask"])]
    states = _states(c)
    state["outputs"] = [torch.empty(states, dtype=t, device=dev) for t in (torch.uint8, torch.int32, torch.int32)]
    return state


def run(s):
    kind = s["kind"]
    if kind == "solve":
        s["problem"].solve(graph=s["graph"])
        return [s["flat"], _summary([s["problem"].read(out=s["out"])])]
    if kind == "query":
        p = G.Problem(s["ctx"], s["abs"], s["case"], s["method"])
        p.solve(graph=s["graph"])
        r = p.read(out=s["out"])
        p.close()
        return [s["flat"], _summary([r])]
    if kind == "run":
        return [s["flat"], _summary([G.run_case(s["case"], method=s["method"], graph=s["graph"], out=s["out"])])]
    if kind == "batch":
        return [s["flat"], _summary(G.run_batch(s["ctx"], s["cases"], outs=s["outs"]))]
    if kind == "serve":
        tickets = [s["srv"].submit(s["models"][k], q, out=o) for (k, q), o in zip(s["queries"], s["outs"])]
        return [s["flat"], _summary([s["srv"].wait(t) for t in tickets])]
    if kind == "simulate":
        r = s["problem"].simulate(s["x0"], s["steps"], s["seed"])
        return [r["trajectories"], r["final_states"], r["steps_done"]]
    summary = G.Result()
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in s["in"] + s["outputs"]]
    st = G.lib().gsc_fixpoint_noalloc((ctypes.c_uint32 * 4)(*s["shape"]), s["inputs"], 2, *ptr[:5],
                                      s["max_iterations"], *ptr[5:], ctypes.byref(summary),
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if st != 0:
        raise G.GscError(st)
    return s["outputs"] + [int(summary.iterations), int(summary.reachable_states),
                           int(summary.certified_candidates)]


def work(case):
    """Results written once (11 bytes a state) and, where the caller hands
    over device arrays, their bytes; one test per (state, input) pair."""
    kind = case["kind"]
    if kind == "batch":
        cases = _instances(case, 1)
    elif kind == "serve":
        cases = [q for _, q in _instances(case, 1)]
    else:
        cases = [_model(case)]
    states = pairs = 0
    for c in cases:
        n, m = C.grid_shape(c)
        states += math.prod(n)
        pairs += math.prod(n) * math.prod(m)
    if kind == "simulate":
        # per substep: two trigonometric values, one wrap and four updates
        sub = case["count"] * case["steps"] * cases[0]["integration_substeps"]
        return {"bytes": 32.0 * case["count"] * (case["steps"] + 3), "flops": 100.0 * sub}
    return {"bytes": 11.0 * states + (9.0 * pairs if kind == "noalloc" else 0.0), "flops": float(pairs)}


# ---- the simulation's values, in plain 64-bit numpy --------------------------------------


def _quantise(lo, hi, lb, eta, n):
    a = np.floor((lo - lb) / eta).astype(np.int64)
    b = np.ceil((hi - lb) / eta).astype(np.int64) - 1
    return np.clip(a, 0, n - 1), np.clip(b, 0, n - 1)


def _plain_controller(c):
    """The lowest satisfied input of every state when it is reached, by the
    backward fixpoint on box counts (hyperbolic family without obstacles)."""
    n, (ma, mw) = C.grid_shape(c)
    lb, ub, eta = (np.array(c["state_" + k]) for k in ("lb", "ub", "eta"))
    centre = [lb[d] + (np.arange(n[d]) + 0.5) * eta[d] for d in range(4)]
    a_in, w_in = (c["input_lb"][d] + (np.arange(k) + 0.5) * c["input_eta"][d] for d, k in ((0, ma), (1, mw)))
    K, T = c["integration_substeps"], c["sample_time"]
    dt, d4 = T / K, c["disturbance_half_width"]
    # grids are [v][theta][y][x]
    x, y = centre[0][None, :], centre[1][:, None]
    p = c["constraint_params"]
    safe2 = (x * x - y * y <= p[0]) & (p[1] * (y * y) - x * x <= p[2])
    shape = (n[3], n[2], n[1], n[0])
    grids = np.meshgrid(*[centre[d] for d in (3, 2, 1, 0)], indexing="ij")

    def inside(lo, hi):
        ok = np.ones(shape, bool)
        for d in range(4):
            ok &= (grids[3 - d] >= lo[d]) & (grids[3 - d] <= hi[d])
        return ok

    valid = inside(c["map_lb"], c["map_ub"]) & safe2[None, None]
    cand = inside(c["candidate_lb"], c["candidate_ub"])
    he = 0.5 * eta
    boxes = []
    for jw in range(mw):
        for ja in range(ma):
            px = np.broadcast_to(centre[0], (n[3], n[2], n[0])).copy()
            py = np.broadcast_to(centre[1], (n[3], n[2], n[1])).copy()
            th, v = list(centre[2]), centre[3].copy()
            for _ in range(K):
                cs = np.array([math.cos(t) for t in th])
                sn = np.array([math.sin(t) for t in th])
                px += dt * (v[:, None] * cs[None, :])[:, :, None]
                py += dt * (v[:, None] * sn[None, :])[:, :, None]
                th = [t + dt * w_in[jw] for t in th]
                th = [t - 2 * C.PI if t >= C.PI else t + 2 * C.PI if t < -C.PI else t for t in th]
                v = v + dt * a_in[ja]
            ok = np.ones(shape, bool)
            lo, hi = [], []
            for d, pos in ((0, px), (1, py)):
                r = (he[d] + T * np.abs(centre[3]) * he[2] + T * he[3] + T * d4[d])[:, None, None]
                ok_d = (pos - r >= lb[d] - 1e-9) & (pos + r <= ub[d] + 1e-9)
                a, b = _quantise(pos - r, pos + r, lb[d], eta[d], n[d])
                grow = (lambda t: t[:, :, None, :]) if d == 0 else (lambda t: t[:, :, :, None])
                ok &= grow(ok_d)
                lo.append(np.broadcast_to(grow(a), shape))
                hi.append(np.broadcast_to(grow(b), shape))
            th, r, span = np.array(th), he[2] + T * d4[2], ub[2] - lb[2]
            wrap = lambda t: t + span * ((t < lb[2]).astype(float) - (t >= ub[2]).astype(float))  # noqa: E731
            a, b = _quantise(wrap(th - r), wrap(th + r), lb[2], eta[2], n[2])
            lo.append(np.broadcast_to(a[None, :, None, None], shape))
            hi.append(np.broadcast_to(b[None, :, None, None], shape))
            r = he[3] + T * d4[3]
            ok &= ((v - r >= lb[3] - 1e-9) & (v + r <= ub[3] + 1e-9))[:, None, None, None]
            a, b = _quantise(v - r, v + r, lb[3], eta[3], n[3])
            lo.append(np.broadcast_to(a[:, None, None, None], shape))
            hi.append(np.broadcast_to(b[:, None, None, None], shape))
            boxes.append((ok & safe2[None, None], lo, hi))

    def table(s):
        t = np.zeros([k + 1 for k in shape], np.int64)
        t[1:, 1:, 1:, 1:] = s.astype(np.int64).cumsum(0).cumsum(1).cumsum(2).cumsum(3)
        return t

    def count(t, lo, hi, z0, z1):
        total = 0
        for m in range(16):
            i = [lo[d] if (m >> d) & 1 else hi[d] + 1 for d in range(4)]
            i[2] = z0 if (m >> 2) & 1 else z1
            total = total + (-1) ** bin(m).count("1") * t[i[3], i[2], i[1], i[0]]
        return total

    def box_count(t, lo, hi):
        seam = lo[2] > hi[2]
        first = count(t, lo, hi, lo[2], np.where(seam, n[2], hi[2] + 1))
        return first + np.where(seam, count(t, lo, hi, 0 * lo[2], hi[2] + 1), 0)

    unsafe = table(np.broadcast_to(~safe2[None, None], shape))
    vtab = table(valid)
    keep = [ok & (box_count(unsafe, lo, hi) == 0) & (box_count(vtab, lo, hi) > 0) for ok, lo, hi in boxes]
    reach = cand.copy()
    controller = np.full(shape, 0xFFFFFFFF, np.int64)
    certified = 0
    for _ in range(c["max_iterations"]):
        left = table(valid & ~reach)
        open_ = valid & (controller == 0xFFFFFFFF)
        before = reach.copy()
        for j, (_, lo, hi) in enumerate(boxes):
            hit = open_ & keep[j]
            at = np.nonzero(hit)
            hit[at] = box_count(left, [q[at] for q in lo], [q[at] for q in hi]) == 0
            controller[hit] = j
            open_ &= ~hit
            reach |= hit
        done = ((controller != 0xFFFFFFFF) & cand).sum()
        if done == cand.sum() or (done == certified and (before == reach).all()):
            break
        certified = done
    return controller.reshape(-1)


def _philox(c0, c1, seed):
    """Philox4x32-10 (Salmon, Moraes, Dror and Shaw, SC 2011) of (c0, c1, 0, 0) keyed by the seed."""
    u, low = np.uint64, np.uint64(0xFFFFFFFF)
    c = [np.broadcast_to(np.asarray(v, u), np.shape(c1)) for v in (c0, c1, 0, 0)]
    k = [u(seed & 0xFFFFFFFF), u((seed >> 32) & 0xFFFFFFFF)]
    for _ in range(10):
        p0, p1 = u(0xD2511F53) * c[0], u(0xCD9E8D57) * c[2]
        c = [(p1 >> u(32)) ^ c[1] ^ k[0], p1 & low, (p0 >> u(32)) ^ c[3] ^ k[1], p0 & low]
        k = [(k[0] + u(0x9E3779B9)) & low, (k[1] + u(0xBB67AE85)) & low]
    return c


def exact(case, seed):
    if case["kind"] != "simulate" or case["obstacles"]:
        return None
    c = _query(case, random.Random(seed))
    n, (ma, mw) = C.grid_shape(c)
    K, count, steps = c["integration_substeps"], case["count"], case["steps"]
    if math.prod(n) * ma * mw > 7e6 or count * steps * K > 1.2e7:
        return None   # more than about 20 seconds
    controller = _plain_controller(c)
    lb, eta = np.array(c["state_lb"]), np.array(c["state_eta"])
    strides = np.array([1, n[0], n[0] * n[1], n[0] * n[1] * n[2]])
    half = np.array(c["disturbance_half_width"])
    gen = np.random.default_rng(seed)
    x = gen.uniform([-0.8, -0.8, -math.pi, 0.0], [0.8, 0.8, math.pi, 1.0], size=(count, 4))
    traj = np.zeros((count, steps + 1, 4))
    traj[:, 0] = x
    ids, last = np.arange(count), x.copy()
    dt = c["sample_time"] / K
    for step in range(steps):
        s = x.copy()
        s[:, 2] = np.arctan2(np.sin(s[:, 2]), np.cos(s[:, 2]))
        cell = np.clip(np.rint((s - lb) / eta).astype(np.int64), 0, np.array(n) - 1)
        j = controller[cell @ strides]
        go = j < ma * mw
        x, j, ids = x[go], j[go], ids[go]
        if not len(ids):
            break
        acc = c["input_lb"][0] + (j % ma + 0.5) * c["input_eta"][0]
        omega = c["input_lb"][1] + (j // ma + 0.5) * c["input_eta"][1]
        for sub in range(K):
            draws = []
            for part in (0, 1):
                r = _philox(2 * (step * K + sub) + part, ids.astype(np.uint64), seed)
                for a, b in ((r[0], r[1]), (r[2], r[3])):
                    draws.append(((a >> np.uint64(5)) * 67108864.0 + (b >> np.uint64(6))) / 9007199254740992.0)
            w = [-half[d] + 2 * half[d] * draws[d] for d in range(4)]
            f = [x[:, 3] * np.cos(x[:, 2]), x[:, 3] * np.sin(x[:, 2]), omega, acc]
            x = np.stack([x[:, d] + dt * (f[d] + w[d]) for d in range(4)], axis=1)
            x[:, 2] = np.arctan2(np.sin(x[:, 2]), np.cos(x[:, 2]))
        traj[ids, step + 1] = x
        last[ids] = x
    return [traj, last, None]
