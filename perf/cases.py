"""The work that a user of the solver has it do, through the public Python entry points.

Every case is one kind of call over graphs of one family.  A pass makes several
calls (or one call over several graphs), because an exact search's time depends
on the graph: a case then stands for its sizes and not for one lucky tree.

Kinds:
  plain    `vcgpu.solve` on one host graph after another, MVC or PVC: the
           drop-in for the reference's one launch per graph
  batch    `vcgpu.solve_batch` over one packed arena of host arrays
  device   the same over an arena whose rows are already on the GPU
  served   one session of `vcgpu.Server`: open, submit a burst, take the
           results as they finish, close
  bounds   the two upper-bound heuristics, `vcgpu.remove_max_ub` and
           `vcgpu.remove_edge_ub`
  matching `vcgpu.mcm`, the maximum-matching mode

Outputs: sizes, decisions and statuses.  The cover itself is asked for and comes
back with each result, but which of a graph's many optimal covers it is depends
on the order in which the warps reach them, two runs of the same code included,
so its size stands in for it (and must equal the optimum).  For the same reason
a PVC "yes" gives its decision alone.  The bounds are deterministic and return
their covers whole.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "parallel-vertex-cover-algorithms-on-gpus_b200"))

import vcgpu  # noqa: E402
from vcgpu import workloads as W  # noqa: E402


def listed():
    return [
        # The smallest calls: G(60, 0.1), where the launch and the copies count.
        {"name": "plain_small", "kind": "plain", "family": "gnp", "count": 8, "n": 60, "n_hi": 60, "d": 5.9, "d_hi": 5.9,
         "pvc": True},
        # The served stream's random 3-regular graphs, of the size class of at most 128 vertices.
        {"name": "plain_regular", "kind": "plain", "family": "regular", "count": 4, "n": 100, "n_hi": 126, "d": 3.0,
         "d_hi": 3.0, "pvc": False},
        # Ordinary sparse graphs of up to 255 vertices: trees of 10^4 to 10^6 nodes.
        {"name": "plain_medium", "kind": "plain", "family": "gnp", "count": 6, "n": 133, "n_hi": 203, "d": 4.5, "d_hi": 6.5,
         "pvc": False},
        # 256 to 640 vertices, degrees in bytes (the served stream's middle sizes).
        {"name": "plain_wide", "kind": "plain", "family": "gnp", "count": 4, "n": 301, "n_hi": 597, "d": 3.2, "d_hi": 3.6,
         "pvc": False},
        # Dense graphs in the manner of the DIMACS-style files: hundreds of vertices of degree in the hundreds.
        {"name": "plain_dense", "kind": "plain", "family": "dense", "count": 3, "n": 300, "n_hi": 450, "d": 0.70,
         "d_hi": 0.78, "pvc": False},
        # Sparse graphs of thousands of vertices: a planted cover of n = 2000 with pendant paths, asked both ways.
        {"name": "plain_planted", "kind": "plain", "family": "planted", "count": 4, "n": 2000, "n_hi": 2000, "d": 3.0,
         "d_hi": 3.0, "pvc": True},
        # A large power-law graph: n = 100000, exponent 2.1, average degree 8, degrees capped at 2000.
        {"name": "plain_power_law", "kind": "plain", "family": "chung_lu", "count": 1, "n": 100000, "n_hi": 100000,
         "d": 8.0, "d_hi": 8.0, "pvc": False},
        # The batched workload: independent G(n, p) of uneven size in one launch (n to 160: the full range's hardest
        # graphs take minutes).
        {"name": "batch_uneven", "kind": "batch", "family": "gnp", "count": 512, "n": 30, "n_hi": 160, "d": 3.0,
         "d_hi": 12.0, "pvc": False, "large": 0},
        # Small graphs beside one large power-law graph, already on the GPU, MVC and PVC mixed.
        {"name": "device_mixed", "kind": "device", "family": "gnp", "count": 512, "n": 100, "n_hi": 100, "d": 7.9,
         "d_hi": 7.9, "pvc": True, "large": 30000},
        # A burst of small requests through a server, MVC and PVC mixed.
        {"name": "served_burst", "kind": "served", "family": "gnp", "count": 400, "n": 50, "n_hi": 120, "d": 3.0,
         "d_hi": 8.0, "pvc": True},
        # Upper bounds of one large graph and of many small ones.
        {"name": "bounds", "kind": "bounds", "family": "gnp", "count": 192, "n": 30, "n_hi": 200, "d": 3.0, "d_hi": 12.0,
         "large": 12000},
        # Maximum matchings: large graphs that have a perfect one, small ones whose whole tree is searched.
        {"name": "matching", "kind": "matching", "family": "planted", "count": 6, "n": 255, "n_hi": 1024, "d": 6.0,
         "d_hi": 6.0},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed kinds; sizes over the same ranges."""
    kind = rng.choice(["plain", "plain", "plain", "plain", "batch", "device", "served", "bounds", "matching"])
    if kind == "plain":
        family = rng.choice(["gnp", "gnp", "regular", "dense", "planted", "chung_lu"])
        if family == "gnp":
            n = _log_uniform(rng, 40, 600)
            # the degree up to which graphs of this size are solved in milliseconds
            top = 9.0 if n <= 110 else (6.0 if n <= 203 else 3.5)
            d = rng.uniform(3.0, top)
            return {"kind": kind, "family": family, "count": rng.randint(3, 8), "n": n, "n_hi": min(600, n + n // 16),
                    "d": round(d, 2), "d_hi": round(d, 2), "pvc": rng.random() < 0.3}
        if family == "regular":
            n = 2 * rng.randint(25, 63)
            return {"kind": kind, "family": family, "count": rng.randint(3, 6), "n": n, "n_hi": n, "d": 3.0, "d_hi": 3.0,
                    "pvc": rng.random() < 0.3}
        if family == "dense":
            n, p = rng.randint(256, 450), round(rng.uniform(0.7, 0.9), 3)
            return {"kind": kind, "family": family, "count": rng.randint(2, 3), "n": n, "n_hi": n, "d": p, "d_hi": p,
                    "pvc": False}
        if family == "planted":
            n = _log_uniform(rng, 1030, 4000)
            return {"kind": kind, "family": family, "count": rng.randint(2, 4), "n": n, "n_hi": n, "d": 3.0, "d_hi": 3.0,
                    "pvc": rng.random() < 0.5}
        n = _log_uniform(rng, 2000, 100000)
        return {"kind": kind, "family": family, "count": 1 if n > 30000 else 2, "n": n, "n_hi": n, "d": 8.0, "d_hi": 8.0,
                "pvc": False}
    if kind == "batch":
        hi = rng.randint(60, 150)
        return {"kind": kind, "family": "gnp", "count": _log_uniform(rng, 16, 512), "n": 30, "n_hi": hi, "d": 3.0,
                "d_hi": round(rng.uniform(6.0, 12.0), 2), "pvc": rng.random() < 0.3, "large": 0}
    if kind == "device":
        n = rng.randint(50, 110)
        return {"kind": kind, "family": "gnp", "count": _log_uniform(rng, 16, 512), "n": n, "n_hi": n,
                "d": round(rng.uniform(3.0, 8.0), 2), "d_hi": 8.0, "pvc": rng.random() < 0.5,
                "large": _log_uniform(rng, 2000, 30000)}
    if kind == "served":
        return {"kind": kind, "family": "gnp", "count": _log_uniform(rng, 16, 400), "n": 50, "n_hi": rng.randint(70, 120),
                "d": 3.0, "d_hi": round(rng.uniform(4.0, 8.0), 2), "pvc": True}
    if kind == "bounds":
        return {"kind": kind, "family": "gnp", "count": rng.randint(16, 192), "n": 30, "n_hi": rng.randint(60, 200),
                "d": 3.0, "d_hi": 12.0, "large": _log_uniform(rng, 1000, 12000)}
    n = rng.randint(64, 1000)
    return {"kind": kind, "family": "planted", "count": rng.randint(3, 6), "n": n, "n_hi": n + 24, "d": 6.0, "d_hi": 6.0}


def _graph(case, rng):
    """One graph of the case's family, its size and density drawn from the case's range."""
    n = rng.randint(case["n"], case["n_hi"])
    d = rng.uniform(case["d"], case["d_hi"])
    seed = rng.randrange(1 << 40)
    family = case["family"]
    if family == "gnp":
        return W.gnp(n, d / (n - 1), seed)
    if family == "regular":
        return W.random_regular(n + n % 2, 3, seed)
    if family == "dense":
        return W.gnp(n, d, seed)
    if family == "chung_lu":
        return W.chung_lu(n, 2.1, d, 2000.0, seed)
    if case["kind"] == "matching":
        return W.planted_matching(n, d, seed)
    return W.planted_cover(n, n * 3 // 20, 3 * n, n // 20, 4, seed)


def _questions(case, graphs):
    """Per graph "mvc" or ("pvc", k): with pvc, every other graph is asked whether half of its vertices (and a few)
    suffice, which is near the optimum of sparse random graphs."""
    out = []
    for i, g in enumerate(graphs):
        if case.get("pvc") and i % 2:
            out.append(("pvc", max(1, g.n * 3 // 20 if case["family"] == "planted" else int(0.56 * g.n))))
        else:
            out.append(("mvc", 0))
    return out


def prepare(case, seed):
    rng = random.Random(seed)
    graphs = [_graph(case, rng) for _ in range(case["count"])]
    kind = case["kind"]
    if kind == "matching":  # and sparse graphs without a perfect matching, whose tree is searched to its end
        graphs += [W.gnp(rng.randint(12, 18), 2.5 / 15, rng.randrange(1 << 40)) for _ in range(4)]
    if case.get("large"):
        graphs.append(W.chung_lu(case["large"], 2.1, 8.0, 2000.0, rng.randrange(1 << 40)))
    state = {"kind": kind, "graphs": graphs, "asked": _questions(case, graphs)}
    if kind in ("batch", "device", "bounds"):
        arena = W.pack(graphs)
        state["arena"] = arena
        if kind == "device":
            state["row_ptr"] = torch.from_numpy(arena.row_ptr.view(np.int32)).cuda()
            state["col"] = torch.from_numpy(arena.col.view(np.int32)).cuda()
    if kind == "bounds":
        state["r"] = rng.randrange(1 << 30)
        state["width"] = case["n_hi"] * case["count"] + case["large"]
    return state


def _answers(asked, solutions):
    """[status, decision, size, size of the cover] per graph (see the file comment for PVC)."""
    rows = []
    for (instance, _), s in zip(asked, solutions):
        if instance == "mvc":
            rows.append((s.status, s.decision, s.size, int(s.cover.sum())))
        else:
            rows.append((s.status, s.decision, 0, 0))
    return np.array(rows, dtype=np.int64)


def _rows(covers, width):
    """The covers one after another, at the end zeros up to the longest that graphs of the case's sizes can give."""
    flat = np.zeros(width, dtype=np.uint8)
    at = 0
    for c in covers:
        flat[at:at + len(c)] = c
        at += len(c)
    return flat


def run(state):
    kind, graphs, asked = state["kind"], state["graphs"], state["asked"]
    if kind == "plain":
        return _answers(asked, [vcgpu.solve(g, instance, k=k) for g, (instance, k) in zip(graphs, asked)])
    if kind in ("batch", "device"):
        on_device = {}
        if kind == "device":
            on_device = {"d_row_ptr": state["row_ptr"].data_ptr(), "d_col": state["col"].data_ptr()}
        status, solutions = vcgpu.solve_batch(state["arena"], [a for a, _ in asked], ks=[k for _, k in asked], **on_device)
        return {"status": status, "answers": _answers(asked, solutions)}
    if kind == "served":
        got = {}
        with vcgpu.Server(max_vertices=255) as server:
            tickets = [server.submit(g, instance, k=k) for g, (instance, k) in zip(graphs, asked)]
            while len(got) < len(tickets):
                for t in server.completed():
                    got[t] = server.poll(t)
        return _answers(asked, [got[t] for t in tickets])
    if kind == "bounds":
        ub_max, cover_max, _ = vcgpu.remove_max_ub(state["arena"])
        ub_edge, cover_edge, _ = vcgpu.remove_edge_ub(state["arena"], state["r"])
        return {"max": np.array(ub_max), "max_cover": _rows(cover_max, state["width"]),
                "edge": np.array(ub_edge), "edge_cover": _rows(cover_edge, state["width"])}
    return np.array([(s.status, s.size) for s in (vcgpu.mcm(g) for g in graphs)], dtype=np.int64)


def work(case):
    """Bytes: every graph's row offsets and neighbour ids read once, its cover and size written once.  The search itself
    is integer work on chip whose amount depends on the graph, not on its size: no floating-point operations."""
    n = (case["n"] + case["n_hi"]) / 2
    d = (case["d"] + case["d_hi"]) / 2
    if case["family"] == "dense":
        d *= n
    elif case["family"] == "planted" and case["kind"] == "plain":
        d = 6.5
    total = case["count"] * (4 * (n + 1) + 4 * n * d + n + 8)
    large = case.get("large", 0)
    total += 45 * large
    return {"bytes": total * (2 if case["kind"] == "bounds" else 1), "flops": 0}


def _cover_size(g):
    """Minimum vertex cover of a small graph, by branching on a vertex of largest degree with the graph as Python
    integers; independent of the library."""
    adj = [0] * g.n
    for u, v in g.edges().tolist():
        adj[u] |= 1 << v
        adj[v] |= 1 << u
    best = g.n

    def search(live, size):
        nonlocal best
        while True:
            top, at, degrees, leaf = 0, -1, 0, -1
            rest = live
            while rest:
                v = (rest & -rest).bit_length() - 1
                rest &= rest - 1
                deg = (adj[v] & live).bit_count()
                if deg == 0:
                    live &= ~(1 << v)
                    continue
                degrees += deg
                if deg == 1:
                    leaf = v
                if deg > top:
                    top, at = deg, v
            if leaf < 0:
                break
            live &= ~(adj[leaf] & live) & ~(1 << leaf)
            size += 1
        if top == 0:
            best = min(best, size)
            return
        if size + (degrees // 2 + top - 1) // top >= best:
            return
        search(live & ~(1 << at), size + 1)
        taken = adj[at] & live
        search(live & ~taken & ~(1 << at), size + taken.bit_count())

    search((1 << g.n) - 1, 0)
    return best


def exact(case, seed):
    """The answers of plain calls on small graphs from a search of its own in plain Python; None where that would take
    too long."""
    if case["kind"] != "plain" or case["n_hi"] > 64 or case["family"] not in ("gnp", "regular"):
        return None
    state = prepare(case, seed)
    rows = []
    for g, (instance, k) in zip(state["graphs"], state["asked"]):
        opt = _cover_size(g)
        rows.append((0, 1, opt, opt) if instance == "mvc" else (0, int(opt <= k), 0, 0))
    return np.array(rows, dtype=np.int64)
