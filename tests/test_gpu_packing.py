"""The packing bound of the dense kernels at the sizes where it can go wrong:
word and kernel-class edges, degrees on both sides of what its counters hold,
odd cycles, triangles and cliques (where the packing is tight, short by one, or
far off).  Unions of small components have known optima; random graphs go to the
CPU oracle."""
import os
import sys

import numpy as np
import pytest

import vcgpu
from vcgpu import workloads as W

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "oracle"))
import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu
TL = 60.0


def _union(n, parts, seed):
    """Disjoint components ("cycle" or "clique" or "star", size) over the first vertices of a random relabelling of n;
    returns the graph and its optimum."""
    perm = np.random.default_rng(seed).permutation(n)
    edges, at, opt = [], 0, 0
    for kind, k in parts:
        if at + k > n:
            break
        ids = perm[at:at + k]
        at += k
        if kind == "cycle":
            edges += [(ids[i], ids[(i + 1) % k]) for i in range(k)]
            opt += (k + 1) // 2
        elif kind == "clique":
            edges += [(ids[i], ids[j]) for i in range(k) for j in range(i)]
            opt += k - 1
        else:  # two hubs joined to all the others: the hubs cover it
            edges += [(ids[h], ids[j]) for h in (0, 1) for j in range(2, k)]
            opt += min(2, k - 2)
    return W.from_edges(n, np.asarray(edges, dtype=np.int64).reshape(-1, 2)), opt


def _check(g, opt, alone=True):
    if alone:
        r = vcgpu.solve(g, "mvc", time_limit=TL)
        assert r.status == vcgpu.VC_OK and r.size == opt and W.is_cover(g, r.cover) and int(r.cover.sum()) == opt
        for k, want in ((opt, 1), (opt - 1, 0)):
            if k >= 0:
                p = vcgpu.solve(g, "pvc", k=k, time_limit=TL)
                assert p.status == vcgpu.VC_OK and p.decision == want, (g.n, k)


@pytest.mark.parametrize("n", [31, 32, 33, 63, 64, 65, 127, 128, 129, 160, 161, 255, 256, 257, 511, 512, 513, 640, 641, 1023,
                               1024])
def test_unions_of_small_components(n):
    cycles = [("cycle", k) for k in (5, 7, 4, 9, 3, 6, 5, 11) * 40]
    cliques = [("clique", k) for k in (3, 4, 5, 3, 2, 6) * 60]
    for i, parts in enumerate((cycles, cliques, cycles[:4] + cliques[:9] + [("star", 20), ("cycle", 13)])):
        g, opt = _union(n, parts, 100 * n + i)
        _check(g, opt)


@pytest.mark.parametrize("hub", [29, 30, 31, 32, 33, 62])
@pytest.mark.parametrize("n", [128, 200, 400, 900])
def test_degrees_around_the_counters(n, hub):
    """Two hubs of that degree beside odd cycles: the bound is off above degree 31 and on once the hubs are gone."""
    g, opt = _union(n, [("star", hub + 2)] + [("cycle", 5), ("cycle", 7)] * 40, n + hub)
    _check(g, opt)


def test_random_graphs_alone_and_batched():
    rng = np.random.default_rng(77)
    graphs, opts = [], []
    while len(graphs) < 60:
        n = int(rng.choice([40, 64, 65, 100, 128, 129, 150, 200, 255, 300]))
        d = float(rng.uniform(2.5, 6.0 if n <= 150 else 3.6))
        g = W.random_regular(n + n % 2, 3, int(rng.integers(1 << 30))) if rng.random() < 0.3 and n <= 100 else \
            W.gnp(n, d / (n - 1), int(rng.integers(1 << 30)))
        st, opt, _, _ = O.mvc(g, node_limit=300_000)
        if st == O.OK:
            graphs.append(g)
            opts.append(opt)
    for g, opt in list(zip(graphs, opts))[:25]:
        _check(g, opt)
    arena = W.pack(graphs)
    st, sols = vcgpu.solve_batch(arena, "mvc", time_limit=TL)
    assert st == vcgpu.VC_OK
    for g, s, opt in zip(graphs, sols, opts):
        assert s.size == opt and W.is_cover(g, s.cover) and int(s.cover.sum()) == opt
    for shift, want in ((0, 1), (-1, 0)):
        st, sols = vcgpu.solve_batch(arena, "pvc", ks=[o + shift for o in opts], time_limit=TL)
        assert st == vcgpu.VC_OK and [s.decision for s in sols] == [want] * len(graphs)
