"""Graphs of more than 1024 vertices: the whole-chip reduction of their root
(sizes around its blocks, rows longer than a lane walks, cascades longer than its
pass limit, what is left of every kernel class or nothing) and the device-side
checks of host-resident graphs, against known optima and the CPU oracle."""
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


def _relabel(n, edges, seed):
    perm = np.random.default_rng(seed).permutation(n)
    e = np.asarray(edges, dtype=np.int64).reshape(-1, 2)
    return W.from_edges(n, perm[e])


def _check(g, opt):
    r = vcgpu.solve(g, "mvc", time_limit=TL)
    assert r.status == vcgpu.VC_OK and r.size == opt and W.is_cover(g, r.cover) and int(r.cover.sum()) == opt
    for ub in (opt + 3, opt, opt - 2):  # min(ub, OPT); a cover comes back if one of at most ub exists
        if ub <= 0:  # no bound
            continue
        u = vcgpu.solve(g, "mvc", ub=ub, time_limit=TL)
        assert u.status == vcgpu.VC_OK and u.size == min(ub, opt)
        assert (u.cover is not None) == (ub >= opt)
    for k, want in ((opt, 1), (opt - 1, 0), (g.n + 7, 1), (0, int(opt == 0))):
        if k < 0:
            continue
        p = vcgpu.solve(g, "pvc", k=k, time_limit=TL)
        assert p.status == vcgpu.VC_OK and p.decision == want, k
        if want:
            assert W.is_cover(g, p.cover) and int(p.cover.sum()) == p.size <= k


@pytest.mark.parametrize("n", [1025, 1535, 1536, 1537, 2048, 4097, 5000])
def test_paths_stars_and_cycles(n):
    # a path: 1250 passes at n = 5000, more than a reduction makes
    _check(_relabel(n, [(i, i + 1) for i in range(n - 1)], n), n // 2)
    # one cycle: nothing to reduce
    _check(_relabel(n, [(i, (i + 1) % n) for i in range(n)], n + 1), (n + 1) // 2)
    # stars whose hubs have rows of 63, 64, 65 and the rest of the vertices
    edges, at, hubs = [], 0, 0
    for k in (63, 64, 65, n - 196):
        edges += [(at, at + j) for j in range(1, k + 1)]
        at += k + 1
        hubs += 1
    _check(_relabel(n, edges, n + 2), hubs)
    _check(W.from_edges(n, np.zeros((0, 2))), 0)


def test_random_graphs_plain_and_batched():
    """Sparse graphs whose rests are empty, of the dense classes, and above 1024 vertices, beside small ones."""
    rng = np.random.default_rng(3)
    graphs, opts = [], []
    for n, d in ((1100, 2.2), (1500, 2.9), (1800, 3.0), (3000, 2.5), (2500, 3.05), (60, 5.0), (300, 3.0), (1025, 3.3)):
        for _ in range(8):
            g = W.gnp(n, d / (n - 1), int(rng.integers(1 << 30)))
            st, opt, _, _ = O.mvc(g, node_limit=60_000)
            if st == O.OK:
                graphs.append(g)
                opts.append(opt)
                break
    g = W.planted_cover(2000, 300, 6000, 100, 4, 9)
    st, opt, _, _ = O.mvc(g, node_limit=1_000_000)
    assert st == O.OK
    graphs.append(g)
    opts.append(opt)
    assert sum(g.n > 1024 for g in graphs) >= 4
    # triangles with one shared vertex each, hung on a long cycle: a rest above 1024 vertices
    m = 1300
    e = [(i, (i + 1) % m) for i in range(m)]
    graphs.append(_relabel(m, e, 5))
    opts.append(m // 2)
    for g, opt in zip(graphs, opts):
        if g.n > 1024:
            _check(g, opt)
    arena = W.pack(graphs)
    st, sols = vcgpu.solve_batch(arena, "mvc", time_limit=TL)
    assert st == vcgpu.VC_OK
    for g, s, opt in zip(graphs, sols, opts):
        assert s.size == opt and W.is_cover(g, s.cover) and int(s.cover.sum()) == opt
    for shift, want in ((0, 1), (-1, 0)):
        st, sols = vcgpu.solve_batch(arena, "pvc", ks=[o + shift for o in opts], time_limit=TL)
        assert st == vcgpu.VC_OK and [s.decision for s in sols] == [want] * len(graphs)
    torch = pytest.importorskip("torch")
    d_rp = torch.from_numpy(arena.row_ptr.astype(np.int32)).cuda()
    d_col = torch.from_numpy(arena.col.astype(np.int32)).cuda()
    torch.cuda.synchronize()
    st, sols = vcgpu.solve_batch(arena, "mvc", time_limit=TL, d_row_ptr=d_rp.data_ptr(), d_col=d_col.data_ptr())
    assert st == vcgpu.VC_OK and [s.size for s in sols] == opts


def _broken(g):
    """Graphs that break one rule each."""
    def copy():
        return W.Graph(g.n, g.row_ptr.copy(), g.col.copy())
    v = int(np.flatnonzero(np.diff(g.row_ptr.astype(np.int64)) >= 3)[5])
    lo, hi = int(g.row_ptr[v]), int(g.row_ptr[v + 1])
    b = copy(); b.col[lo] = g.n + 2; yield "id out of range", b
    b = copy(); b.col[hi - 1] = v; yield "self loop", b
    b = copy(); b.col[lo], b.col[lo + 1] = int(g.col[lo + 1]), int(g.col[lo]); yield "unsorted", b
    b = copy(); b.col[lo + 1] = b.col[lo]; yield "duplicate", b
    b = copy(); b.row_ptr[v + 1] = lo - 1; yield "decreasing offsets", b
    b = copy(); b.row_ptr[v + 1] = 2 * g.m + 9; yield "offset past the end", b
    other = next(x for x in range(g.n) if x != v and x not in g.col[lo:hi].tolist() and x > int(g.col[hi - 1]))
    b = copy(); b.col[hi - 1] = other; yield "one direction only", b
    b = copy(); b.row_ptr[g.n] = 2 * g.m - 2; yield "row_ptr[n] is not 2m", b


@pytest.mark.parametrize("n,d", [(400, 8.0), (700, 9.0), (1500, 5.0), (6000, 4.0)])
def test_device_checks_of_host_graphs(n, d):
    """A host-resident graph with more entries than the host checks itself is refused as before, alone and in a batch, and
    the next call is exact."""
    g = W.gnp(n, d / (n - 1), 1000 + n)
    assert 2 * g.m > 2048
    small = W.config1_graph()
    good = vcgpu.solve(small).size
    for what, b in _broken(g):
        assert vcgpu.solve(b).status == vcgpu.VC_ERR_INVALID, what
        if what != "row_ptr[n] is not 2m":  # a batch takes 2m from the rows
            st, sols = vcgpu.solve_batch(W.pack([small, b, small]), time_limit=TL)
            assert st == vcgpu.VC_ERR_INVALID and all(s.status == vcgpu.VC_ERR_INVALID for s in sols), what
    assert vcgpu.solve(small).size == good
