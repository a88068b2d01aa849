"""A host-resident batch with a graph that fails its checks is refused before any
graph is searched: in the class of the long search, in a later one, in an earlier
one, and among large graphs that are reduced first."""
import time

import numpy as np
import pytest

import vcgpu
from vcgpu import workloads as W

pytestmark = pytest.mark.gpu
LIMIT = 6.0  # seconds that the long search is given


def _broken(g):
    """One entry names another vertex: the edge is in one direction only."""
    col = g.col.copy()
    for v in range(g.n):
        lo, hi = int(g.row_ptr[v]), int(g.row_ptr[v + 1])
        after = [x for x in range(int(col[hi - 1]) + 1 if hi > lo else g.n, g.n) if x != v]
        if after:
            col[hi - 1] = after[-1]
            break
    return W.Graph(g.n, g.row_ptr, col)


LONG = W.gnp(250, 0.06, 11)          # seconds of search
WIDE_LONG = W.gnp(400, 0.02, 11)


@pytest.mark.parametrize("long,bad", [
    (LONG, W.gnp(120, 0.05, 1)), (LONG, W.gnp(400, 0.01, 1)), (LONG, W.gnp(500, 0.7, 1)), (LONG, W.gnp(1500, 0.002, 1)),
    (WIDE_LONG, W.gnp(60, 0.1, 1)), (WIDE_LONG, W.planted_cover(2000, 300, 6000, 100, 4, 9)),
])
def test_refused_before_the_search(long, bad):
    ok = [W.config1_graph(), W.gnp(1300, 0.001, 2)]
    good = [vcgpu.solve(g).size for g in ok]
    arena = W.pack([ok[0], long, _broken(bad), ok[1]])
    for instances, ks in (("mvc", None), ("pvc", [30, 100, 40, 300])):
        t0 = time.perf_counter()
        st, sols = vcgpu.solve_batch(arena, instances, ks=ks, time_limit=LIMIT)
        assert time.perf_counter() - t0 < LIMIT / 4
        assert st == vcgpu.VC_ERR_INVALID
        for s in sols:
            assert s.status == vcgpu.VC_ERR_INVALID and s.size == 0 and s.cover is None and s.tree_nodes == 0
    st, sols = vcgpu.solve_batch(W.pack(ok), "mvc")
    assert st == vcgpu.VC_OK and [s.size for s in sols] == good


def test_valid_batches_of_every_class_pass_their_checks():
    graphs = [W.gnp(60, 0.1, 1), W.gnp(200, 0.02, 2), W.gnp(400, 0.007, 3), W.gnp(500, 0.7, 4), W.gnp(900, 0.0025, 5),
              W.gnp(1500, 0.0015, 6), W.chung_lu(5000, 2.1, 8.0, 2000.0, 7)]
    opts = [vcgpu.solve(g, time_limit=60.0).size for g in graphs]
    for keep in (range(7), (0, 2, 3), (1,), (5, 6), (3, 4)):
        st, sols = vcgpu.solve_batch(W.pack([graphs[i] for i in keep]), "mvc", time_limit=60.0)
        assert st == vcgpu.VC_OK and [s.size for s in sols] == [opts[i] for i in keep]
