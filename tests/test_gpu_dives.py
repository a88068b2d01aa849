"""The greedy dives at the start of plain solves of 256 to 1024 vertices: covers
they report stand, whatever the graph looks like (isolated vertices, one hub, dense
beside the rule's edge of average degree 16, ids at word edges), and PVC answers by a
dive are right on both sides of the optimum."""
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


def _check(g, opt):
    r = vcgpu.solve(g, "mvc", time_limit=TL)
    assert r.status == vcgpu.VC_OK and r.size == opt and W.is_cover(g, r.cover) and int(r.cover.sum()) == opt
    u = vcgpu.solve(g, "mvc", ub=opt, time_limit=TL)
    assert u.status == vcgpu.VC_OK and u.size == opt and int(u.cover.sum()) == opt
    for k in (opt - 1, opt, opt + 1, g.n):
        if k < 0:
            continue
        p = vcgpu.solve(g, "pvc", k=k, time_limit=TL)
        assert p.status == vcgpu.VC_OK and p.decision == int(k >= opt), k
        if p.decision:
            assert W.is_cover(g, p.cover) and int(p.cover.sum()) == p.size <= k


@pytest.mark.parametrize("n", [256, 257, 287, 288, 512, 513, 639, 640, 641, 700, 1023, 1024])
def test_sparse_graphs_and_forests(n):
    for d, seed in ((1.5, 1), (2.9, 2)):
        g = W.gnp(n, d / (n - 1), 31 * n + seed)
        st, opt, _, _ = O.mvc(g, node_limit=500_000)
        assert st == O.OK
        _check(g, opt)
    _check(W.from_edges(n, np.array([[n - 1, i] for i in range(n - 1)])), 1)       # one hub
    _check(W.from_edges(n, np.array([[0, n - 1], [31, 32], [n // 2, n // 2 + 1]])), 3)  # nearly all isolated


@pytest.mark.parametrize("d", [15.5, 16.5])
def test_around_the_rule(d):
    """A clique beside sparse parts, with the average degree on either side of the line."""
    n = 400
    k = int((d * n) ** 0.5)  # a clique of k vertices has about d * n entries
    e = [(i, j) for i in range(k) for j in range(i)] + [(i, i + 1) for i in range(k, n - 1, 2)]
    opt = k - 1 + len(range(k, n - 1, 2))
    _check(W.from_edges(n, np.asarray(e)), opt)
