"""Plain solves of dense graphs from n roots: sizes at word and kernel edges, both
sides of the density rule, ties throughout the order (regular graphs), vertices of
degree n - 1, and bounds that cut most roots, against known optima and the oracle."""
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
    for ub in (0, opt, opt + 2, opt - 1):
        if ub < 0:
            continue
        r = vcgpu.solve(g, "mvc", ub=ub, time_limit=TL)
        assert r.status == vcgpu.VC_OK and r.size == (min(ub, opt) if ub else opt)
        if r.cover is not None:
            assert W.is_cover(g, r.cover) and int(r.cover.sum()) == opt
    for k in (opt - 1, opt, g.n - 1, g.n):
        if k >= 0:
            p = vcgpu.solve(g, "pvc", k=k, time_limit=TL)
            assert p.status == vcgpu.VC_OK and p.decision == int(k >= opt), k
            if p.decision:
                assert W.is_cover(g, p.cover) and int(p.cover.sum()) == p.size <= k


@pytest.mark.parametrize("n", [63, 64, 65, 128, 129, 255, 256, 257, 512, 513, 640, 641, 1024])
def test_known_dense_graphs(n):
    pairs = np.stack(np.triu_indices(n, 1), axis=1)
    _check(W.from_edges(n, pairs), n - 1)                                   # complete
    if n % 2 == 0:                                                          # complete but for a perfect matching
        keep = ~((pairs[:, 0] % 2 == 0) & (pairs[:, 1] == pairs[:, 0] + 1))
        _check(W.from_edges(n, pairs[keep]), n - 2)
    side = pairs[:, 0] % 2 != pairs[:, 1] % 2                               # complete bipartite: density one half
    _check(W.from_edges(n, pairs[side]), n // 2)


@pytest.mark.parametrize("n,p", [(64, 0.39), (64, 0.42), (100, 0.6), (130, 0.5), (200, 0.75), (256, 0.85), (300, 0.7), (520, 0.9)])
def test_random_dense_graphs(n, p):
    g = W.gnp(n, p, int(1000 * p) + n)
    st, opt, _, _ = O.mvc(g, node_limit=20_000_000)
    assert st == O.OK
    _check(g, opt)
