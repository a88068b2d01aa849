"""The upper-bound heuristics where a moved row's vertices are marked (rows of up to 8
entries) and where they are not (longer ones), and around the sizes at which the cached
maxima change, against the exact restatements (bounds and covers)."""
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


def _triangles(n, k, seed):
    """Random triangles, k per vertex on average: rows of some 2k entries, with degree-2 vertices on triangles."""
    rng = np.random.default_rng(seed)
    t = rng.integers(0, n, size=(max(1, n * k // 3), 3))
    e = np.concatenate([t[:, [0, 1]], t[:, [1, 2]], t[:, [0, 2]]])
    return W.from_edges(n, e[e[:, 0] != e[:, 1]])


def _check(graphs):
    ubs, covers, _ = vcgpu.remove_max_ub(W.pack(graphs))
    for g, u, c in zip(graphs, ubs, covers):
        want, mask = O.remove_max_ub(g)[:2]
        assert u == want and np.array_equal(c, np.asarray(mask, dtype=bool)), g.n
    ubs, covers, _ = vcgpu.remove_edge_ub(W.pack(graphs), 5)
    for g, u, c in zip(graphs, ubs, covers):
        want, mask = O.remove_edge_ub(g, 5)[:2]
        assert u == want and np.array_equal(c, np.asarray(mask, dtype=bool)), g.n


def test_short_and_long_rows():
    _check([_triangles(n, k, 10 * n + k) for n in (3, 31, 32, 33, 200, 700) for k in (1, 2, 3, 4, 5, 9)])


@pytest.mark.parametrize("n", [127, 128, 129, 2047, 2048, 2049, 8191, 8192, 8193, 13990, 14060, 16384, 16385, 17000])
def test_regular_graphs_around_the_cached_maxima(n):
    _check([W.random_regular(n + n % 2, 3, n), W.gnp(n, 3.0 / n, n)])
