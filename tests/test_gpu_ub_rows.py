"""The upper-bound heuristics where their rows and state change form: deletions of
more neighbours than a block has threads, rows that lose a vertex together and hold
one another, and graphs around what shared memory holds, against the exact
restatements (bounds and covers)."""
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


def _hubs(n, hubs, seed):
    """Hubs joined to random halves of the rest and to one another, triangles and pendant vertices beside them."""
    rng = np.random.default_rng(seed)
    e = [(h, int(v)) for h in range(hubs) for v in rng.choice(np.arange(hubs, n), size=n // 2, replace=False)]
    e += [(a, b) for a in range(hubs) for b in range(a)]
    e += [(int(a), int(b)) for a, b in rng.integers(hubs, n, size=(n // 3, 2)) if a != b]
    perm = rng.permutation(n)
    return W.from_edges(n, perm[np.asarray(e, dtype=np.int64)])


@pytest.mark.parametrize("n,hubs", [(40, 3), (600, 5), (1100, 2), (1500, 12), (3000, 4)])
def test_rows_longer_than_a_block_and_crossing_rows(n, hubs):
    """Deletions that change more rows than the block has threads, and rows that lose a vertex together and hold one
    another; the covers are the restatement's vertex by vertex."""
    g = _hubs(n, hubs, n + hubs)
    ubs, covers, _ = vcgpu.remove_max_ub(W.pack([g, W.gnp(30, 0.2, 3)]))
    want, mask = O.remove_max_ub(g)[:2]
    assert ubs[0] == want and np.array_equal(covers[0], np.asarray(mask, dtype=bool))
    for r in (0, 5, 1804289383):
        ubs, covers, _ = vcgpu.remove_edge_ub(W.pack([g]), r)
        want, mask = O.remove_edge_ub(g, r)[:2]
        assert ubs[0] == want and np.array_equal(covers[0], np.asarray(mask, dtype=bool))


@pytest.mark.parametrize("n", [14000, 14100, 26000, 30000])
def test_around_what_shared_memory_holds(n):
    """The largest graphs whose degrees and offsets sit in shared memory, and those that keep their bitmaps only."""
    g = W.gnp(n, 2.6 / (n - 1), n)
    ubs, covers, _ = vcgpu.remove_max_ub(W.pack([g]))
    want, mask = O.remove_max_ub(g)[:2]
    assert ubs[0] == want and np.array_equal(covers[0], np.asarray(mask, dtype=bool))
    ubs, covers, _ = vcgpu.remove_edge_ub(W.pack([g]), 99)
    want, mask = O.remove_edge_ub(g, 99)[:2]
    assert ubs[0] == want and np.array_equal(covers[0], np.asarray(mask, dtype=bool))
