"""The three ways to reduce a large graph's root -- one CTA, a cluster of CTAs, the
whole chip -- on both sides of the sizes and counts where one takes over from
another: known optima, rows longer than a lane walks, bounds that make the
high-degree rule fire, and the same graph by different ways."""
import numpy as np
import pytest

import vcgpu
from vcgpu import workloads as W

pytestmark = pytest.mark.gpu
TL = 60.0


def _relabel(n, edges, seed):
    perm = np.random.default_rng(seed).permutation(n)
    return W.from_edges(n, perm[np.asarray(edges, dtype=np.int64).reshape(-1, 2)])


def _path(n):
    return _relabel(n, [(i, i + 1) for i in range(n - 1)], n), n // 2


def _stars(n):
    edges, at = [], 0
    for k in (1, 31, 32, 33, 63, 64, 65, n - 297):
        edges += [(at, at + j) for j in range(1, k + 1)]
        at += k + 1
    return _relabel(n, edges, n), 8


def _ok(g, s, opt):
    assert s.status == vcgpu.VC_OK and s.size == opt and W.is_cover(g, s.cover) and int(s.cover.sum()) == opt


@pytest.mark.parametrize("n", [1025, 1056, 2047, 2049, 7399, 7400, 7401, 7405, 24576, 24577])
def test_sizes_alone_and_in_batches(n):
    for make in (_path, _stars):
        g, opt = make(n)
        _ok(g, vcgpu.solve(g, "mvc", time_limit=TL), opt)
        for k, want in ((opt, 1), (opt - 1, 0)):
            p = vcgpu.solve(g, "pvc", k=k, time_limit=TL)
            assert p.status == vcgpu.VC_OK and p.decision == want
        u = vcgpu.solve(g, "mvc", ub=opt - 1, time_limit=TL)
        assert u.status == vcgpu.VC_OK and u.size == opt - 1 and u.cover is None
        for count in (2, 5):
            st, sols = vcgpu.solve_batch(W.pack([g] * count), "mvc", time_limit=TL)
            assert st == vcgpu.VC_OK
            for s in sols:
                _ok(g, s, opt)


@pytest.mark.parametrize("n", [6000, 9000, 20000, 26000, 40000])
def test_the_same_graph_by_different_ways(n):
    """Alone, and among enough others of its size that it is reduced in another way; with a rest to search and without."""
    for g in (W.chung_lu(n, 2.1, 8.0, 2000.0, n), W.gnp(n, 2.3 / n, n)):
        alone = vcgpu.solve(g, "mvc", time_limit=TL)
        _ok(g, alone, alone.size)
        no = vcgpu.solve(g, "pvc", k=alone.size - 1, time_limit=TL)
        assert no.status == vcgpu.VC_OK and no.decision == 0
        for count in (3, 20):
            st, sols = vcgpu.solve_batch(W.pack([g] * count), "mvc", time_limit=TL)
            assert st == vcgpu.VC_OK
            for s in sols:
                _ok(g, s, alone.size)
        st, sols = vcgpu.solve_batch(W.pack([g] * 3), "pvc", ks=[alone.size, alone.size - 1, alone.size], time_limit=TL)
        assert st == vcgpu.VC_OK and [s.decision for s in sols] == [1, 0, 1]
