"""Batches of many graphs of more than 1024 vertices: their roots are reduced side by
side, a cluster of CTAs each (sizes around a cluster's threads, rows longer than a lane
walks, cascades longer than the pass limit), a very large one among them by the whole
chip; host-resident and device-resident, against known optima and the plain solve."""
import numpy as np
import pytest

import vcgpu
from vcgpu import workloads as W

pytestmark = pytest.mark.gpu
TL = 60.0


def _relabel(n, edges, seed):
    perm = np.random.default_rng(seed).permutation(n)
    return W.from_edges(n, perm[np.asarray(edges, dtype=np.int64).reshape(-1, 2)])


def _pool():
    out = []  # (graph, optimum)
    for n in (1025, 1535, 1537, 2048, 2049, 4096, 4097):
        out.append((_relabel(n, [(i, i + 1) for i in range(n - 1)], n), n // 2))
        out.append((_relabel(n, [(i, (i + 1) % n) for i in range(n)], n + 1), (n + 1) // 2))
    for n in (1300, 2500):  # stars whose hubs have rows of 63, 64, 65 and the rest of the vertices
        edges, at = [], 0
        for k in (63, 64, 65, n - 196):
            edges += [(at, at + j) for j in range(1, k + 1)]
            at += k + 1
        out.append((_relabel(n, edges, n + 2), 4))
    out.append((W.from_edges(1100, np.zeros((0, 2))), 0))
    graphs = [W.planted_cover(n, n * 3 // 20, 3 * n, n // 20, 4, n) for n in (1200, 2000)]
    graphs += [W.gnp(n, 2.6 / n, n) for n in (1030, 1700, 3000)] + [W.chung_lu(5000, 2.1, 8.0, 2000.0, 3)]
    for g in graphs:
        r = vcgpu.solve(g, "mvc", time_limit=TL)
        assert r.status == vcgpu.VC_OK
        out.append((g, r.size))
    return out


@pytest.mark.parametrize("count,large", [(2, 0), (3, 20000), (5, 0), (23, 0), (41, 60000), (80, 0), (300, 0)])
def test_many_large_graphs(count, large):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(count)
    pool = _pool()
    pick = [pool[i] for i in (range(count) if count <= len(pool) else rng.integers(0, len(pool), count))]
    if large:
        g = W.chung_lu(large, 2.1, 8.0, 2000.0, 11)
        pick.insert(count // 2, (g, vcgpu.solve(g, "mvc", time_limit=TL).size))
    small = W.config1_graph()
    pick.insert(1, (small, vcgpu.solve(small).size))
    graphs, opts = [g for g, _ in pick], [o for _, o in pick]
    arena = W.pack(graphs)
    d_rp = torch.from_numpy(arena.row_ptr.view(np.int32)).cuda()
    d_col = torch.from_numpy(arena.col.view(np.int32)).cuda()
    torch.cuda.synchronize()
    for where in ({}, {"d_row_ptr": d_rp.data_ptr(), "d_col": d_col.data_ptr()}, {"validate": False}):
        st, sols = vcgpu.solve_batch(arena, "mvc", time_limit=TL, **where)
        assert st == vcgpu.VC_OK
        for g, s, opt in zip(graphs, sols, opts):
            assert s.status == vcgpu.VC_OK and s.size == opt and int(s.cover.sum()) == opt and W.is_cover(g, s.cover)
    for shift, want in ((0, 1), (-1, 0)):
        st, sols = vcgpu.solve_batch(arena, "pvc", ks=[max(o + shift, 0) for o in opts], time_limit=TL)
        assert st == vcgpu.VC_OK
        for g, s, opt in zip(graphs, sols, opts):
            if opt or not shift:
                assert s.decision == want
            if s.decision:
                assert W.is_cover(g, s.cover) and int(s.cover.sum()) == s.size <= max(opt + shift, 0)


def test_broken_large_graphs_in_a_device_batch():
    """Only the graphs that break the layout are refused; the others keep their answers."""
    torch = pytest.importorskip("torch")
    pool = _pool()[:20]
    arena = W.pack([g for g, _ in pool])
    col = arena.col.copy()
    bad = [0, 7, 15]
    for i in bad:
        col[int(arena.col_off[i]) + 1] = int(arena.n[i]) + 3
    d_rp = torch.from_numpy(arena.row_ptr.view(np.int32)).cuda()
    d_col = torch.from_numpy(col.view(np.int32)).cuda()
    torch.cuda.synchronize()
    st, sols = vcgpu.solve_batch(arena, "mvc", time_limit=TL, d_row_ptr=d_rp.data_ptr(), d_col=d_col.data_ptr())
    assert st == vcgpu.VC_ERR_INVALID
    for i, ((g, opt), s) in enumerate(zip(pool, sols)):
        if i in bad:
            assert s.status == vcgpu.VC_ERR_INVALID
        else:
            assert s.status == vcgpu.VC_OK and s.size == opt and W.is_cover(g, s.cover)
