"""Device-resident graphs of more than 1024 vertices whose edges are partly in one
direction only: a wrong answer is allowed, an access outside an array is not.  The
root's reduction finds that rows and degrees part, leaves the rest alone and the
graph is searched as it is; graphs beside it keep their answers."""
import numpy as np
import pytest

import vcgpu
from vcgpu import workloads as W

pytestmark = pytest.mark.gpu
TL = 3.0


def _rows(n, rows):
    if sum(map(len, rows)) % 2:  # the caller states half of the entries
        rows[n - 1].add(0)
    rp = np.zeros(n + 1, dtype=np.uint32)
    rp[1:] = np.cumsum([len(r) for r in rows])
    return W.Graph(n, rp, np.array([u for r in rows for u in sorted(r)], dtype=np.uint32))


def _cycle(n, m):
    rows = [set() for _ in range(n)]
    for i in range(m):
        rows[i] |= {(i + 1) % m, (i - 1) % m}
    return rows


def _to_empty(n):
    """A long cycle (its vertices stay) whose rows also list vertices that have no row."""
    rows = _cycle(n, 1300)
    for i in range(0, 1300, 3):
        rows[i].add(1400 + i % 700)
    return _rows(n, rows)


def _taken_down(n):
    """Vertices that are taken (each has a leaf) list cycle vertices that do not list them."""
    rows = _cycle(n, 1300)
    for j in range(40):
        hub, leaf = 1400 + 2 * j, 1401 + 2 * j
        rows[hub] |= {leaf} | {(17 * j + 100 * i) % 1300 for i in range(6)}
        rows[leaf].add(hub)
    return _rows(n, rows)


def _lists_taken(n):
    """Cycle vertices list vertices that are taken and do not list them: fewer entries are left than the degree."""
    rows = _cycle(n, 1300)
    for j in range(40):
        hub, leaf = 1400 + 2 * j, 1401 + 2 * j
        rows[hub].add(leaf)
        rows[leaf].add(hub)
        for i in range(6):
            rows[(17 * j + 100 * i) % 1300].add(hub)
    return _rows(n, rows)


def _directed(n):
    rng = np.random.default_rng(n)
    return _rows(n, [set(int(u) for u in rng.integers(0, n, rng.integers(1, 4)) if u != v) for v in range(n)])


@pytest.mark.parametrize("n", [2177, 3000])
@pytest.mark.parametrize("make", [_to_empty, _taken_down, _lists_taken, _directed])
def test_one_directional_rows_are_searched_as_they_are(make, n):
    torch = pytest.importorskip("torch")
    g = make(n)
    d_rp = torch.from_numpy(g.row_ptr.view(np.int32)).cuda()
    d_col = torch.from_numpy(g.col.view(np.int32)).cuda()
    torch.cuda.synchronize()
    for instance, k in (("mvc", 0), ("pvc", n // 2)):
        r = vcgpu.solve_device(n, g.m, d_rp.data_ptr(), d_col.data_ptr(), instance, k=k, time_limit=TL)
        assert r.status in (vcgpu.VC_OK, vcgpu.VC_TIMEOUT)
        assert int(vcgpu.debug_stats()[1][4]) >= n  # the kernel for n vertices, not for a rest
    good = [W.config1_graph(), W.planted_cover(2000, 300, 6000, 100, 4, 9), W.from_edges(n, [(i, (i + 1) % n) for i in range(n)])]
    want = [vcgpu.solve(x).size for x in good]
    arena = W.pack([good[0], g, good[1], good[2]])
    d_rp = torch.from_numpy(arena.row_ptr.view(np.int32)).cuda()
    d_col = torch.from_numpy(arena.col.view(np.int32)).cuda()
    torch.cuda.synchronize()
    _, sols = vcgpu.solve_batch(arena, time_limit=TL, d_row_ptr=d_rp.data_ptr(), d_col=d_col.data_ptr())
    assert sols[1].status in (vcgpu.VC_OK, vcgpu.VC_TIMEOUT)
    assert [sols[i].size for i in (0, 2, 3)] == want
    for i, x in ((0, good[0]), (2, good[1]), (3, good[2])):
        assert sols[i].status == vcgpu.VC_OK and W.is_cover(x, sols[i].cover)
