"""Bitmap rows of graphs with hubs: whether a vertex lies on a triangle is found along
its neighbours' rows, by a lane each or, for long ones, by the warp."""
import numpy as np
import pytest

import vcgpu
from vcgpu import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [34, 35, 36, 66, 130, 255, 300, 640, 1000, 1024])
@pytest.mark.parametrize("place", ["first", "middle", "last"])
def test_triangles_on_two_hubs(n, place):
    """Every other vertex hangs on both of two joined hubs, so its triangle shows only in their rows (n - 1 entries,
    where 32 are the most that one lane walks).  The triangle rule takes both at the root: the tree is one node."""
    a = {"first": 0, "middle": n // 2, "last": n - 2}[place]
    others = [v for v in range(n) if v not in (a, a + 1)]
    g = W.from_edges(n, np.array([(a, a + 1)] + [(h, v) for v in others for h in (a, a + 1)]))
    r = vcgpu.solve(g)
    assert (r.status, r.size, r.tree_nodes) == (vcgpu.VC_OK, 2, 1)
    assert r.cover[a] and r.cover[a + 1]


@pytest.mark.parametrize("n", [2, 3, 33, 34, 255, 600, 1024])
def test_stars(n):
    """Leaves do not walk the hub's row: with 1000 of them, one lane each, that took the kernels 0.6 ms."""
    g = W.from_edges(n, np.array([(n - 1, v) for v in range(n - 1)]))
    runs = [vcgpu.solve(g) for _ in range(5)]
    assert all(r.status == vcgpu.VC_OK and r.size == 1 for r in runs)
    assert min(r.kernel_ms for r in runs) < 0.3
