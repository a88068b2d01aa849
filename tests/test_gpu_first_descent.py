"""The packing bound is left out as long as all vertices may be taken; where the line
lies (k or a hint of n and n - 1) the answers are the oracle's."""
import pytest

import oracle as O
import vcgpu
from vcgpu import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p", [(12, 0.5), (33, 0.95), (50, 0.7), (65, 0.2), (70, 0.05), (200, 0.02), (300, 0.008)])
def test_bounds_of_n(n, p):
    g = W.gnp(n, p, n)
    st, opt, _, _ = O.mvc(g)
    assert st == O.OK
    assert vcgpu.solve(g).size == opt
    for k in (opt - 1, opt, n - 1, n, n + 1):
        assert vcgpu.solve(g, "mvc", ub=k).size == min(opt, k, n)
        r = vcgpu.solve(g, "pvc", k=k)
        assert r.status == vcgpu.VC_OK and r.decision == (1 if k >= opt else 0)
        if r.decision:
            assert W.is_cover(g, r.cover) and int(r.cover.sum()) == r.size <= k
    st, sols = vcgpu.solve_batch(W.pack([g] * 3), ["mvc", "pvc", "mvc"], ks=[0, opt - 1, 0], ubs=[0, 0, n])
    assert st == vcgpu.VC_OK and [s.size for s in sols] == [opt, 0, opt] and sols[1].decision == 0
