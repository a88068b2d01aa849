"""A search of the dense kernels stops close to its time limit, alone and in a batch."""
import pytest

import vcgpu
from vcgpu import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(250, 15.0), (640, 6.0), (1024, 6.0)])
def test_stops_close_to_its_limit(n, d):
    g = W.gnp(n, d / (n - 1), n + 1)
    r = vcgpu.solve(g, "mvc", time_limit=0.2)
    assert r.status == vcgpu.VC_TIMEOUT and 200.0 <= r.kernel_ms < 216.0
    st, sols = vcgpu.solve_batch(W.pack([g, g]), "mvc", time_limit=0.2)
    assert st == vcgpu.VC_TIMEOUT and 200.0 <= sols[0].kernel_ms < 216.0
    assert W.is_cover(g, sols[0].cover) and int(sols[0].cover.sum()) == sols[0].size
