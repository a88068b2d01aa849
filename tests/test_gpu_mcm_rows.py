"""vc_mcm on both sides of the rows that fit a CTA's shared memory (64 KB: the complete
graph of 127 vertices, not that of 128): both kernels find the matching."""
import numpy as np
import pytest

import vcgpu
from vcgpu import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [126, 127, 128, 129, 513, 1024])
def test_complete_graphs(n):
    i, j = np.triu_indices(n, 1)
    r = vcgpu.mcm(W.from_edges(n, np.stack([i, j], axis=1)), time_limit=30.0)
    assert r.status == vcgpu.VC_OK and r.size == 2 * (n // 2)


@pytest.mark.parametrize("n,d", [(1000, 15.0), (1000, 15.3), (1000, 15.5)])
def test_rows_just_below_and_above(n, d):
    """Perfect matchings planted where the rows take 63,940 to 65,956 bytes."""
    g = W.planted_matching(n, d, 7)
    r = vcgpu.mcm(g, time_limit=30.0)
    assert r.status == vcgpu.VC_OK and r.size == n
