"""A host-resident graph that is both invalid and above the vertex limit is invalid,
with few entries or many (the many are otherwise checked on the device); a valid one
is too large."""
import numpy as np

import vcgpu
from vcgpu import workloads as W

LIMIT = 1 << 26


def _star(n, m, bad):
    rp = np.full(n + 1, 2 * m, dtype=np.uint32)
    rp[0] = 0
    rp[1:m + 2] = m + np.arange(m + 1)
    col = np.zeros(2 * m, dtype=np.uint32)
    col[:m] = np.arange(1, m + 1)
    if bad:
        col[2 * m - 1] = m  # the last leaf's row names itself
    return W.Graph(n, rp, col)


def test_invalid_before_too_large():
    for m in (3, 1500):
        assert vcgpu.solve(_star(LIMIT + 1, m, True)).status == vcgpu.VC_ERR_INVALID
        assert vcgpu.solve(_star(LIMIT + 1, m, False)).status == vcgpu.VC_ERR_TOO_LARGE
