"""The upper-bound heuristics report the first graph that is at fault: an invalid graph
before one above the vertex limit makes the call invalid, after it too large."""
import ctypes

import numpy as np
import pytest

import vcgpu
from vcgpu import workloads as W

LIMIT = 1 << 26


def _status(graphs, entry):
    arena = W.pack([W.Graph(g.n, g.row_ptr, g.col) for g in graphs])
    ub = np.zeros(len(graphs), dtype=np.uint32)
    a = vcgpu._arena_struct(arena)
    p = ub.ctypes.data_as(ctypes.c_void_p)
    if entry == "max":
        return vcgpu.lib().vc_remove_max_ub(ctypes.byref(a), -1, p, None, None)
    return vcgpu.lib().vc_remove_edge_ub(ctypes.byref(a), 1, -1, p, None, None)


@pytest.mark.parametrize("entry", ["max", "edge"])
def test_first_fault_counts(entry):
    bad = W.Graph(3, np.array([0, 1, 2, 2], dtype=np.uint32), np.array([1, 2], dtype=np.uint32))  # 1 lists 2, 2 nothing
    large = W.Graph(LIMIT + 1, np.zeros(LIMIT + 2, dtype=np.uint32), np.zeros(0, dtype=np.uint32))
    assert _status([bad, large], entry) == vcgpu.VC_ERR_INVALID
    assert _status([large, bad], entry) == vcgpu.VC_ERR_TOO_LARGE
