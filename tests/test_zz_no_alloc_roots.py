"""Graphs that have a launch to themselves, on both sides of the sizes and densities
from which they are searched from n roots: the allocation-free entry point and the
plain solve against the CPU oracle, and against a batch, which searches from one."""
import ctypes
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
TL = 60.0


def _noalloc(torch, g, instance, k=0, node_limit=0):
    f = vcgpu.lib().vc_solve_noalloc
    f.argtypes = [ctypes.POINTER(vcgpu.Csr), ctypes.POINTER(vcgpu.Request), ctypes.c_void_p, ctypes.c_void_p]
    f.restype = ctypes.c_int
    d_rp = torch.from_numpy(g.row_ptr.astype(np.int32)).cuda()
    d_col = torch.from_numpy(g.col.astype(np.int32)).cuda()
    res = torch.zeros(8, dtype=torch.int32, device="cuda")
    cover = torch.zeros(8, dtype=torch.int32, device="cuda")
    csr = vcgpu.Csr(g.n, g.m, d_rp.data_ptr(), d_col.data_ptr(), None)
    req = vcgpu._request(instance, k, 0, node_limit, TL, vcgpu.VC_FLAG_DEVICE_INPUT, -1, torch.cuda.current_stream().cuda_stream)
    assert f(ctypes.byref(csr), ctypes.byref(req), res.data_ptr(), cover.data_ptr()) == vcgpu.VC_OK
    torch.cuda.synchronize()
    words = cover.cpu().numpy().astype(np.uint32)
    return res.cpu().numpy(), np.array([(words[v >> 5] >> (v & 31)) & 1 for v in range(g.n)], dtype=bool)


@pytest.mark.parametrize("n", [15, 16, 17, 31, 32, 33, 63, 64, 65, 128, 129, 191, 192, 193, 255])
def test_roots_by_size_and_density(n):
    torch = pytest.importorskip("torch")
    tiny = W.gnp(8, 0.4, 3)
    graphs = [W.gnp(n, p, 7 * n) for p in (0.05, 0.14, 0.16, 0.3, 0.39, 0.42, 0.7, 0.95) if n < 190 or p < 0.1 or p > 0.3]
    graphs.append(W.from_edges(n, [(i, j) for i in range(n) for j in range(i)]))                              # complete
    graphs.append(W.from_edges(n, [(i, j) for i in range(n) for j in range(i) if i // 3 != j // 3]))          # parts of 3
    graphs.append(W.from_edges(n, [(i, j) for i in range(n // 2) for j in range(n // 2, n) if (i * j) % 3]))  # bipartite
    for g in graphs:
        if g.m == 0:
            continue
        st, sols = vcgpu.solve_batch(W.pack([g, tiny]), "mvc", time_limit=TL)
        assert st == vcgpu.VC_OK
        opt = sols[0].size
        if n <= 65:
            st, want, _, _ = O.mvc(g, node_limit=2_000_000)
            assert st != O.OK or want == opt
        r = vcgpu.solve(g, "mvc", time_limit=TL)
        assert r.status == vcgpu.VC_OK and r.size == opt and W.is_cover(g, r.cover) and int(r.cover.sum()) == opt
        out, mask = _noalloc(torch, g, "mvc")
        assert tuple(out[:4]) == (vcgpu.VC_OK, opt, 1, 1) and W.is_cover(g, mask) and int(mask.sum()) == opt
        for k, want in ((opt, 1), (opt - 1, 0), (n, 1)):
            p = vcgpu.solve(g, "pvc", k=k, time_limit=TL)
            assert p.status == vcgpu.VC_OK and p.decision == want
            out, mask = _noalloc(torch, g, "pvc", k)
            assert out[0] == vcgpu.VC_OK and out[2] == want
            if want:
                assert W.is_cover(g, mask) and int(mask.sum()) == out[1] <= k
    out, _ = _noalloc(torch, graphs[4 if n < 190 else 1], "mvc", node_limit=1)
    assert out[0] in (vcgpu.VC_OK, vcgpu.VC_BUDGET)
    out, _ = _noalloc(torch, g, "mvc")
    assert out[0] == vcgpu.VC_OK and out[1] == opt
