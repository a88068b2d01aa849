"""A wait on the global ring that runs out (a record that is never published, a slot
that is never given back): it ends by itself, the launch is marked as stopped by the
ring whatever the time limit says later, and that is an internal error, not the
caller's time limit."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(REPO, "parallel-vertex-cover-algorithms-on-gpus_b200")

SRC = r"""
#include <cstdio>
#include <cstring>
#include <cuda_runtime.h>
#include "vc_host.h"
#include "vc_search.cuh"
using namespace vcg;

__global__ void k_waits(Params P, int what, int *got)
{
    unsigned long long pos = 0;
    if (what == 0) *got = ring_claim_deq(P, pos);       // counted as published, but it is not
    else if (what == 1) *got = ring_claim_enq(P, pos);  // the slot has not come back
    else *got = 0;
    stop_launch(P, kStopTime);
}

int main()
{
    unsigned long long *ctl, *seq;
    int *got;
    cudaMallocManaged(&ctl, 8 * kCtlWords);
    cudaMallocManaged(&seq, 8 * 64);
    cudaMallocManaged(&got, 4);
    for (int what = 0; what < 3; ++what) {
        memset(ctl, 0, 8 * kCtlWords);
        for (int i = 0; i < 64; ++i) seq[i] = i;
        if (what == 0) ctl[kAvail] = 1;
        if (what == 1) seq[0] = 1;
        Params P;
        memset(&P, 0, sizeof(P));
        P.ctl = ctl;
        P.pool_seq = seq;
        P.q_mask = 63;
        *got = -1;
        k_waits<<<1, 1>>>(P, what, got);
        if (cudaDeviceSynchronize() != cudaSuccess) return 1;
        printf("%d %llu %d\n", *got, ctl[kAbort], (int)vch::stopped_status(ctl[kAbort]));
    }
    return 0;
}
"""


def test_ring_wait_that_runs_out(tmp_path):
    vcgpu = pytest.importorskip("vcgpu")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "waits.cu", tmp_path / "waits"
    src.write_text(SRC)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-I" + os.path.join(PKG, "csrc"),
                    "-I" + os.path.join(REPO, "include"), "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.split("\n")
    assert out[:3] == [f"0 2 {vcgpu.VC_ERR_INTERNAL}", f"0 2 {vcgpu.VC_ERR_INTERNAL}", f"0 1 {vcgpu.VC_TIMEOUT}"]
