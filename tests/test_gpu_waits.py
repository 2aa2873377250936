"""A CTA's bounded wait ends the same way in all its threads: one thread that ran out is reported by every thread, so the
thread that reports a failed copy sees it and no warp diverges."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from multigridsoftbody_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "kernels_mlp.cuh"
using namespace mgsb;
// late: the thread whose wait may not poll at all (none: -1); the phase is complete before the wait.
__global__ void wait_all(int late, int* out) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(&bar, 0);
    }
    __syncthreads();
    out[threadIdx.x] = cta_wait(&bar, 0, (int)threadIdx.x == late ? 0 : 1 << 16);
}
extern "C" int run(int late, int threads, int* out) {
    int* d = nullptr;
    if (cudaMalloc(&d, threads * sizeof(int))) return 1;
    wait_all<<<1, threads>>>(late, d);
    const int e = cudaMemcpy(out, d, threads * sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("waits"))
    src, out = os.path.join(d, "waits.cu"), os.path.join(d, "waits.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build._nvcc(), *build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I" + build.CSRC, "-shared",
                    "-Xcompiler", "-fPIC", "-o", out, src], check=True, capture_output=True)
    return C.CDLL(out).run


@pytest.mark.parametrize("threads", [64, 96, 512])
@pytest.mark.parametrize("late", ["none", 0, 1, 33, "last"])
def test_one_late_thread_is_everyones(run, threads, late):
    late = {"none": -1, "last": threads - 1}.get(late, late)
    out = np.full(threads, -1, np.int32)
    assert run(late, threads, out.ctypes.data_as(C.POINTER(C.c_int))) == 0
    assert (out == 0).all() if late >= 0 else (out != 0).all()
