"""The bounded wait of the whole-try kernels' exchange (records.cuh, poll16),
from a one-warp kernel over the library's own header: a record with the right
tag is returned whole; one that never comes ends the wait after its read limit,
about a second, with NaN, RED_ERR_TIMEOUT and the halted flag on the system,
and the CTA's later waits end at once.  The context stays usable."""
import ctypes as C
import os
import subprocess
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "red.cuda_gb300", "csrc")

SHIM = r'''
#include "records.cuh"
using namespace redgb;

__global__ void k_wait(uint4* rec, unsigned tag, DevSys* S, uint4* out, int* dead_out)
{
    __shared__ int dead;
    if (threadIdx.x == 0) dead = 0;
    __syncthreads();
    if (threadIdx.x == 0) st_rec16(rec, 11u, 22u, 33u, 7u);
    __syncthreads();
    out[threadIdx.x] = poll16(rec, tag, S, &dead);
    __syncthreads();
    out[32 + threadIdx.x] = poll16(rec, tag, S, &dead);
    if (threadIdx.x == 0) *dead_out = dead;
}

extern "C" int run_wait(unsigned tag, unsigned* out, int* status, int* halted, int* dead)
{
    uint4 *rec = nullptr, *o = nullptr;
    DevSys *S = nullptr, h;
    int* d = nullptr;
    cudaMalloc(&rec, sizeof(uint4));
    cudaMalloc(&o, 64 * sizeof(uint4));
    cudaMalloc(&S, sizeof(DevSys));
    cudaMalloc(&d, sizeof(int));
    cudaMemset(rec, 0, sizeof(uint4));
    cudaMemset(S, 0, sizeof(DevSys));
    k_wait<<<1, 32>>>(rec, tag, S, o, d);
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess) {
        cudaMemcpy(out, o, 64 * sizeof(uint4), cudaMemcpyDeviceToHost);
        cudaMemcpy(dead, d, sizeof(int), cudaMemcpyDeviceToHost);
        e = cudaMemcpy(&h, S, sizeof(DevSys), cudaMemcpyDeviceToHost);
        *status = h.status;
        *halted = h.halted;
    }
    cudaFree(rec);
    cudaFree(o);
    cudaFree(S);
    cudaFree(d);
    return (int)e;
}
'''


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("exchange")
    src = d / "shim.cu"
    src.write_text(SHIM)
    so = d / "shim.so"
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.check_call([nvcc, "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_103a,code=sm_103a",
                           "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-ftz=true",
                           "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-o", str(so), str(src)])
    return C.CDLL(str(so))


@pytest.mark.parametrize("tag", [7, 8])
def test_wait(shim, tag):
    out = np.zeros((64, 4), np.uint32)
    status, halted, dead = C.c_int(-1), C.c_int(-1), C.c_int(-1)
    for _ in range(2):   # the context is usable after a wait that ran out
        t0 = time.perf_counter()
        rc = shim.run_wait(C.c_uint(tag), out.ctypes.data_as(C.c_void_p), C.byref(status), C.byref(halted),
                           C.byref(dead))
        assert rc == 0 and time.perf_counter() - t0 < 30.0
        if tag == 7:
            assert np.array_equal(out, np.tile(np.array([11, 22, 33, 7], np.uint32), (64, 1)))
            assert (status.value, halted.value, dead.value) == (0, 0, 0)
        else:
            assert np.isnan(out[:, :3].copy().view(np.float32)).all() and (out[:, 3] == 0).all()
            assert (status.value, halted.value, dead.value) == (4, 1, 1)
