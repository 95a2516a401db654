"""The accept / reject decision of a whole try reaches every CTA whole.

* The exchange's two-word records (records.cuh, st_pair and poll_pair) in a ping-pong of
  many CTAs, the first word alternating as a decision's does: a reader never meets a
  new tag beside an old word, also where it needs the first word alone.  The three-word
  records (st_rec16 and poll16) beside them.
* Adaptive runs in which every second try or so is rejected: each body ends where its
  Kepler orbit has it at the handle's time.  The protoplanets and planetesimals have a
  mass of 1e-25, so that the star alone acts; RKF7(8) at a tolerance of 1e-10 keeps the
  orbits to far better than 1e-6, and a CTA that acts on the wrong decision leaves
  its bodies a step (>= 1e-2) away."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "red.cuda_gb300", "csrc")

SHIM = r'''
#include "records.cuh"
using namespace redgb;

// CTA 0 sends round n to everyone and waits for every answer; one cooperative launch
__global__ void k_rounds(uint4* word, uint4* three, uint4* answer, int rounds, DevSys* S, unsigned* wrong)
{
    __shared__ int dead;
    if (threadIdx.x == 0) dead = 0;
    __syncthreads();
    const int n_cta = gridDim.x - 1;
    for (int n = 1; n <= rounds; n++) {
        if (blockIdx.x == 0) {
            if (threadIdx.x == 0) st_pair(word, n & 1, 0u, n);
            if (threadIdx.x == 32) st_rec16(three, n, ~(unsigned)n, 5u * n, n);
            for (int j = threadIdx.x; j < n_cta; j += blockDim.x)
                if (poll_pair(answer + j, n, S, &dead).x != (unsigned)n * 3u) atomicAdd(wrong + 1, 1u);
        } else if (threadIdx.x == 32) {
            const uint4 v = poll16(three, n, S, &dead);
            if (v.x != (unsigned)n || v.y != ~(unsigned)n || v.z != 5u * n) atomicAdd(wrong + 2, 1u);
        } else if (threadIdx.x == 0) {
            if (poll_pair(word, n, S, &dead).x != (unsigned)(n & 1)) atomicAdd(wrong, 1u);
            st_pair(answer + blockIdx.x - 1, (unsigned)n * 3u, ~(unsigned)n, n);
        }
        __syncthreads();
        if (dead) break;
    }
}

extern "C" int run_rounds(int n_cta, int rounds, unsigned* wrong, int* status)
{
    uint4* rec = nullptr;
    DevSys *S = nullptr, h;
    unsigned* w = nullptr;
    cudaMalloc(&rec, (n_cta + 2) * sizeof(uint4));
    cudaMalloc(&S, sizeof(DevSys));
    cudaMalloc(&w, 3 * sizeof(unsigned));
    cudaMemset(rec, 0, (n_cta + 2) * sizeof(uint4));
    cudaMemset(S, 0, sizeof(DevSys));
    cudaMemset(w, 0, 3 * sizeof(unsigned));
    uint4 *three = rec + 1, *answer = rec + 2;
    void* args[] = {&rec, &three, &answer, &rounds, &S, &w};
    cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_rounds, dim3(n_cta + 1), dim3(64), args, 0, 0);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(wrong, w, 3 * sizeof(unsigned), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&h, S, sizeof(DevSys), cudaMemcpyDeviceToHost);
    *status = h.status;
    cudaFree(rec);
    cudaFree(S);
    cudaFree(w);
    return (int)e;
}
'''


def test_records_are_whole(tmp_path):
    src, so = tmp_path / "shim.cu", tmp_path / "shim.so"
    src.write_text(SHIM)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.check_call([nvcc, "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_103a,code=sm_103a",
                           "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-ftz=true",
                           "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-o", str(so), str(src)])
    wrong, status = (C.c_uint * 3)(), C.c_int(-1)
    assert C.CDLL(str(so)).run_rounds(140, 20000, wrong, C.byref(status)) == 0
    assert status.value == 0 and list(wrong) == [0, 0, 0]


def vec(a):
    return np.stack([a["x"], a["y"], a["z"]], axis=1)


def kepler(r, v, t):
    """The two-body orbits of unit mass after a time t."""
    d = np.linalg.norm(r, axis=1)
    a = 1.0 / (2.0 / d - np.sum(v * v, axis=1))
    n = a ** -1.5
    ec, es = 1.0 - d / a, np.sum(r * v, axis=1) / np.sqrt(a)   # e cos E, e sin E
    x = n * t                                                  # the change of E
    for _ in range(50):
        x -= (x - ec * np.sin(x) + es * (1.0 - np.cos(x)) - n * t) / (1.0 - ec * np.cos(x) + es * np.sin(x))
    f = 1.0 - a / d * (1.0 - np.cos(x))
    g = t + (np.sin(x) - x) / n
    return f[:, None] * r + g[:, None] * v


@pytest.mark.parametrize("precision", ["mixed", "fp32", "fp64"])
def test_rejections(rg, precision):
    rng = np.random.Generator(np.random.MT19937(3))
    s = rg.ic.build_system(rng, pp_a=np.linspace(0.75, 1.45, 4), pp_mass=1e-25, pl_a=rng.uniform(0.7, 1.5, 5000),
                           pl_mass=1e-25)
    for x in (s.r, s.v):
        for c in "xyz":
            x[c] -= x[c][0]
    with rg.Sim(s, integrator="rkf78", adaptive=True, tolerance=1e-10, dt=60.0 * rg.ic.K, precision=precision) as sim:
        before = sim.kernel_launches
        sim.launch_tries(1)
        sim.synchronize()
        assert sim.kernel_launches - before == 1
        passed = 0
        for _ in range(60):
            sim.launch_tries(1)
            sim.synchronize()
            i = sim.info(0)
            if i.n_passed != passed and i.n_passed % 2:   # after every second step one far too long
                sim.set_dt_next(0, 3.0 * i.dt_next)
            passed = i.n_passed
        o, i = sim.get_state(0), sim.info(0)
    assert i.status == 0 and i.n_failed >= 10 and i.n_passed >= 20
    err = np.linalg.norm(vec(o.r)[1:] - kepler(vec(s.r)[1:], vec(s.v)[1:], i.t), axis=1)
    assert err.max() < 1e-6, (err.max(), np.count_nonzero(err > 1e-6))
