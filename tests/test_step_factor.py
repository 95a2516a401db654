"""The step-size factor (tol / err)^(1/order) of the step control (control.cuh).

inverse_root: an FP32 power z of the root's exponent, error e <= 4 ulp of FP32, then a
third-order step on t = 1 - x z^n, |t| <= n e.  What the step leaves is (n + 1)(2 n + 1) /
(6 n^3) t^3 < 1e-18; x z^n carries at most three roundings of 2^-53, which come to 3/7
of one in the root (n = 7), and the last fma adds half an ulp: 1 ulp at most.  The
orders of the schemes (1, 2, 4, 7), the whole range and its edges, against extended
precision; and no less exact than the library's pow(tol / err, 1 / order), which other
arguments take.

control_system: dt_next = 0.9 dt factor on both sides of the range's ends, within 4 ulp
(the quotient's rounding over the order, the factor's ulp, two products; the library's pow
is good to 2 ulp, and the rounded exponent 1 / order costs it |ln x| / order 2^-53 / 2)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "red.cuda_gb300", "csrc")

SHIM = r'''
#include "control.cuh"
using namespace redgb;

__global__ void k_root(const double* x, int n, int order, double* root, double* lib)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    root[i] = inverse_root(x[i], order);
    lib[i] = pow(1.0 / x[i], 1.0 / (double)order);
}
__global__ void k_step(const double* err, int n, int order, double tol, double dt, double* dt_next)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    ControlParams P = {};
    P.adaptive = 1;
    P.order = order;
    P.lambda = 1.0;
    P.tolerance = tol;
    DevSys S = {};
    S.dt_try = dt;
    S.active = 1;
    control_system(P, S, (unsigned long long)__double_as_longlong(err[i]));
    dt_next[i] = S.dt_next;
}

extern "C" int run(int which, const double* a, int n, int order, double tol, double dt, double* o0, double* o1)
{
    double *d = nullptr, *r0 = nullptr, *r1 = nullptr;
    cudaMalloc(&d, n * sizeof(double));
    cudaMalloc(&r0, n * sizeof(double));
    cudaMalloc(&r1, n * sizeof(double));
    cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice);
    if (which == 0) k_root<<<(n + 127) / 128, 128>>>(d, n, order, r0, r1);
    else k_step<<<(n + 127) / 128, 128>>>(d, n, order, tol, dt, r0);
    cudaMemcpy(o0, r0, n * sizeof(double), cudaMemcpyDeviceToHost);
    if (which == 0) cudaMemcpy(o1, r1, n * sizeof(double), cudaMemcpyDeviceToHost);
    const cudaError_t e = cudaDeviceSynchronize();
    cudaFree(d);
    cudaFree(r0);
    cudaFree(r1);
    return (int)e;
}
'''


@pytest.fixture(scope="module", params=["-ftz=true", "-ftz=false"])   # try.cu's and kernels.cu's
def run(request, tmp_path_factory):
    d = tmp_path_factory.mktemp("factor")
    src, so = d / "shim.cu", d / "shim.so"
    src.write_text(SHIM)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.check_call([nvcc, "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_103a,code=sm_103a",
                           "-O3", "-std=c++17", "--expt-relaxed-constexpr", request.param,
                           "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-o", str(so), str(src)])
    lib = C.CDLL(str(so))

    def call(which, a, order, tol=0.0, dt=0.0):
        a = np.ascontiguousarray(a, np.float64)
        o0, o1 = np.zeros_like(a), np.zeros_like(a)
        p = [x.ctypes.data_as(C.c_void_p) for x in (a, o0, o1)]
        assert lib.run(which, p[0], len(a), order, C.c_double(tol), C.c_double(dt), p[1], p[2]) == 0
        return o0, o1

    return call


def ulps(got, exact):
    """Errors in units in the last place of the exact values (extended precision)."""
    return np.abs(got.astype(np.longdouble) - exact) / np.spacing(exact.astype(np.float64)).astype(np.longdouble)


def exact_root(x, order):
    return np.exp2(-np.log2(x.astype(np.longdouble)) / order)


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 100, reason="needs quadruple precision on the host")
@pytest.mark.parametrize("order", [1, 2, 4, 7])
def test_inverse_root(run, order):
    rng = np.random.default_rng(order)
    x = np.concatenate([10.0 ** rng.uniform(-30, 30, 20000), 10.0 ** rng.uniform(-3, 1, 20000),
                        1.0 + rng.uniform(-1e-6, 1e-6, 2000),
                        np.nextafter([1e-30, 1e30, 1.0, 1.0, 2.0, 128.0], [1.0, 1.0, 0.0, 2.0, 0.0, 0.0]),
                        [1.0, 2.0, 4.0, 128.0, 0.5, 2.0 ** -99, 2.0 ** 99]])
    root, lib = run(0, x, order)
    e, f = ulps(root, exact_root(x, order)), ulps(lib, exact_root(x, order))
    print("order %d: largest error %.3f ulp, pow %.3f ulp" % (order, e.max(), f.max()))
    assert e.max() <= 1.0 and e.max() <= f.max()


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 100, reason="needs quadruple precision on the host")
@pytest.mark.parametrize("order", [1, 2, 4, 7])
def test_step_at_the_ends_of_the_range(run, order):
    tol, dt = 2.0 ** -33, 2.0 ** -6
    x = np.array([1e-31, 0.99e-30, 1e-30, 1.01e-30, 1e-29, 1e-3, 0.999, 1.0, 1.001, 1e3, 1e29, 0.99e30, 1e30, 1.01e30, 1e31])
    err = x * tol / dt   # lambda = 1; exact in these powers of two
    got, _ = run(1, err, order, tol, dt)
    exact = np.longdouble(0.9) * np.longdouble(dt) * exact_root(x, order)
    slack = 4.0 + np.where((x <= 1e-30) | (x >= 1e30), np.abs(np.log(x)) / order / 2 * 2, 0.0)
    assert np.all(ulps(got, exact) <= slack)
    # an error of nothing doubles the step
    assert run(1, np.zeros(1), order, tol, dt)[0][0] == 2.0 * dt
