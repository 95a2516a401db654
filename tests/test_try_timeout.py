"""A whole try in which a record of the exchange never comes (k_try, k_try64): the system
stops with RED_ERR_TIMEOUT, and its state, time and counters are those before the try, in
fixed and in adaptive steps, whichever record it is.

The kernels are compiled here from the library's own sources with a short read limit
and a sender that drops the records of one CTA with one tag; the rest of the library is
linked as it is.  Nothing waits longer than the limit, and the next handle in the same
process works."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "red.cuda_gb300")

SHIM = r'''
#define st_rec16 st_rec16_sent
#define st_pair st_pair_sent
#include "records.cuh"
#undef st_rec16
#undef st_pair
namespace redgb {
namespace {
__device__ int g_drop[2] = {-1, -1};   // the CTA and the tag within the try
__device__ __forceinline__ bool dropped(unsigned tag)
{
    return (int)blockIdx.x == g_drop[0] && (int)(tag & 15u) == g_drop[1];
}
__device__ __forceinline__ void st_rec16(uint4* p, unsigned x, unsigned y, unsigned z, unsigned tag)
{
    if (!dropped(tag)) st_rec16_sent(p, x, y, z, tag);
}
__device__ __forceinline__ void st_pair(uint4* p, unsigned lo, unsigned hi, unsigned tag)
{
    if (!dropped(tag)) st_pair_sent(p, lo, hi, tag);
}
}  // namespace
}  // namespace redgb
#include "%s.cu"
extern "C" int drop_%s(int cta, int tag)
{
    const int v[2] = {cta, tag};
    return (int)cudaMemcpyToSymbol(redgb::g_drop, v, sizeof(v));
}
'''

RUN = r'''
import ctypes, json, sys
import numpy as np
sys.path.insert(0, %(root)r)
import __graft_entry__
rg = __graft_entry__.load_package()
L = rg.lib.load(%(lib)r)
vec = lambda a: np.stack([a["x"], a["y"], a["z"]], axis=1)
rng = np.random.Generator(np.random.MT19937(5))
s = rg.ic.build_system(rng, pp_a=np.linspace(0.75, 1.45, 4), pp_mass=0.1 * rg.ic.EARTH_TO_SOLAR,
                       pl_a=rng.uniform(0.7, 1.5, 700), pl_mass=rg.ic.EARTH_TO_SOLAR / 700, cd=0.44)
out = []
for precision, integrator, adaptive, gas, cta, tag in json.load(sys.stdin):
    drop = L.drop_try64 if precision == "fp64" else L.drop_try
    g = rg.ic.gas_params(rg.ic.gas_disk_config3()) if gas else None
    with rg.Sim(s, integrator=integrator, adaptive=adaptive, tolerance=1e-6, dt=0.5 * rg.ic.K, precision=precision,
                gas=g, collision_factor=1.0) as sim:
        sim.launch_tries(1)   # one that goes well
        before = sim.kernel_launches
        sim.synchronize()
        r, v, i = vec(sim.get_state(0).r), vec(sim.get_state(0).v), sim.info(0)
        assert drop(cta, tag) == 0
        sim.launch_tries(3)
        code = 0
        try:
            sim.synchronize()
        except rg.lib.RedError as e:
            code = e.code
        assert drop(-1, -1) == 0
        o, j = sim.get_state(0), sim.info(0)
        same = np.array_equal(vec(o.r), r) and np.array_equal(vec(o.v), v)
        out.append([code, j.status, j.halted, bool(same), j.t == i.t, j.n_passed - i.n_passed, j.n_tried - i.n_tried,
                    j.n_failed - i.n_failed, j.dt_did == i.dt_did, j.dt_next == i.dt_next])
print(json.dumps(out))
'''

# (precision, integrator, adaptive, gas, CTA, tag): 700 small bodies in 22 CTAs (44 in FP64), 5 large ones.
# The partial sums of stage s have the tag s + 1 and the positions of stage s too; the errors 14.
CASES = []
for _p, _last in (("mixed", 21), ("fp32", 21), ("fp64", 43)):
    for _i, _a, _n in (("euler", False, 1), ("rk4", False, 4), ("rk4", True, 5), ("rkf78", True, 13)):
        CASES += [(_p, _i, _a, False, _last, 1), (_p, _i, _a, False, _last, _n), (_p, _i, _a, False, 1, _n),
                  (_p, _i, _a, False, 1, 14)]
        if _a:
            CASES += [(_p, _i, _a, False, _last, 14)]
CASES += [("mixed", "rkf78", True, True, 21, 1), ("mixed", "rkf78", True, True, 1, 3), ("mixed", "rk4", False, True, 21, 4)]


def test_missing_records(rg, tmp_path):
    rg.build()
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    arch = ["-gencode", "arch=compute_103a,code=sm_103a"]
    procs, objs = [], []
    for u in ("try", "try64"):
        src, obj = tmp_path / ("shim_%s.cu" % u), tmp_path / ("shim_%s.o" % u)
        src.write_text(SHIM % (u, u))
        objs.append(str(obj))
        procs.append(subprocess.Popen([nvcc, "-c", *arch, "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
                                       "--expt-relaxed-constexpr", "-ftz=true" if u == "try" else "-ftz=false",
                                       "-DREDGB_TRY_POLL_LIMIT=4096", "-I" + os.path.join(ROOT, "include"),
                                       "-I" + os.path.join(PKG, "csrc"), "-o", str(obj), str(src)]))
    assert [p.wait() for p in procs] == [0, 0]
    build = os.path.join(PKG, "_build")
    rest = [os.path.join(build, f) for f in sorted(os.listdir(build))
            if f.endswith(".o") and f not in ("try.cu.o", "try64.cu.o")]
    lib = str(tmp_path / "libredgb_short.so")
    subprocess.check_call([nvcc, "-shared", *arch, "-o", lib, *objs, *rest, "-lcudart"])
    p = subprocess.run([sys.executable, "-c", RUN % {"root": ROOT, "lib": lib}], input=json.dumps(CASES),
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    got = json.loads(p.stdout)
    bad = [(c, g) for c, g in zip(CASES, got) if g != [4, 4, 1, True, True, 0, 0, 0, True, True]]
    assert len(got) == len(CASES) and not bad, bad
