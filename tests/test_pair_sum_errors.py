"""All-pairs gravity with each pair formed once (k_pairs) in MIXED is no less accurate than
the one-sided tiles (REDGB_PAIRS=0): the median over the bodies of the relative error of
an acceleration against FP64_EXACT, in a field of protoplanets and in a cube of unit
masses, both without a star.  An Euler step of 1e6 time units gives the acceleration.

The two medians are of the same ~18000 bodies; either is good to 1.25 / sqrt(18000)
= 0.9 % of the errors' spread, which is about the median, so 3 % is beyond chance.
(FP32 sums of 32 terms are 10 % worse here.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = 1.0e6


def vec(a):
    return np.stack([a["x"], a["y"], a["z"]], axis=1)


def field(rg, n, seed):
    rng = np.random.Generator(np.random.MT19937(seed))
    s = rg.ic.build_system(rng, pp_a=np.linspace(0.75, 1.45, 16), pp_mass=0.1 * rg.ic.EARTH_TO_SOLAR,
                           pl_a=rng.uniform(0.7, 1.5, n - 16), pl_mass=rg.ic.EARTH_TO_SOLAR / n)
    md = s.md[1:].copy()
    md["body_type"] = rg.types.PROTOPLANET
    return rg.types.System(s.r[1:], s.v[1:], s.p[1:], md, np.array([0, 0, 0, n, 0, 0, 0], np.uint32))


def cube(rg, n, seed):
    rng = np.random.default_rng(seed)
    r, v, p, md = (np.zeros(n, t) for t in (rg.types.VAR4, rg.types.VAR4, rg.types.PARAM, rg.types.BMD))
    for k in "xyz":
        r[k] = rng.uniform(-50.0, 50.0, n)
    p["mass"], p["radius"], p["density"] = 1.0, 1e-3, 1.0
    md["body_type"], md["id"] = rg.types.PROTOPLANET, np.arange(1, n + 1)
    return rg.types.System(r, v, p, md, np.array([0, 0, 0, n, 0, 0, 0], np.uint32))


def acceleration(rg, s, precision):
    with rg.Sim(s, integrator="euler", adaptive=False, dt=DT, precision=precision) as sim:
        before = sim.kernel_launches
        sim.launch_tries(1)
        sim.synchronize()
        launches = sim.kernel_launches - before
        return vec(sim.get_state(0).v) / DT, launches


@pytest.mark.parametrize("make", [field, cube])
def test_median_error(rg, monkeypatch, make):
    err, n_launch = {"0": [], "1": []}, {}
    for seed in range(3):
        s = make(rg, 6000, seed)
        ref, _ = acceleration(rg, s, "fp64_exact")
        for once in err:
            monkeypatch.setenv("REDGB_PAIRS", once)
            a, n_launch[once] = acceleration(rg, s, "mixed")
            err[once].append(np.linalg.norm(a - ref, axis=1) / np.linalg.norm(ref, axis=1))
    assert n_launch["1"] == n_launch["0"] + 1   # the pair kernel before the stage
    tiles, once = (np.median(np.concatenate(err[k])) for k in "01")
    print("median relative error: one-sided tiles %.3e, each pair once %.3e" % (tiles, once))
    assert once <= 1.03 * tiles
