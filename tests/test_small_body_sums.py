"""The whole-try kernels' FP32 sums over the protoplanets are no less accurate than one
launch per stage's (REDGB_TRY=0): the median over the planetesimals of the relative
error of an acceleration against FP64_EXACT, in disks without a star, whose
acceleration is the pair terms alone.  An Euler step of 1e6 time units gives it.

The two medians are of the same ~20000 bodies; either is good to 1.25 / sqrt(20000)
= 0.9 % of the errors' spread, which is about the median, so 3 % is beyond chance.
(FP32 sums of eight terms are 5 and 10 % worse here.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = 1.0e6


def vec(a):
    return np.stack([a["x"], a["y"], a["z"]], axis=1)


def disk(rg, n_pp, n_pl, seed):
    rng = np.random.Generator(np.random.MT19937(seed))
    s = rg.ic.build_system(rng, pp_a=np.linspace(0.75, 1.45, n_pp), pp_mass=0.1 * rg.ic.EARTH_TO_SOLAR,
                           pl_a=rng.uniform(0.7, 1.5, n_pl), pl_mass=rg.ic.EARTH_TO_SOLAR / n_pl)
    n = s.n - 1
    return rg.types.System(s.r[1:], s.v[1:], s.p[1:], s.md[1:], np.array([0, 0, 0, n_pp, 0, n - n_pp, 0], np.uint32))


def accelerations(rg, systems, precision):
    with rg.Sim(systems, integrator="euler", adaptive=False, dt=DT, precision=precision) as sim:
        before = sim.kernel_launches
        sim.launch_tries(1)
        sim.synchronize()
        launches = sim.kernel_launches - before
        return [vec(sim.get_state(k).v) / DT for k in range(len(systems))], launches


@pytest.mark.parametrize("n_pp,sizes", [(16, [20000]), (8, [130 + 97 * k for k in range(16)])])
def test_median_error(rg, monkeypatch, n_pp, sizes):
    err = {"0": [], "1": []}
    for seed in range(1 if len(sizes) == 1 else 2):
        systems = [disk(rg, n_pp, n, 100 * seed + k) for k, n in enumerate(sizes)]
        ref, _ = accelerations(rg, systems, "fp64_exact")
        for whole in err:
            monkeypatch.setenv("REDGB_TRY", whole)
            acc, launches = accelerations(rg, systems, "mixed")
            assert (launches == 1) == (whole == "1")
            for a, e in zip(acc, ref):
                err[whole].append(np.linalg.norm(a - e, axis=1)[n_pp:] / np.linalg.norm(e, axis=1)[n_pp:])
    stages, whole = (np.median(np.concatenate(err[k])) for k in "01")
    print("median relative error: stages %.3e, whole tries %.3e" % (stages, whole))
    assert whole <= 1.03 * stages
