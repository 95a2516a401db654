"""red_step on an ensemble in which some systems need a second try: their states after
it, whole tries against one launch per stage (REDGB_TRY=0).

A rejected step's estimate E is many times the tolerance (the next step is ~1/10 of it:
E ~ 10^7 tol = 1e-3), and the paths' accelerations differ by ~1e-12, which is ~1e-13 in
the estimate (41/840 dt times four of them): the next step agrees to 1e-10 / 7, and so
does the time.  The positions agree to 1e-10 of the scale, as after an accepted step,
and to the motion in the difference of the times."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def vec(a):
    return np.stack([a["x"], a["y"], a["z"]], axis=1)


def disk(rg, n_pp, n_pl, seed):
    rng = np.random.Generator(np.random.MT19937(seed))
    return rg.ic.build_system(rng, pp_a=np.linspace(0.75, 1.45, n_pp), pp_mass=0.1 * rg.ic.EARTH_TO_SOLAR,
                              pl_a=rng.uniform(0.7, 1.5, n_pl), pl_mass=rg.ic.EARTH_TO_SOLAR / n_pl)


@pytest.mark.parametrize("n_sys", [1, 5])
def test_states_after_a_second_try(rg, monkeypatch, n_sys):
    systems = [disk(rg, 4, 200 + 300 * k, 70 + k) for k in range(n_sys)]
    dt = np.array([30.0, 0.5, 1.0, 40.0, 0.5])[:n_sys] * rg.ic.K
    out = []
    for whole in ("0", "1"):
        monkeypatch.setenv("REDGB_TRY", whole)
        with rg.Sim(systems, integrator="rkf78", adaptive=True, tolerance=1e-10, dt=dt) as sim:
            sim.step()
            out.append([(sim.info(k), vec(sim.get_state(k).r), vec(sim.get_state(k).v)) for k in range(n_sys)])
    for k, ((i0, r0, v0), (i1, r1, v1)) in enumerate(zip(*out)):
        assert (i1.n_passed, i1.n_failed) == (i0.n_passed, i0.n_failed)
        assert i0.n_failed > 0 or dt[k] < 20.0 * rg.ic.K
        assert abs(i1.t - i0.t) <= 1e-10 * i0.t
        shift = 1.01 * np.linalg.norm(v0, axis=1).max() * abs(i1.t - i0.t)
        assert np.linalg.norm(r1 - r0, axis=1).max() <= 1e-10 * np.abs(r0).max() + shift
        assert np.linalg.norm(v1 - v0, axis=1).max() <= 1e-10 * np.abs(v0).max() + 10.0 * shift
