"""A try as one cooperative launch (the default for one sparse system in the
FP32 modes) against one launch per stage (REDGB_TRY=0), which the other tests
hold to the oracle: every scheme, with gas drag, inactive bodies, without a
star, sizes at the edges of the launch's shape (one small body, one CTA's 32,
a ragged last CTA, parts of one to four, the largest number of large bodies,
one body more than that).

Tolerance: the two paths share the double-single star term and the FP32 pair
terms and differ in the order of FP32 sums (~1e-7 of the pair terms, which are
<= 1e-3 of an acceleration here) and in the rounding of the FP64 stage sums; a
step moves a velocity by dt a <= 0.1, so a few steps stay within 1e-10 of the
scale."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def vec(a):
    return np.stack([a["x"], a["y"], a["z"]], axis=1)


def disk(rg, n_pp, n_pl, seed=5, cd=0.0):
    rng = np.random.Generator(np.random.MT19937(seed))
    return rg.ic.build_system(rng, pp_a=np.linspace(0.75, 1.45, n_pp), pp_mass=0.1 * rg.ic.EARTH_TO_SOLAR,
                              pl_a=rng.uniform(0.7, 1.5, n_pl), pl_mass=rg.ic.EARTH_TO_SOLAR / max(n_pl, 1), cd=cd)


def run(rg, s, monkeypatch, whole, tries, **kw):
    monkeypatch.setenv("REDGB_TRY", "1" if whole else "0")
    with rg.Sim(s, **kw) as sim:
        before = sim.kernel_launches
        sim.launch_tries(tries)
        sim.synchronize()
        out = sim.get_state(0)
        return vec(out.r), vec(out.v), sim.info(0), sim.kernel_launches - before


def check(rg, s, monkeypatch, tries=3, whole_used=True, **kw):
    kw = dict(dict(dt=0.5 * rg.ic.K, collision_factor=1.0), **kw)
    r0, v0, i0, n0 = run(rg, s, monkeypatch, False, tries, **kw)
    r1, v1, i1, n1 = run(rg, s, monkeypatch, True, tries, **kw)
    assert (n1 < n0) == whole_used, (n0, n1)
    assert (i1.n_passed, i1.n_tried, i1.halted, i1.status) == (i0.n_passed, i0.n_tried, i0.halted, i0.status)
    assert i1.t == i0.t
    assert np.abs(r1 - r0).max() <= 1e-10 * np.abs(r0).max()
    assert np.abs(v1 - v0).max() <= 1e-10 * np.abs(v0).max()
    return i0, i1


@pytest.mark.parametrize("integrator", ["euler", "rk2", "rk4", "rkf78"])
@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_fixed_step_schemes(rg, monkeypatch, integrator, precision):
    check(rg, disk(rg, 4, 700), monkeypatch, integrator=integrator, adaptive=False, precision=precision,
          whole_used=True)


@pytest.mark.parametrize("integrator,tol", [("rk4", 1e-6), ("rkf78", 1e-10)])
def test_adaptive_schemes(rg, monkeypatch, integrator, tol):
    i0, i1 = check(rg, disk(rg, 8, 3000), monkeypatch, tries=1, integrator=integrator, adaptive=True, tolerance=tol)
    assert i0.n_passed == 1
    # a step far too long: rejected by both, the state untouched
    s = disk(rg, 8, 3000)
    for whole in (False, True):
        r, v, i, _ = run(rg, s, monkeypatch, whole, 1, integrator=integrator, adaptive=True, tolerance=tol,
                         dt=60.0 * rg.ic.K)
        assert i.n_passed == 0 and i.dt_next < 60.0 * rg.ic.K
        assert np.array_equal(r, vec(s.r)) and np.array_equal(v, vec(s.v))


@pytest.mark.parametrize("integrator,dt,tol", [("rk4", 0.5, 1e-6), ("rkf78", 1.5, 1e-10)])
def test_error_estimate(rg, monkeypatch, integrator, dt, tol):
    """At a step whose estimate is the method's error, ~0.1 of the tolerance or
    more: the rounding noise of the stage accelerations (2e-14, times lambda dt)
    is ~1e-5 of it or less, so the next step agrees to 1e-4."""
    s = rg.ic.config2(seed=3, n_pp=8, n_pl=3000)
    i = [run(rg, s, monkeypatch, whole, 1, integrator=integrator, adaptive=True, tolerance=tol, dt=dt * rg.ic.K)[2]
         for whole in (False, True)]
    assert i[0].n_passed == i[1].n_passed
    assert abs(i[1].dt_next - i[0].dt_next) <= 1e-4 * i[0].dt_next


@pytest.mark.parametrize("n_pp,n_pl", [(1, 1), (2, 32), (2, 33), (3, 152 * 32 + 1), (5, 10000), (6, 20001), (2, 40000),
                                       (63, 900), (64, 900)])
def test_shapes(rg, monkeypatch, n_pp, n_pl):
    # 64 protoplanets and the star are one large body too many
    check(rg, disk(rg, n_pp, n_pl), monkeypatch, tries=2, integrator="rkf78", adaptive=False,
          whole_used=n_pp < 64)


@pytest.mark.parametrize("n_pl", [500, 65503])
def test_gas_drag(rg, monkeypatch, n_pl):
    s = rg.ic.config3(n_pp=32, n_pl=n_pl)
    check(rg, s, monkeypatch, tries=2, integrator="rkf78", adaptive=True, tolerance=1e-8, output_interval=0.5 * rg.ic.K,
          gas=rg.ic.gas_params(rg.ic.gas_disk_config3()))


def test_inactive_bodies_and_no_star(rg, monkeypatch):
    s = disk(rg, 6, 900)
    s.md["id"][[2, 50, 333]] *= -1
    check(rg, s, monkeypatch, integrator="rk4", adaptive=False)
    n = s.n - 1
    t = rg.types.System(s.r[1:], s.v[1:], s.p[1:], s.md[1:], np.array([0, 0, 0, 6, 0, n - 6, 0], np.uint32))
    check(rg, t, monkeypatch, integrator="rk4", adaptive=False)


def test_two_handles_at_once(rg, monkeypatch):
    """Two handles, each on its own thread and stream: both launches need the
    whole GPU, and both finish."""
    monkeypatch.setenv("REDGB_TRY", "1")
    systems = [disk(rg, 4, 9000, seed=k) for k in (1, 2)]
    kw = dict(integrator="rk4", adaptive=False, dt=0.1 * rg.ic.K, precision="mixed")
    alone = []
    for s in systems:
        with rg.Sim(s, **kw) as sim:
            sim.launch_tries(200)
            sim.synchronize()
            alone.append(vec(sim.get_state(0).r))
    sims = [rg.Sim(s, **kw) for s in systems]
    failed = []

    def work(sim):
        try:
            for _ in range(10):
                sim.launch_tries(20)
            sim.synchronize()
        except Exception as e:   # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=work, args=(sim,)) for sim in sims]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    together = [vec(sim.get_state(0).r) for sim in sims]
    for sim in sims:
        sim.close()
    assert not failed
    assert all(np.array_equal(a, b) for a, b in zip(alone, together))
