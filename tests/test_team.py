"""Tries of an ensemble of sparse systems as one cluster launch (the default in
the FP32 modes) against one launch per stage (REDGB_TRY=0): ensembles whose
teams differ in size and share clusters, systems at the edges (one small body,
one CTA's 512, eight CTAs' 4096, 16 large bodies), every scheme, inactive
bodies, a system that is finished, retries with a step quota.

Tolerance as for single systems in whole tries: 1e-10 of the scale after a few
steps (FP32 pair terms of <= 1e-3 of an acceleration in another order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def vec(a):
    return np.stack([a["x"], a["y"], a["z"]], axis=1)


def disk(rg, n_pp, n_pl, seed):
    rng = np.random.Generator(np.random.MT19937(seed))
    return rg.ic.build_system(rng, pp_a=np.linspace(0.75, 1.45, n_pp), pp_mass=0.1 * rg.ic.EARTH_TO_SOLAR,
                              pl_a=rng.uniform(0.7, 1.5, n_pl), pl_mass=rg.ic.EARTH_TO_SOLAR / max(n_pl, 1))


def run(rg, systems, monkeypatch, whole, tries, **kw):
    monkeypatch.setenv("REDGB_TRY", "1" if whole else "0")
    with rg.Sim(systems, **kw) as sim:
        before = sim.kernel_launches
        sim.launch_tries(tries)
        sim.synchronize()
        launches = sim.kernel_launches - before
        out = [sim.get_state(k) for k in range(len(systems))]
        return [vec(o.r) for o in out], [vec(o.v) for o in out], [sim.info(k) for k in range(len(systems))], launches


def check(rg, systems, monkeypatch, tries=3, **kw):
    kw = dict(dict(dt=0.5 * rg.ic.K, collision_factor=1.0), **kw)
    r0, v0, i0, n0 = run(rg, systems, monkeypatch, False, tries, **kw)
    r1, v1, i1, n1 = run(rg, systems, monkeypatch, True, tries, **kw)
    assert n1 < n0
    for k in range(len(systems)):
        assert (i1[k].n_passed, i1[k].n_tried, i1[k].halted, i1[k].status, i1[k].active) == \
               (i0[k].n_passed, i0[k].n_tried, i0[k].halted, i0[k].status, i0[k].active)
        assert i1[k].t == i0[k].t
        assert np.abs(r1[k] - r0[k]).max() <= 1e-10 * np.abs(r0[k]).max()
        assert np.abs(v1[k] - v0[k]).max() <= 1e-10 * np.abs(v0[k]).max()
    return i0, i1


SIZES = [(1, 1), (2, 511), (3, 512), (4, 513), (8, 2047), (15, 900), (5, 4096), (2, 1500), (6, 130)]


@pytest.mark.parametrize("integrator", ["euler", "rk2", "rk4", "rkf78"])
@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_fixed_step_schemes(rg, monkeypatch, integrator, precision):
    systems = [disk(rg, a, b, 10 + k) for k, (a, b) in enumerate(SIZES)]
    systems[3].md["id"][[2, 40]] *= -1
    check(rg, systems, monkeypatch, integrator=integrator, adaptive=False, precision=precision)


@pytest.mark.parametrize("n_sys", [2, 40, 130])
def test_adaptive_ensembles(rg, monkeypatch, n_sys):
    """40: teams of fewer bodies, all resident; 130: several waves of clusters."""
    systems = [disk(rg, 2 + k % 7, 100 + (k * 977) % 4000, 100 + k) for k in range(n_sys)]
    check(rg, systems, monkeypatch, tries=2, integrator="rkf78", adaptive=True, tolerance=1e-9,
          output_interval=0.5 * rg.ic.K)


def test_different_steps_and_rejections(rg, monkeypatch):
    """Every system its own step; one far too long (rejected, its state
    untouched), one past its length after the first step."""
    systems = [disk(rg, 4, 300 + 400 * k, 50 + k) for k in range(4)]
    dt = np.array([0.5, 1.0, 60.0, 0.25]) * rg.ic.K
    kw = dict(integrator="rkf78", adaptive=True, tolerance=1e-10, dt=dt)
    r0, _, i0, _ = run(rg, systems, monkeypatch, False, 1, **kw)
    r1, _, i1, _ = run(rg, systems, monkeypatch, True, 1, **kw)
    assert [i.n_passed for i in i1] == [i.n_passed for i in i0] == [1, 1, 0, 1]
    assert np.array_equal(r1[2], vec(systems[2].r))
    for k in (0, 1, 3):
        assert np.abs(r1[k] - r0[k]).max() <= 1e-10 * np.abs(r0[k]).max()
    check(rg, systems, monkeypatch, tries=4, integrator="rk4", adaptive=False, length=0.9 * rg.ic.K)


def test_step_by_step(rg, monkeypatch):
    """red_step on the ensemble: every system one accepted step, the systems that
    need a second try retried while the others wait."""
    systems = [disk(rg, 4, 200 + 300 * k, 70 + k) for k in range(5)]
    dt = np.array([0.5, 30.0, 1.0, 40.0, 0.5]) * rg.ic.K
    out = []
    for whole in ("0", "1"):
        monkeypatch.setenv("REDGB_TRY", whole)
        with rg.Sim(systems, integrator="rkf78", adaptive=True, tolerance=1e-10, dt=dt) as sim:
            sim.step()
            out.append([(sim.info(k).n_passed, vec(sim.get_state(k).r)) for k in range(5)])
    assert [p for p, _ in out[1]] == [1] * 5
    for k in (0, 2, 4):
        assert np.abs(out[1][k][1] - out[0][k][1]).max() <= 1e-10 * np.abs(out[0][k][1]).max()
