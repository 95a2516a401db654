"""Tries of an all-pairs disk with each pair formed once (the default from 5120
large bodies on) against one-sided tiles (REDGB_PAIRS=0, which the gravity
tests hold to the oracle) and against the oracle's own steps: body counts at
the edges of the blocks of 512 and sub-blocks of 128, with test particles,
inactive bodies, and without a star.

Tolerance: FP32 pair terms in another grouping (~1e-7 of the pair part of an
acceleration, <= 1e-2 of it here, so 1e-9 of the acceleration at most; FP32
mode has its coordinate rounding besides, the same in both), over steps that
move a velocity by dt a <= 0.02: 1e-10 of the scale between the two paths,
1e-9 (MIXED) and 1e-7 (FP32) against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def vec(a):
    return np.stack([a["x"], a["y"], a["z"]], axis=1)


def disk(rg, n, n_tp=0, star=True):
    rng = np.random.Generator(np.random.MT19937(n))
    s = rg.ic.build_system(rng, pp_a=np.array([0.8, 1.2]), pp_mass=0.1 * rg.ic.EARTH_TO_SOLAR,
                           pl_a=rng.uniform(0.6, 1.8, n - 3), pl_mass=rg.ic.EARTH_TO_SOLAR / n, sigma_i=0.05,
                           n_tp=n_tp)
    s = s.relabel_all_SI()
    if not star:
        p = s.playing.copy()
        p[0] = 0
        s = rg.types.System(s.r[1:], s.v[1:], s.p[1:], s.md[1:], p)
    return s


def run(rg, s, monkeypatch, pairs, precision, steps=2, **kw):
    monkeypatch.setenv("REDGB_PAIRS", "1" if pairs else "0")
    with rg.Sim(s, dt=0.5 * rg.ic.K, precision=precision, **kw) as sim:
        before = sim.kernel_launches
        sim.launch_tries(steps)
        sim.synchronize()
        out = sim.get_state(0)
        return vec(out.r), vec(out.v), sim.info(0), sim.kernel_launches - before


@pytest.mark.parametrize("n,n_tp,star", [(5121, 0, True), (5122, 0, True), (5633, 5, True), (5760, 0, False),
                                        (6145, 33, True), (7017, 0, True), (5120, 0, True)])
@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_paths_agree(rg, orc, monkeypatch, precision, n, n_tp, star):
    s = disk(rg, n, n_tp, star)
    s.md["id"][[5, 700]] *= -1
    kw = dict(integrator="rk4", adaptive=False)
    r0, v0, i0, n0 = run(rg, s, monkeypatch, False, precision, **kw)
    r1, v1, i1, n1 = run(rg, s, monkeypatch, True, precision, **kw)
    assert (n1 > n0) == (n - star >= 5120)   # one more launch per stage
    assert i1.n_passed == i0.n_passed == 2 and i1.t == i0.t
    assert np.abs(r1 - r0).max() <= 1e-10 * np.abs(r0).max()
    assert np.abs(v1 - v0).max() <= 1e-10 * np.abs(v0).max()
    if n_tp == 0:
        b = orc.Body(s.r, s.v, s.p, s.md, s.playing)
        ig = orc.make_integrator(orc.RK4, 0.5 * rg.ic.K, sem=orc.SEM_GPU, nthreads=16)
        t = 0.0
        for _ in range(2):
            _, t = orc.step(ig, b, t)
        tol = 1e-9 if precision == "mixed" else 1e-7
        assert np.abs(r1 - vec(b.r)).max() <= tol * np.abs(r1).max()
        assert np.abs(v1 - vec(b.v)).max() <= tol * np.abs(v1).max()


def test_adaptive_and_after_an_evaluation(rg, monkeypatch):
    """Adaptive tries, with a force evaluation (one-sided tiles, other partial
    records) before and between them."""
    s = disk(rg, 6000)
    monkeypatch.setenv("REDGB_PAIRS", "1")
    kw = dict(integrator="rkf78", adaptive=True, tolerance=1e-9, dt=0.5 * rg.ic.K, output_interval=0.5 * rg.ic.K,
              collision_factor=1.0)
    out = []
    for evaluate in (False, True):
        with rg.Sim(s, **kw) as sim:
            for _ in range(2):
                if evaluate:
                    sim.calc_dydx(0, 1, 0.0)
                sim.launch_tries(1)
                sim.synchronize()
            out.append(vec(sim.get_state(0).r))
            assert sim.info(0).n_passed == 2
    assert np.array_equal(out[0], out[1])
    r0 = run(rg, s, monkeypatch, False, "mixed", integrator="rkf78", adaptive=True, tolerance=1e-9,
             output_interval=0.5 * rg.ic.K)[0]
    assert np.abs(out[0] - r0).max() <= 1e-10 * np.abs(r0).max()
