"""Stage sums, error and solution of the whole-try kernels (k_try, k_team) are FP64.

Disks whose protoplanets and planetesimals have a mass of 1e-25: their pair terms
vanish, and a body's acceleration a is its star term, a function of positions good to
2^-48 that the kernels share with one launch per stage (REDGB_TRY=0), whose sums are
FP64.  One step against that path, body by body: a position is off by 4 ulp and
4e-14 dt^2 |a| at most, a velocity by 4 ulp and 4e-14 dt |a|.  A sum in FP32 is off by
~6e-8 of the same increments; the CPU test puts that mistake into a restatement and
finds every second body or more outside the bound."""
import numpy as np
import pytest

U = 2.0 ** -52


def vec(a):
    return np.stack([a["x"], a["y"], a["z"]], axis=1)


def disk(rg, n_pp, n_pl, seed):
    rng = np.random.Generator(np.random.MT19937(seed))
    s = rg.ic.build_system(rng, pp_a=np.linspace(0.75, 1.45, n_pp), pp_mass=1e-25,
                           pl_a=rng.uniform(0.2, 1.5, n_pl), pl_mass=1e-25)
    s.r["x"] -= s.r["x"][0]
    s.r["y"] -= s.r["y"][0]
    s.r["z"] -= s.r["z"][0]
    return s


def bounds(s, dt):
    r, v = vec(s.r), vec(s.v)
    d = np.linalg.norm(r[1:], axis=1)
    a = s.p["mass"][0] / d ** 2
    n = np.linalg.norm(v[1:], axis=1)
    return 4 * U * d + 4e-14 * dt * dt * a, 4 * U * n + 4e-14 * dt * a


def step(rg, systems, precision, dt, **kw):
    with rg.Sim(systems, dt=dt, precision=precision, **kw) as sim:
        before = sim.kernel_launches
        sim.launch_tries(1)
        sim.synchronize()
        launches = sim.kernel_launches - before
        return [(vec(sim.get_state(k).r), vec(sim.get_state(k).v), sim.info(k)) for k in range(len(systems))], launches


SCHEMES = [("euler", False, 0.5), ("rk2", False, 1.0), ("rk4", False, 2.0), ("rk4", True, 2.0), ("rkf78", False, 3.0),
           ("rkf78", True, 3.0)]


@pytest.mark.gpu
@pytest.mark.parametrize("integrator,adaptive,days", SCHEMES)
@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("n_sys", [1, 5])
def test_against_stages(rg, monkeypatch, integrator, adaptive, days, precision, n_sys):
    systems = [disk(rg, 3 + k, 400 + 301 * k, 7 + k) for k in range(n_sys)]
    dt = days * rg.ic.K
    kw = dict(integrator=integrator, adaptive=adaptive, tolerance=1e-3)
    monkeypatch.setenv("REDGB_TRY", "0")
    ref, _ = step(rg, systems, precision, dt, **kw)
    monkeypatch.setenv("REDGB_TRY", "1")
    got, launches = step(rg, systems, precision, dt, **kw)
    assert launches == 1
    for s, (r0, v0, i0), (r1, v1, i1) in zip(systems, ref, got):
        assert i1.n_passed == i0.n_passed == 1
        br, bv = bounds(s, dt)
        assert np.all(np.linalg.norm(r1 - r0, axis=1)[1:] <= br)
        assert np.all(np.linalg.norm(v1 - v0, axis=1)[1:] <= bv)
        if adaptive:
            # the estimate is lambda dt times a difference of four accelerations (two in
            # RK4), or of their sums times dt: 4 x 3.1e-14 of the largest acceleration
            lam, order = (41.0 / 840.0, 7) if integrator == "rkf78" else (0.1, 4)
            est = 1e-3 * (0.9 * dt / i0.dt_next) ** order
            noise = lam * dt * 4 * 3.1e-14 * np.max(s.p["mass"][0] / np.sum(vec(s.r)[1:] ** 2, axis=1))
            assert abs(i1.dt_next - i0.dt_next) <= (noise / est / order + 1e-14) * i0.dt_next


@pytest.mark.gpu
@pytest.mark.parametrize("integrator", ["euler", "rk2"])
@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("n_sys", [1, 5])
def test_fp64_to_the_last_bits(rg, monkeypatch, integrator, precision, n_sys):
    """A step of 1000 time units, whose increments are the whole result: the accelerations
    of these schemes do not depend on the sums, so both paths have the same ones, and
    three roundings of FP64 each lie between their results.  Sums of 2^-47 are out by ~32 ulp."""
    systems = [disk(rg, 3 + k, 400 + 301 * k, 7 + k) for k in range(n_sys)]
    dt = 1000.0
    out = []
    for whole in ("0", "1"):
        monkeypatch.setenv("REDGB_TRY", whole)
        out.append(step(rg, systems, precision, dt, integrator=integrator, adaptive=False))
    assert out[1][1] == 1 < out[0][1]
    for s, (r0, v0, _), (r1, v1, _) in zip(systems, out[0][0], out[1][0]):
        r, v = vec(s.r)[1:], vec(s.v)[1:]
        d, n = np.linalg.norm(r, axis=1), np.linalg.norm(v, axis=1)
        # rk2's accelerations are those after a straight half step
        a = np.linalg.norm(v0[1:] - v, axis=1) / dt
        a0 = s.p["mass"][0] / d ** 2
        assert np.all(np.linalg.norm(v1 - v0, axis=1)[1:] <= 4 * U * (n + dt * a))
        assert np.all(np.linalg.norm(r1 - r0, axis=1)[1:] <= 4 * U * (d + dt * n + dt * dt * a0))


def test_the_bound_sees_fp32_sums(rg):
    """An RK4 step in numpy, its velocity and position increments summed in FP64 and in FP32."""
    s = disk(rg, 3, 400, 7)
    dt = 2.0 * rg.ic.K
    r, v = vec(s.r)[1:], vec(s.v)[1:]

    def acc(x):
        return -s.p["mass"][0] * x / np.linalg.norm(x, axis=1)[:, None] ** 3

    def rk4(sums):
        k = [acc(r)]
        for c in (0.5, 0.5, 1.0):
            m = len(k)
            pos = np.zeros_like(r) if m == 1 else 0.5 * c * k[m - 2]   # Nystroem's row
            k.append(acc(r + c * dt * v + dt * dt * sums([pos])))
        return (r + dt * v + dt * dt * sums([k[0] / 6, k[1] / 6, k[2] / 6]),
                v + dt * sums([k[0] / 6, k[1] / 3, k[2] / 3, k[3] / 6]))

    r0, v0 = rk4(lambda t: sum(t))
    r1, v1 = rk4(lambda t: sum(x.astype(np.float32) for x in t).astype(np.float64))
    br, bv = bounds(s, dt)
    assert np.mean(np.linalg.norm(v1 - v0, axis=1) > bv) > 0.5
    assert np.mean(np.linalg.norm(r1 - r0, axis=1) > br) > 0.5
