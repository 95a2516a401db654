"""The brute-force collision check at the edges of its tiles (128 bodies i,
512 later ones j) and of its FP32 filter, against red's FP64 test over every
pair: the same pairs and distances, to the bit.  Pairs sit just inside and just
outside contact, at distances from the origin where an FP32 coordinate is
coarser than the radii, and across the sign of a coordinate; some bodies are
inactive or not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def field(rg, n_si, n_small, scale, seed):
    """n_si protoplanets and n_small planetesimals, a third of them close to
    contact with an earlier body."""
    rng = np.random.Generator(np.random.MT19937(seed))
    n = n_si + n_small
    s = rg.ic.build_system(rng, pp_a=np.linspace(0.75, 1.45, n_si - 1), pp_mass=1e-9,
                           pl_a=rng.uniform(0.7, 1.5, max(n_small, 1)), pl_mass=1e-12)
    r = rng.uniform(-scale, scale, (s.n, 3))
    radius = 10.0 ** rng.uniform(-8, -4, s.n)
    for j in range(1, s.n):
        if rng.random() < 0.3:
            i = rng.integers(0, min(j, n_si))
            u = rng.normal(size=3)
            u /= np.linalg.norm(u)
            gap = (radius[i] + radius[j]) * (1.0 + rng.choice([-1e-3, 1e-3, -1e-7, 1e-7]))
            r[j] = r[i] + gap * u
    for c, k in enumerate("xyz"):
        s.r[k] = r[:, c]
    s.p["radius"] = radius
    s.md["id"][rng.choice(np.arange(1, s.n), s.n // 20, replace=False)] *= -1
    return s, n


def pairs_of(s, n_si, factor):
    """red's test (check_for_collision: 0 < id_i, id_j not negative), rounded
    operation by operation, of every pair with a large body."""
    x, y, z = s.r["x"], s.r["y"], s.r["z"]
    R, ident = s.p["radius"], s.md["id"]
    out = {}
    f = np.float64(factor) * np.float64(factor)
    with np.errstate(all="ignore"):
        for i in range(n_si):
            if ident[i] <= 0:
                continue
            j = np.arange(i + 1, s.n)
            w = ((x[j] - x[i]) ** 2 + (y[j] - y[i]) ** 2) + (z[j] - z[i]) ** 2
            rs = R[i] + R[j]
            hit = (w < f * (rs * rs)) & (ident[j] >= 0)
            for jj, d in zip(j[hit], np.sqrt(w[hit])):
                out[(i, int(jj))] = d
    return out


@pytest.mark.parametrize("n_si,n_small", [(2, 1), (3, 509), (3, 510), (127, 1), (129, 600), (513, 2)])
@pytest.mark.parametrize("scale,factor", [(1.0, 1.0), (1.0e4, 1.0), (1.0, 50.0)])
def test_pairs(rg, n_si, n_small, scale, factor):
    s, _ = field(rg, n_si, n_small, scale, seed=n_si + n_small)
    ref = pairs_of(s, n_si, factor)
    with rg.Sim(s, dt=0.01, collision_factor=factor, event_capacity=1 << 16) as sim:
        ev = sim.check_for_collision(cap=1 << 16)
    got = {tuple(sorted((int(e["idx1"]), int(e["idx2"])))): float(e["d"]) for e in ev}
    got = {k: d for k, d in got.items() if k[0] < n_si}
    assert len(ref) >= 0.02 * s.n - 1
    assert got == ref


def test_far_and_not_finite(rg):
    s, _ = field(rg, 140, 400, 1.0, seed=9)
    s.r["x"][[5, 139, 200]] = [np.inf, np.nan, -np.inf]
    s.r["y"][[7, 300]] = 1.0e30
    s.r["x"][300], s.r["z"][300] = s.r["x"][7], s.r["z"][7]
    s.p["radius"][7] = s.p["radius"][300] = 1.0
    s.md["id"][[7, 300]] = [8, 301]
    ref = pairs_of(s, 140, 1.0)
    assert (7, 300) in ref
    with rg.Sim(s, dt=0.01, collision_factor=1.0, event_capacity=1 << 16) as sim:
        ev = sim.check_for_collision(cap=1 << 16)
    got = {tuple(sorted((int(e["idx1"]), int(e["idx2"])))): float(e["d"]) for e in ev}
    assert {k: d for k, d in got.items() if k[0] < 140} == ref
