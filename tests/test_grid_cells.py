"""The collision check of the small bodies through the hash grid looks up a
neighbouring cell only when the body is within a collision distance of it:
red's exact pair set, to the bit, for bodies placed at the faces, edges and
corners of cells, on both sides of zero, near and beyond the distance where
FP32 still tells a body's place in its cell (2^18 cells), and in one cell."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [0.0, 1.0, 2.0 ** 18, 2.0 ** 22, 3.0e9])
@pytest.mark.parametrize("spread", [3.0, 40.0])
def test_pairs(rg, far, spread):
    """Pairs a little inside and outside contact, centred on points of the grid
    of cell edges (any cell size up to 8 collision distances divides 8 of them),
    `far` cells from the origin."""
    n, radius = 1500, 1.0e-6
    rng = np.random.Generator(np.random.MT19937(int(spread) + int(np.log2(far + 1))))
    s = rg.ic.build_system(rng, pp_a=np.array([1.0]), pp_mass=1e-9, pl_a=rng.uniform(0.7, 1.5, n), pl_mass=1e-12)
    reach = 2.0 * radius * (1.0 + 1.0e-6)
    r = np.zeros((s.n, 3))
    r[:2] = [[50.0, 0.0, 0.0], [60.0, 0.0, 0.0]]       # the star and the protoplanet, out of the way
    m = n // 2
    corner = rng.integers(-int(spread), int(spread) + 1, (m, 3)) * (4.0 * reach) + np.array([far, -far, 0.0]) * (4.0 * reach)
    corner += rng.choice([0.0, 0.5 * reach, 2.0 * reach], (m, 3))
    u = rng.normal(size=(m, 3)) * rng.choice([0.0, 1.0], (m, 3), p=[0.3, 0.7])
    u[np.all(u == 0, axis=1)] = [1.0, 0.0, 0.0]
    u /= np.linalg.norm(u, axis=1)[:, None]
    half = 0.5 * reach * rng.choice([0.2, 0.999, 1.001], m)[:, None]
    t = rng.uniform(-1, 1, (m, 1)) * half
    r[2:2 + m] = corner + (t - half) * u
    r[2 + m:2 + 2 * m] = corner + (t + half) * u
    for c, k in enumerate("xyz"):
        s.r[k] = r[:, c]
    s.p["radius"][:] = radius
    ref = {}
    x, y, z, R = s.r["x"], s.r["y"], s.r["z"], s.p["radius"]
    for i in range(s.n):
        j = np.arange(i + 1, s.n)
        w = ((x[j] - x[i]) ** 2 + (y[j] - y[i]) ** 2) + (z[j] - z[i]) ** 2
        rs = R[i] + R[j]
        hit = w < rs * rs
        ref.update({(i, int(jj)): d for jj, d in zip(j[hit], np.sqrt(w[hit]))})
    assert len(ref) >= m // 4
    with rg.Sim(s, dt=0.01, collision_factor=1.0, event_capacity=1 << 20) as sim:
        ev = sim.check_for_collision(cap=1 << 18)
    got = {tuple(sorted((int(e["idx1"]), int(e["idx2"])))): float(e["d"]) for e in ev}
    assert len(ev) == len(ref) and got == ref
