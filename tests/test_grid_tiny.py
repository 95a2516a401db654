"""The collision check of small bodies whose grid cells are too small for FP32 (radii of
1e-40): red's exact pair set.  A body's place in its cell cannot be told from the FP32
copies there, so every neighbouring cell has to be looked up."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [1.0e-36, 1.0e-40, 1.0e-43])
def test_pairs(rg, radius):
    n = 1200
    rng = np.random.Generator(np.random.MT19937(9))
    s = rg.ic.build_system(rng, pp_a=np.array([1.0]), pp_mass=1e-9, pl_a=rng.uniform(0.7, 1.5, n), pl_mass=1e-12)
    r = rng.uniform(-15.0, 15.0, (s.n, 3)) * radius
    r[:2] = [[50.0, 0.0, 0.0], [60.0, 0.0, 0.0]]       # the star and the protoplanet, out of the way
    for c, k in enumerate("xyz"):
        s.r[k] = r[:, c]
    s.p["radius"][:] = radius
    ref = set()
    for i in range(2, s.n):
        d = np.linalg.norm((r[i + 1:] - r[i]) / radius, axis=1)
        ref.update((i, i + 1 + int(j)) for j in np.flatnonzero(d < 2.0))
    assert len(ref) > 100
    with rg.Sim(s, dt=0.01, collision_factor=1.0, event_capacity=1 << 20) as sim:
        ev = sim.check_for_collision(cap=1 << 18)
    got = {tuple(sorted((int(e["idx1"]), int(e["idx2"])))) for e in ev}
    assert len(ev) == len(ref) and got == ref
