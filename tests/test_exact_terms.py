"""The red-exact gravity forms its pair terms in parallel and adds them in red's
order: bit-identical to the oracle where the split changes shape -- source
lists at and past one tile (the first chunked length), ragged last chunks,
tiles of 1, 31, 32 and 33 sinks, a batch that does not divide the tile,
inactive bodies among sinks and sources."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def vec(a):
    return np.stack([a["x"], a["y"], a["z"]], axis=1)


@pytest.mark.parametrize("n_pp,n_pl,n_tp", [
    (1, 126, 0),      # 128 sources: one tile, not chunked
    (1, 127, 1),      # 129 sources: chunks of 32, the last of one source
    (2, 700, 33),     # ragged last chunk, a test-particle tile of one sink
    (30, 1000, 0),    # 31 large bodies
    (31, 1000, 5),    # 32: a full tile
    (32, 1003, 0),    # 33: two tiles of the large-body class
    (4, 11000, 0),    # chunks longer than 32 sources
    (600, 50, 0),     # many large-body tiles, batches of 16 sources
])
def test_terms_added_in_red_order(rg, orc, n_pp, n_pl, n_tp):
    rng = np.random.Generator(np.random.MT19937(7 + n_pp))
    s = rg.ic.build_system(rng, pp_a=rng.uniform(0.8, 1.4, n_pp), pp_mass=0.1 * rg.ic.EARTH_TO_SOLAR,
                           pl_a=rng.uniform(0.7, 1.5, n_pl), pl_mass=rg.ic.EARTH_TO_SOLAR / n_pl, n_tp=n_tp)
    dead = np.array([1, 1 + n_pp + n_pl // 2])
    s.md["id"][dead] *= -1
    s.inactive[3], s.inactive[5] = 1, 1
    with rg.Sim(s, integrator="rk4", adaptive=False, dt=0.01, precision="fp64_exact") as sim:
        a = [vec(sim.calc_dydx(0, 1, 0.0)) for _ in range(2)]
    rc, ref = orc.grav_accel(orc.Body(s.r, s.v, s.p, s.md, s.playing), sem=orc.SEM_GPU)
    assert rc == 0
    assert np.array_equal(a[0], vec(ref))
    assert np.array_equal(a[1], vec(ref))
