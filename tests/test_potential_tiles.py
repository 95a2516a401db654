"""The potential sums of the integrals at the edges of their tiles: system sizes
around one tile of 128 bodies and around the ranges of 32 that one partial
covers, no large body, test particles and inactive bodies inside.

Tolerance: every term is positive, each carries a few roundings and the sums
are at most ~1000 terms deep per partial, so U is good to ~1e-13 relative;
E = T - U is compared on the scale T + U."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_pp,n_pl,n_tp", [(0, 126, 0), (1, 126, 0), (2, 126, 0), (31, 0, 0), (32, 95, 1), (40, 1237, 3),
                                            (3, 4091, 2)])
def test_energies_match_extended_precision(rg, n_pp, n_pl, n_tp):
    rng = np.random.Generator(np.random.MT19937(11 + n_pl))
    s = rg.ic.build_system(rng, pp_a=rng.uniform(0.8, 1.4, n_pp), pp_mass=0.1 * rg.ic.EARTH_TO_SOLAR,
                           pl_a=rng.uniform(0.7, 1.5, n_pl), pl_mass=1e-3, n_tp=n_tp)
    if n_pl > 100:
        s.md["id"][1 + n_pp + np.array([0, 64])] *= -1
    with rg.Sim(s, dt=0.01) as sim:
        E_all = sim.calc_integral(0)[-1]
        E_int = sim.energy_interacting(0)[0]
    ld = np.longdouble
    live = s.md["id"] > 0
    m = np.where(live, s.p["mass"], 0.0).astype(ld)
    r = np.stack([s.r[c] for c in "xyz"], axis=1).astype(ld)
    v2 = sum(s.v[c].astype(ld) ** 2 for c in "xyz")
    U, U_int = ld(0), ld(0)
    n_massive = s.n_SI + s.n_NSI
    for i in range(s.n):
        d = np.sqrt(((r[i + 1:] - r[i]) ** 2).sum(axis=1))
        u = m[i] * m[i + 1:] / d
        U += u.sum()
        if i < s.n_SI:
            U_int += u[:max(0, n_massive - i - 1)].sum()
    T = (m * v2).sum() / 2
    T_int = (m * v2)[:n_massive].sum() / 2
    assert abs(E_all - (T - U)) <= 1e-13 * (T + U)
    assert abs(E_int - (T_int - U_int)) <= 1e-13 * (T_int + U_int)
