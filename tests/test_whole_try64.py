"""A try as one cooperative launch in FP64 against one launch per stage: every
scheme, adaptive steps, inactive bodies, no star, sizes at the edges of the
launch's shape (16 small bodies to a warp, one to four shares of the pairs, an
odd and an even number of large bodies, fewer than one group of four, the
largest).

Tolerance: both paths are FP64 and differ in the order of sums and in the
combinations of the stages, a few ulp (1e-16 of the scale) per stage; a pair's
term of a body at distance d amplifies that by dt m / d^3 <= 3e-6 (m 3e-7, dt
0.01, d >= 1e-3 in these disks) beside the star's ~0.01: 1e-13 of the scale is
~100 ulp for up to 39 stages.  The error estimate is a cancelling combination of
accelerations: its rounding, 4e-16 of them, is 2e-7 of an estimate near the
tolerance (1e-10 / (lambda dt))."""
import numpy as np
import pytest
from test_whole_try import disk, run, vec

pytestmark = pytest.mark.gpu


def check(rg, s, monkeypatch, tries=3, **kw):
    kw = dict(dict(dt=0.5 * rg.ic.K, collision_factor=1.0, precision="fp64"), **kw)
    r0, v0, i0, n0 = run(rg, s, monkeypatch, False, tries, **kw)
    r1, v1, i1, n1 = run(rg, s, monkeypatch, True, tries, **kw)
    assert n1 < n0
    assert (i1.n_passed, i1.n_tried, i1.halted, i1.status) == (i0.n_passed, i0.n_tried, i0.halted, i0.status)
    assert i1.t == i0.t
    assert np.abs(r1 - r0).max() <= 1e-13 * np.abs(r0).max()
    assert np.abs(v1 - v0).max() <= 1e-13 * np.abs(v0).max()
    return i0, i1


@pytest.mark.parametrize("integrator", ["euler", "rk2", "rk4", "rkf78"])
def test_fixed_step_schemes(rg, monkeypatch, integrator):
    s = disk(rg, 6, 900)
    s.md["id"][[2, 50, 333]] *= -1
    check(rg, s, monkeypatch, integrator=integrator, adaptive=False)


@pytest.mark.parametrize("integrator,dt,tol", [("rk4", 0.5, 1e-6), ("rkf78", 1.5, 1e-10)])
def test_adaptive_schemes(rg, monkeypatch, integrator, dt, tol):
    s = rg.ic.config2(seed=3, n_pp=8, n_pl=3000)
    i0, i1 = check(rg, s, monkeypatch, tries=1, integrator=integrator, adaptive=True, tolerance=tol, dt=dt * rg.ic.K)
    assert abs(i1.dt_next - i0.dt_next) <= 1e-5 * i0.dt_next
    r, v, i, _ = run(rg, s, monkeypatch, True, 1, integrator=integrator, adaptive=True, tolerance=tol,
                     dt=60.0 * rg.ic.K, precision="fp64")   # rejected: the state untouched
    assert i.n_passed == 0 and np.array_equal(r, vec(s.r)) and np.array_equal(v, vec(s.v))


@pytest.mark.parametrize("n_pp,n_pl", [(1, 1), (2, 32), (7, 33), (8, 152 * 32 + 1), (16, 10000), (33, 20001),
                                       (2, 40000), (62, 900), (63, 900)])
def test_shapes(rg, monkeypatch, n_pp, n_pl):
    check(rg, disk(rg, n_pp, n_pl), monkeypatch, tries=2, integrator="rkf78", adaptive=False)


def test_no_star(rg, monkeypatch):
    s = disk(rg, 6, 900)
    n = s.n - 1
    t = rg.types.System(s.r[1:], s.v[1:], s.p[1:], s.md[1:], np.array([0, 0, 0, 6, 0, n - 6, 0], np.uint32))
    check(rg, t, monkeypatch, integrator="rk4", adaptive=False)
