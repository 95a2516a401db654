"""Gas drag in a whole try (k_try) against one launch per stage (REDGB_TRY=0), which
test_drag_mixed holds to the oracle: both FP32 modes, and a first body without mass,
whose gas is at rest (circular speed 0) and whose drag is finite.

Tolerance: both paths form the drag with drag_factor_fast and differ in the rounding
of its inputs (positions of 2^-48) and in the order of FP32 pair sums (~1e-7 of the
pair terms, <= 1e-3 of an acceleration): 1e-10 of the scale after a few steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def vec(a):
    return np.stack([a["x"], a["y"], a["z"]], axis=1)


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("star_mass", [1.0, 0.0])
def test_drag(rg, monkeypatch, precision, star_mass):
    s = rg.ic.config3(n_pp=5, n_pl=700)
    s.p["mass"][0] = star_mass
    out = []
    for whole in ("0", "1"):
        monkeypatch.setenv("REDGB_TRY", whole)
        with rg.Sim(s, integrator="rkf78", adaptive=False, dt=0.5 * rg.ic.K, precision=precision,
                    gas=rg.ic.gas_params(rg.ic.gas_disk_config3())) as sim:
            before = sim.kernel_launches
            sim.launch_tries(2)
            _, halted = sim.synchronize()
            o, i = sim.get_state(0), sim.info(0)
            out.append((vec(o.r), vec(o.v), (halted, i.status, i.n_passed), sim.kernel_launches - before))
    (r0, v0, i0, n0), (r1, v1, i1, n1) = out
    assert n1 < n0 and i1 == i0 == (0, 0, 2)
    assert np.isfinite(r1).all() and np.isfinite(v1).all()
    assert np.abs(r1 - r0).max() <= 1e-10 * np.abs(r0).max()
    assert np.abs(v1 - v0).max() <= 1e-10 * np.abs(v0).max()
