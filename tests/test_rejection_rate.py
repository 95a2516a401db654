"""Whole tries reject as often as one launch per stage (REDGB_TRY=0): a 16384-body disk,
adaptive RKF7(8) at 1e-12 in MIXED, where two tries in five are rejected, because close
encounters bring FP32 pair noise into the estimate.  A CTA that acts on the wrong
decision, or an estimate with other noise, shows here in the fraction and in the energy.

Over 4000 tries each fraction has a standard deviation of sqrt(0.25 / 4000) = 0.8 %; the
two runs part after a few close encounters, so they differ by 1.1 %, and 5 % is beyond
chance."""
import pytest

pytestmark = pytest.mark.gpu


def test_fraction(rg, monkeypatch):
    s = rg.ic.config2(seed=2)
    frac, drift = [], []
    for whole in ("0", "1"):
        monkeypatch.setenv("REDGB_TRY", whole)
        with rg.Sim(s, integrator="rkf78", adaptive=True, tolerance=1e-12, dt=0.5 * rg.ic.K) as sim:
            e0 = sim.energy_interacting(0)[0]
            for _ in range(8):
                sim.launch_tries(500)
                sim.synchronize()
            i = sim.info(0)
            e1 = sim.energy_interacting(0)[0]
        assert i.status == 0 and i.n_tried >= 3900
        frac.append(i.n_failed / i.n_tried)
        drift.append(abs((e1 - e0) / e0))
    print("rejected: stages %.4f, whole tries %.4f; |dE/E| %.2e, %.2e" % (*frac, *drift))
    assert abs(frac[1] - frac[0]) < 0.05
    assert max(drift) < 1e-10
