"""The energy step is (udot 2) dth in the reference's order (sim/sph.go:121-193):
2 udot overflows for |udot| >= 2^1023, where udot (2 dth) would stay finite."""
import numpy as np
import pytest

from sphugo_gb300 import ics
from sphugo_gb300 import sim as S

pytestmark = pytest.mark.gpu


def test_energy_rates_beyond_half_the_largest_double(gpu, oracle):
    n, k = 600, 32
    r = np.random.default_rng(4)
    x, y, vx, vy, u = r.random(n), r.random(n), r.normal(0, 1e9, n), r.normal(0, 1e9, n), np.full(n, 2.5e302)
    conf = ics.periodic_config(n, k, 2e-300)
    conf.ParticleMass = 1.0
    g = S.Simulation(conf, x, y, vx, vy, u)
    o = oracle.OracleSim(oracle.make_params(n, k, mass=1.0, dth=1e-300, alpha=1.0, beta=2.0), x, y, vx, vy, u)
    g.Step(1)
    o.step(1)
    got, want = g.state(), o.state()
    assert np.isfinite(want["udot"]).all() and np.isinf(want["u"]).sum() == 3
    for key in got:
        assert np.array_equal(got[key], want[key]), key
