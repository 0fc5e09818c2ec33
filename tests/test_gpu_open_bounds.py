"""The bounding box of open axes is reduced per block and per warp before its
atomics: simulations of every size against a block's range, and ensembles whose
members (some open in one axis, some in both, some periodic) end inside blocks
and warps, must equal the oracle bit for bit."""
import numpy as np
import pytest

from sphugo_gb300 import ics
from sphugo_gb300 import sim as S

pytestmark = pytest.mark.gpu


def make(n, seed, hor, vert):
    conf = ics.periodic_config(n, 16, 1e-4)
    conf.HorPeriodicity, conf.VertPeriodicity = hor, vert
    x, y, _, _, u = ics.uniform_blast(n, seed)
    r = np.random.default_rng(seed)
    if hor == S.OPEN:
        x = 1.25 * x - 0.7
    return conf, (x, y, r.normal(0, 0.5, n), r.normal(0, 0.5, n), u)


def oracle_of(O, conf, arrs):
    o = O.OracleSim(O.make_params(
        len(arrs[0]), 16, kernel=0, knn_mode=O.KNN_EXACT, gamma=conf.Gamma, mass=conf.ParticleMass, dth=conf.DeltaTHalf,
        accel=(0, 0), hor=conf.HorPeriodicity, vert=conf.VertPeriodicity,
        refl=(-S.DBL_MAX, S.DBL_MAX, -S.DBL_MAX, S.DBL_MAX), alpha=conf.ViscosityAlpha, beta=conf.ViscosityBeta,
        etasq=conf.ViscosityEtaSq), *arrs)
    o.step(2)
    return o.state()


@pytest.mark.parametrize("n", [255, 256, 1001, 155_649, 200_001])
def test_open_box_sizes(gpu, oracle, n):
    conf, arrs = make(n, n, S.OPEN, S.OPEN)
    s = S.Simulation(conf, *arrs)
    s.Step(2)
    got, want = s.state(), oracle_of(oracle, conf, arrs)
    for k in got:
        assert np.array_equal(got[k], want[k]), k


def test_open_ensemble(gpu, oracle):
    unit = (0.0, 1.0)
    kinds = [(S.OPEN, S.OPEN), (unit, S.OPEN), (unit, unit), (S.OPEN, unit)]
    sims = [make(n, 40 + i, *kinds[i % 4]) for i, n in enumerate([137, 300, 1000, 164, 2500, 131, 700, 133, 5000, 129, 190, 257])]
    e = S.Ensemble([c for c, _ in sims], [a for _, a in sims])
    e.Step(2)
    got = e.state()
    for (conf, arrs), o0, o1 in zip(sims, e.offsets[:-1], e.offsets[1:]):
        want = oracle_of(oracle, conf, arrs)
        for k in got:
            assert np.array_equal(got[k][o0:o1], want[k]), (k, o0)
