"""The lists handed to the caller are sorted a warp per query, one, two or four
entries per lane: list lengths on both sides of each line, in the FP64 form
(already in order), the mixed form (a set) and with many equal distances (ordered
by particle and image), must equal the oracle's."""
import numpy as np
import pytest

from sphugo_gb300 import ics
from sphugo_gb300 import sim as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,sites", [(k, s) for k in (3, 5, 31, 32, 33, 64, 65, 80, 100, 128) for s in (False, True)
                                     if k > 30 or not s])  # a short list of equal distances has density 0
def test_lists_equal_the_oracle(gpu, oracle, k, sites):
    n = 1501
    x, y, vx, vy, u = ics.uniform_blast(n, 5)
    if sites:  # random sites of a 64 x 64 lattice
        p = np.random.default_rng(5).permutation(64 * 64)[:n]
        x, y = (p % 64 + 0.5) / 64, (p // 64 + 0.5) / 64
    o = oracle.OracleSim(oracle.make_params(n, k, knn_mode=oracle.KNN_EXACT), x, y, vx, vy, u)
    o.forces()
    want = o.neighbours()
    for precision in ("Exact", "Mixed"):
        s = S.Simulation(ics.periodic_config(n, k, 1e-4, precision), x, y, vx, vy, u)
        s.CalculateForces()
        got = s.neighbours()
        s.close()
        for a, b, name in zip(got, want, ("ids", "dist", "images")):
            if name == "dist" or not sites:
                assert np.array_equal(a, np.asarray(b).reshape(n, k)), (precision, name)
        if sites:  # equal distances: the farthest may be cut between equals; inside, by particle
            d, i = got[1], got[0]
            tie = d[:, 1:] == d[:, :-1]
            assert tie.any() and np.all(i[:, 1:][tie] <= i[:, :-1][tie])
