"""Boxes far below the unit box, down to where the tiles' FP32 squared
distances and the scan's approximate root reach the end of the normal range:
neighbour sets, images and distances on the tiles' path equal the oracle's, and
so does the density. A box of 2^-53 is the unit box's state scaled exactly, so
that its rounding is the unit box's."""
import numpy as np
import pytest

from sphugo_gb300 import ics
from sphugo_gb300 import sim as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,path", [(32, 8), (21, 8), (45, 4), (90, 2)])
@pytest.mark.parametrize("box", [2.0**-20, 1e-9, 2.0**-40, 1e-13, 2.0**-46, 2.0**-50, 2.0**-53, 3e-18, 1e-18, 4e-19])
def test_small_boxes(gpu, oracle, box, k, path):
    n = 3000
    x, y, vx, vy, u = ics.uniform_blast(n, 8)
    conf = ics.periodic_config(n, k, 1e-30)
    conf.HorPeriodicity = conf.VertPeriodicity = (0.0, box)
    x, y = x * box, y * box
    s = S.Simulation(conf, x, y, vx, vy, u)
    s.SetSearch(path)
    o = oracle.OracleSim(oracle.make_params(n, k, dth=conf.DeltaTHalf, alpha=1.0, beta=2.0, hor=(0.0, box), vert=(0.0, box)),
                         x, y, vx, vy, u)
    for _ in range(2):  # the second evaluation has radii, which the tiles need
        s.CalculateForces()
    o.forces()
    for a, b in zip(s.neighbours(), o.neighbours()):
        assert np.array_equal(a, b)
    d, w = s.derived(), o.state()
    for key in ("rho", "h"):
        assert np.array_equal(d[key], w[key]), key
    if box > 1e-14 and k <= 80:
        assert s.search_stats()[1] < n // 2
    s.close()
