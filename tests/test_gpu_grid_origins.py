"""The binning takes positions to cells without FP64 arithmetic where a
periodic axis starts at 0 and its cells per unit are a power of two, and with it
elsewhere, per axis: boxes on both sides of that line, their particles drifting
across their edges, must equal the oracle bit for bit."""
import numpy as np
import pytest

from sphugo_gb300 import ics
from test_gpu_pair_tiles import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hor,vert", [((0.0, 1.0), (0.0, 1.0)), ((0.0, 2.0), (0.0, 0.75)), ((-1.0, 1.0), (0.0, 0.5)),
                                      ((0.0, 1.5), (5.0, 6.0)), ((0.0, 0.125), (0.0, 0.125))])
def test_boxes_equal_the_oracle(gpu, oracle, hor, vert):
    n = 3001
    w = hor[1] - hor[0], vert[1] - vert[0]
    conf = ics.periodic_config(n, 24, 0.01)
    conf.HorPeriodicity, conf.VertPeriodicity = hor, vert
    x, y, _, _, u = ics.uniform_blast(n, 21)
    r = np.random.default_rng(21)
    check(oracle, conf, (hor[0] + x * w[0], vert[0] + y * w[1], r.normal(0, w[0], n), r.normal(0, w[1], n), u * min(w) ** 2), steps=3)
