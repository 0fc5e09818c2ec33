"""The binning's scan runs as one block, as tile sums and starts, or with a pass
over the sums between, by the cell table's size; grouping and ranking are passes
of their own or part of the scan and the permute, by the particle count. An
FP64 evaluation does not depend on the binning level, so every table size must
give the same bits."""
import numpy as np
import pytest

from sphugo_gb300 import ics
from sphugo_gb300 import sim as S

pytestmark = pytest.mark.gpu


def run(n, level, steps=2):
    conf = ics.periodic_config(n, 20, 1e-5, "Exact", grid_level=level)
    x, y, _, _, u = ics.uniform_blast(n, 9)
    r = np.random.default_rng(1)
    s = S.Simulation(conf, x, y, r.normal(0, 0.3, n), r.normal(0, 0.3, n), u)
    s.Step(steps)
    out = {**s.state(), **s.derived()}
    s.close()
    return out


@pytest.mark.parametrize("n,levels", [(4096, (1, 5, 7, 8, 13)), (4097, (4, 7, 9, 12)), (524_289, (7, 9, 11))])
def test_every_scan_path(gpu, n, levels):
    want = run(n, 6 if n < 10_000 else 10)
    for level in levels:
        got = run(n, level)
        for k in want:
            assert np.array_equal(got[k], want[k]), (level, k)
