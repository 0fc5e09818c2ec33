"""The block tiles sort only the first 16, 32 or 64 of a query's 24, 40 or 72
candidates and scan the rows of cells four at a time: list lengths on both
sides of each of those lines, with rows of one particle and of many, must give
the per-query search's lists and FP64 results bit for bit."""
import numpy as np
import pytest

from sphugo_gb300 import ics
from sphugo_gb300 import sim as S

pytestmark = pytest.mark.gpu


def run(arrs, k, precision, tiles):
    s = S.Simulation(ics.periodic_config(len(arrs[0]), k, 1e-5, precision), *arrs)
    s.SetSearch(tiles)
    s.CalculateForces()
    s.CalculateForces()  # the first has no previous smoothing lengths: per-query search
    out = s.neighbours(), s.derived(), s.state()
    s.close()
    return out


@pytest.mark.parametrize("k", [3, 13, 15, 16, 17, 20, 31, 33, 45, 63, 65])
@pytest.mark.parametrize("ic", [ics.uniform_blast, ics.clustered])
def test_lists_equal_the_per_query_search(gpu, ic, k):
    x, y, _, _, u = ic(20_011, 6)
    r = np.random.default_rng(6)
    arrs = x, y, r.normal(0, 0.3, len(x)), r.normal(0, 0.3, len(x)), u
    for precision in ("Exact", "Mixed"):
        ref = run(arrs, k, precision, 0)
        for tiles in (8, 4, 2) if k <= 37 else (4, 2):
            got = run(arrs, k, precision, tiles)
            for a, b in zip(got[0], ref[0]):
                assert np.array_equal(a, b), (precision, tiles)
            if precision == "Exact":
                for f, g in zip(got[1:], ref[1:]):
                    for key in g:
                        assert np.array_equal(f[key], g[key]), (tiles, key)
