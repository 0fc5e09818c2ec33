"""Lattices, rows and columns, at rest and after a small displacement: many
squared distances equal or within FP32's rounding of one another, in the lists
and at their ends. Neighbour sets, their order and everything that follows must
equal the oracle bit for bit on every search path."""
import numpy as np
import pytest

from sphugo_gb300 import ics
from sphugo_gb300 import sim as S

pytestmark = pytest.mark.gpu


def lattice(m, jx=0.0, jy=0.0):
    """An m x m lattice in the unit box, x and y moved by up to 0.3 of a site times jx and jy."""
    r = np.random.default_rng(1)
    x, y = [a.ravel() for a in np.meshgrid((np.arange(m) + 0.5) / m, (np.arange(m) + 0.5) / m)]
    return x + jx * r.uniform(-0.3, 0.3, m * m) / m, y + jy * r.uniform(-0.3, 0.3, m * m) / m


def against_oracle(O, conf, arrs, steps=2, path=None):
    n = len(arrs[0])
    g = S.Simulation(conf, *arrs)
    if path is not None:
        g.SetSearch(path)
    o = O.OracleSim(O.make_params(
        n, conf.NeighbourCount, kernel=0 if conf.Kernel == "Monahan" else 1, gamma=conf.Gamma, mass=conf.ParticleMass,
        dth=conf.DeltaTHalf, hor=conf.HorPeriodicity, vert=conf.VertPeriodicity, alpha=conf.ViscosityAlpha,
        beta=conf.ViscosityBeta, etasq=conf.ViscosityEtaSq), *arrs)
    g.Step(steps)
    o.step(steps)
    for a, b in zip(g.neighbours(), o.neighbours()):
        assert np.array_equal(a, b)
    got, want = {**g.state(), **g.derived()}, o.state()
    g.close()
    for key in got:
        assert np.array_equal(got[key], want[key]), (key, int(np.sum(got[key] != want[key])))


@pytest.mark.parametrize("kernel", ["Monahan", "Wendtland"])
@pytest.mark.parametrize("jx,jy", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("m", [31, 131])
def test_lattices_rows_and_columns(gpu, oracle, m, jx, jy, kernel):
    n, r = m * m, np.random.default_rng(2)
    conf = ics.periodic_config(n, 28, 1e-6)
    conf.Kernel = kernel
    z, v = np.zeros(n), r.normal(0, 0.3, n)
    for vx, vy in ((z, z), (v, z)):
        against_oracle(oracle, conf, (*lattice(m, jx, jy), vx, vy, r.uniform(0.5, 2.0, n)))


# 28, 60 and 88 close a shell of the lattice; the others end inside one
@pytest.mark.parametrize("path", [0, 2, 4, 8])
@pytest.mark.parametrize("k", [16, 28, 32, 60, 64, 80, 88, 100, 128])
def test_nearly_equal_distances(gpu, oracle, k, path):
    if (path == 8 and k > 37) or (path == 4 and k > 80):
        pytest.skip("no block tiles of that many warps for this k")
    m, r = 47, np.random.default_rng(3)
    for noise in (0.0, 1e-8, 1e-6, 1e-5):
        against_oracle(oracle, ics.periodic_config(m * m, k, 1e-6), (
            *lattice(m, noise, noise), r.normal(0, 0.1, m * m), r.normal(0, 0.1, m * m), np.ones(m * m)), path=path)


def test_three_near_ties_in_a_long_list(gpu, oracle):
    """A list of 128 of 100,003 random particles has a few such cases."""
    n, r = 100_003, np.random.default_rng(12)
    x, y, _, _, u = ics.uniform_blast(n, 12)
    against_oracle(oracle, ics.periodic_config(n, 128, 1e-5), (x, y, r.normal(0, 0.3, n), r.normal(0, 0.3, n), u), steps=1)


# lists of up to 32, 64 and 80 entries (each closes a shell, so that the tiles decide the sets)
@pytest.mark.parametrize("k,path", [(28, 8), (28, 4), (60, 4), (80, 4)])
def test_equal_distances_in_block_tiles(gpu, oracle, k, path):
    """A lattice whose distances within a shell are equal in FP64, its ids in
    random order: the block tiles' lists are ordered by (distance, id, image)."""
    m, r = 64, np.random.default_rng(5)
    n = m * m
    x, y = lattice(m)
    p = r.permutation(n)
    z, conf = np.zeros(n), ics.periodic_config(n, k, 1e-6)
    arrs = (x[p], y[p], z, z, np.ones(n))
    against_oracle(oracle, conf, arrs, steps=2, path=path)
    g = S.Simulation(conf, *arrs)
    g.SetSearch(path)
    g.Step(2)
    assert g.search_stats()[1] < n // 2
    g.close()
