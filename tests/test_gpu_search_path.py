"""Which search a handle runs, seen by how many queries are left to the
per-query one: without a choice that search for FP64 handles of up to 16,384
particles and tiles for the others; an explicit choice of tiles is one."""
import numpy as np
import pytest

from sphugo_gb300 import _lib as L
from sphugo_gb300 import ics
from sphugo_gb300 import sim as S
import test_gpu_parity as parity

pytestmark = pytest.mark.gpu


def run(n, k, precision="Exact", path=None, steps=2):
    x, y, vx, vy, u = ics.uniform_blast(n, 9)
    s = S.Simulation(ics.periodic_config(n, k, 1e-5, precision), x, y, vx, vy, u)
    if path is not None:
        s.SetSearch(path)
    s.Step(steps)
    return s


@pytest.mark.parametrize("n,k", [(6000, 8), (6000, 32), (6000, 64), (16_384, 100), (16_384, 128)])
def test_tiles_on_request(gpu, n, k):
    """1 means tiles at every particle count; their results are the default's."""
    a, b, c = run(n, k), run(n, k, path=True), run(n, k, path=0)
    assert a.search_stats() == (n, n) and c.search_stats() == (n, n)
    assert b.search_stats()[1] < (n if k > 80 else n // 4)
    sa, sb = a.state(), b.state()
    for key in sa:
        assert np.array_equal(sa[key], sb[key]), key
    for p, q in zip(a.neighbours(), b.neighbours()):
        assert np.array_equal(p, q)


@pytest.mark.parametrize("n,precision,tiles", [(16_384, "Exact", False), (16_385, "Exact", True), (6000, "Mixed", True)])
def test_default(gpu, n, precision, tiles):
    d = run(n, 32, precision).search_stats()[1]
    assert d < n // 4 if tiles else d == n


def append(s, gpu, x, y):
    L.check(gpu.sph_append(s._h, len(x), L.dptr(x), L.dptr(y), None, None, None, None))
    s.n += len(x)


@pytest.mark.parametrize("path", [None, 8, 2])
def test_default_goes_on_after_a_checkpoint(gpu, tmp_path, path):
    """A run below 16,384 particles, saved, loaded and grown beyond by sph_append
    takes the search that the uninterrupted run takes, with its results; a choice
    of tiles stays."""
    n, more, k = 16_000, 900, 32
    r = np.random.default_rng(4)
    x, y = r.random(more), r.random(more)
    a = run(n, k, path=path)
    a.Save(tmp_path / "s.ck")
    xi, yi, vx, vy, u = ics.uniform_blast(n, 9)
    b = S.Simulation(ics.periodic_config(n, k, 1e-5), xi, yi, vx, vy, u)
    b.Load(tmp_path / "s.ck")
    a.Step(1)
    b.Step(1)
    assert a.search_stats() == b.search_stats()
    for s in (a, b):
        append(s, gpu, x, y)
        s.Step(2)
        assert s.search_stats()[0] == n + more and s.search_stats()[1] < n // 4
    sa, sb = a.state(), b.state()
    for key in sa:
        assert np.array_equal(sa[key], sb[key]), key


def scene(name, seed=9):
    """Small states whose default search is the per-query one, and whether tiles settle most of their queries."""
    if name == "walls":  # open axes, gravity, reflections
        n = 2000
        x, y, vx, vy, u = ics.uniform_blast(n, seed)
        conf = S.SphConfig(DeltaTHalf=5e-4, Gamma=5 / 3, ParticleMass=1.0 / n, Acceleration=S.Vec2(0.0, 0.5), Kernel="Wendtland",
                           Reflections=S.Reflections(L=0.31, R=S.DBL_MAX, U=-S.DBL_MAX, D=0.69), ViscosityAlpha=1.0,
                           ViscosityBeta=2.0)
        return conf, (0.3 + 0.4 * x, 0.2 + 0.5 * y, vx, vy, u), 10, True
    if name == "box":  # neither unit nor square
        n = 1500
        x, y, vx, vy, u = ics.uniform_blast(n, seed)
        conf = S.SphConfig(DeltaTHalf=1e-4, Gamma=5 / 3, ParticleMass=1.0 / n, HorPeriodicity=(0.2, 0.8),
                           VertPeriodicity=(-1.0, 1.0), ViscosityAlpha=1.0, ViscosityBeta=2.0)
        return conf, (0.2 + 0.6 * x, -1.0 + 2.0 * y, vx, vy, u), 6, True
    if name == "far":  # far from the origin
        n = 2000
        x, y, vx, vy, u = ics.uniform_blast(n, seed)
        conf = S.SphConfig(DeltaTHalf=1e-4, Gamma=5 / 3, ParticleMass=1.0 / n, HorPeriodicity=(1000.0, 1001.0),
                           VertPeriodicity=(-3000.0, -2998.0), ViscosityAlpha=1.0, ViscosityBeta=2.0)
        return conf, (1000.0 + x, -3000.0 + 2.0 * y, vx, vy, u), 6, True
    n, k = {"images": (64, 32), "few": (40, 16), "long": (200, 64), "blast": (10_000, 32), "k45": (3000, 45)}[name]
    return ics.periodic_config(n, k, 1e-4), ics.uniform_blast(n, n), 3, n > 1000


@pytest.mark.parametrize("path", [1, 2, 4, 8])
@pytest.mark.parametrize("name", ["walls", "box", "far", "images", "few", "long", "blast", "k45"])
def test_tiles_of_small_states(gpu, oracle, name, path):
    conf, arrs, steps, most = scene(name)
    k = conf.NeighbourCount
    if path in (4, 8) and k > (37 if path == 8 else 80):
        pytest.skip("no block tiles of that many warps for this k")
    g, o = parity.pair(oracle, conf, arrs)
    g.SetSearch(path)
    g.Step(steps)
    o.step(steps)
    parity.assert_bitwise(g, o)
    if most:
        assert g.search_stats()[1] < len(arrs[0])
    g.close()
