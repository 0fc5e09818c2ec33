"""Lattices and rows, states at rest, cold gases and runs without viscosity are
ordinary: pairs with zeros among their operands cost the FP64 density and force
about what others do. (Their bits: test_gpu_near_ties.py and
test_gpu_pair_tiles.py; pairs with several of these zeros together here.)"""
import numpy as np
import pytest

from sphugo_gb300 import _lib as L
from sphugo_gb300 import ics
from sphugo_gb300 import sim as S

pytestmark = pytest.mark.gpu
M = 500


def lattice(j=0.0, m=M):
    """An m x m lattice in the unit box, moved by up to 0.3 of a site times j."""
    r = np.random.default_rng(1)
    x, y = [a.ravel() for a in np.meshgrid((np.arange(m) + 0.5) / m, (np.arange(m) + 0.5) / m)]
    return x + j * r.uniform(-0.3, 0.3, m * m) / m, y + j * r.uniform(-0.3, 0.3, m * m) / m


def stages(xy, v=0.0, u=1.0, alpha=1.0, beta=2.0):
    """Stage times in milliseconds, the fastest of three profiles of four steps."""
    n, r = len(xy[0]), np.random.default_rng(2)
    conf = ics.periodic_config(n, 28, 1e-6, alpha=alpha, beta=beta)
    s = S.Simulation(conf, *xy, r.normal(0, 1, n) * v, r.normal(0, 1, n) * v, np.full(n, u))
    s.Step(1)
    best = np.full(L.NUM_STAGES, np.inf)
    for _ in range(3):
        st = np.zeros(L.NUM_STAGES)
        L.check(L.load().sph_step_profiled(s._h, 4, L.dptr(st)))
        best = np.minimum(best, st)
    s.close()
    return dict(zip(L.STAGES, best))


def test_density_of_a_lattice(gpu):
    """At rest a uniform lattice stays one. Four times the jittered lattice's
    time with such pairs on the hardware's path; the bound leaves room for a few
    instructions a pair and for the spread of short kernels."""
    at, jit = stages(lattice()), stages(lattice(1))
    assert at["density"] < 1.5 * jit["density"], (at, jit)


def test_search_of_a_lattice(gpu):
    """Every list of a perfect lattice has equal distances and is ordered again
    in FP64: 2.7 times a jittered one's search, 3.3 before lists in order were
    left as they are."""
    at, jit = stages(lattice(0, 1024)), stages(lattice(1, 1024))
    assert at["knn"] < 3.0 * jit["knn"], (at, jit)


@pytest.mark.parametrize("name,state", [
    ("lattice at rest", dict(xy=lattice())), ("lattice, cold", dict(xy=lattice(), v=0.1, u=0.0)),
    ("cold", dict(xy=lattice(1), v=0.1, u=0.0)), ("cold at rest", dict(xy=lattice(1), u=0.0)),
    ("no alpha", dict(xy=lattice(1), v=0.1, alpha=0.0)), ("inviscid", dict(xy=lattice(1), v=0.1, alpha=0.0, beta=0.0))])
def test_force_of_states_with_zeros(gpu, name, state):
    """1.6 to 3.3 times a jittered warm lattice's time with the hardware's
    arithmetic for such pairs; 0.7 to 1.1 without."""
    at, jit = stages(**state), stages(lattice(1), v=0.1)
    assert at["force_integrate"] < 1.4 * jit["force_integrate"], (name, at, jit)


@pytest.mark.parametrize("m", [23, 61])
@pytest.mark.parametrize("alpha,beta", [(1.0, 2.0), (0.0, 2.0), (1.0, 0.0), (0.0, 0.0)])
def test_zeros_together(gpu, oracle, m, alpha, beta):
    """Zeros in r_AB, v_AB, c and the viscosities in one state, coincident
    coordinates beside differences below 2^-150, and energies that are zero for
    some of the particles."""
    n, r = m * m, np.random.default_rng(6)
    x, y = [a.ravel() for a in np.meshgrid((np.arange(m) + 0.5) / m, (np.arange(m) + 0.5) / m)]
    jx, jy = x + np.where(r.random(n) < 0.5, 0.0, r.uniform(-0.2, 0.2, n) / m), y.copy()
    for vx, vy in ((np.zeros(n), np.zeros(n)), (r.integers(-1, 2, n) * 0.25, r.integers(-1, 2, n) * 0.25),
                   (r.integers(-1, 2, n) * 1e-50, r.integers(-1, 2, n) * 0.5)):
        for u in (np.zeros(n), np.where(r.random(n) < 0.5, 0.0, 1.0), np.ones(n)):
            conf = ics.periodic_config(n, 20, 1e-5, alpha=alpha, beta=beta)
            for px, py in ((x, y), (jx, jy)):
                g = S.Simulation(conf, px, py, vx, vy, u)
                o = oracle.OracleSim(oracle.make_params(n, 20, dth=conf.DeltaTHalf, alpha=alpha, beta=beta), px, py, vx, vy, u)
                for steps in (1, 2):
                    g.Step(steps)
                    o.step(steps)
                    got, want = {**g.state(), **g.derived()}, o.state()
                    for key in got:
                        assert np.array_equal(got[key], want[key]), (key, int(np.sum(got[key] != want[key])))
                g.close()
