"""Lattices and rows are ordinary initial states: pairs on a common row or
column cost the FP64 density about what others do. (Their bits:
test_gpu_near_ties.py, test_gpu_pair_tiles.py.)"""
import numpy as np
import pytest

from sphugo_gb300 import _lib as L
from sphugo_gb300 import ics
from sphugo_gb300 import sim as S

pytestmark = pytest.mark.gpu
M = 500


def lattice(j=0.0):
    """An M x M lattice in the unit box, moved by up to 0.3 of a site times j."""
    r = np.random.default_rng(1)
    x, y = [a.ravel() for a in np.meshgrid((np.arange(M) + 0.5) / M, (np.arange(M) + 0.5) / M)]
    return x + j * r.uniform(-0.3, 0.3, M * M) / M, y + j * r.uniform(-0.3, 0.3, M * M) / M


def stages(xy, v=0.0, u=1.0, alpha=1.0, beta=2.0):
    """Stage times in milliseconds, the fastest of three profiles of four steps."""
    n, r = M * M, np.random.default_rng(2)
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
