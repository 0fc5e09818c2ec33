"""The FP64 density and force deal (particle, entry) pairs over warps in tiles
of W = 1 .. 32 particles, W by the particle count: every width, ragged last
tiles, lists of two entries to several ragged chunks, both kernels, and the
operands the unchecked integer arithmetic leaves to the hardware (coincident
coordinates, equal velocities, tiny and huge values, viscosity off) must equal
the oracle bit for bit."""
import numpy as np
import pytest

from sphugo_gb300 import ics
from sphugo_gb300 import sim as S

pytestmark = pytest.mark.gpu

STATE = ["x", "y", "vx", "vy", "u", "ax", "ay", "udot"]


def check(O, conf, arrs, steps=1):
    n = len(arrs[0])
    g = S.Simulation(conf, *arrs)
    r = conf.Reflections
    o = O.OracleSim(O.make_params(
        n, conf.NeighbourCount, kernel=0 if conf.Kernel == "Monahan" else 1, knn_mode=O.KNN_EXACT, gamma=conf.Gamma,
        mass=conf.ParticleMass, dth=conf.DeltaTHalf, accel=(conf.Acceleration.X, conf.Acceleration.Y),
        hor=conf.HorPeriodicity, vert=conf.VertPeriodicity, refl=(r.L, r.R, r.U, r.D), alpha=conf.ViscosityAlpha,
        beta=conf.ViscosityBeta, etasq=conf.ViscosityEtaSq), *arrs)
    g.Step(steps)
    o.step(steps)
    gs, gd, os_ = g.state(), g.derived(), o.state()
    g.close()
    for k in STATE:
        assert np.array_equal(gs[k], os_[k]), (k, int(np.sum(gs[k] != os_[k])))
    for k in ("rho", "c", "h"):
        assert np.array_equal(gd[k], os_[k]), (k, int(np.sum(gd[k] != os_[k])))


def flow(n, seed):
    x, y, _, _, u = ics.uniform_blast(n, seed)
    r = np.random.default_rng(seed)
    return x, y, r.normal(0, 0.3, n), r.normal(0, 0.3, n), u


# 2,432 to 4,864 warps are resident at once: the widths change at their multiples
@pytest.mark.parametrize("n", [129, 2433, 4867, 9731, 19461, 38913, 77827])
@pytest.mark.parametrize("k,kernel", [(32, "Monahan"), (21, "Wendtland")])
def test_every_tile_width(gpu, oracle, n, k, kernel):
    conf = ics.periodic_config(n, k, 1e-4)
    conf.Kernel = kernel
    check(oracle, conf, flow(n, 11))


@pytest.mark.parametrize("k", [2, 7, 8, 9, 16, 17, 31, 33, 47, 65, 96])
def test_every_chunk_shape(gpu, oracle, k):
    for n in (301, 100_003):  # one particle per warp, and 32
        check(oracle, ics.periodic_config(n, k, 1e-5), flow(n, 12))


@pytest.mark.parametrize("n", [900, 90_000])
def test_operands_left_to_the_hardware(gpu, oracle, n):
    r = np.random.default_rng(3)
    g = int(np.sqrt(n))
    x, y = (r.integers(0, g, n) + 0.5) / g, r.random(n)  # columns: differences of zero in x
    z = np.zeros(n)
    for vx, vy, dt in [(z, z, 1e-4),                                        # at rest
                       (np.full(n, 0.25), r.normal(0, 1e-170, n), 1e-4),    # equal, and tiny, velocities
                       (r.normal(0, 1e-306, n), r.normal(0, 1e-306, n), 1e-300),  # products below the normal range
                       (1e37 * np.sign(np.sin(7 * x)), z, 1e-100)]:         # huge ones
        check(oracle, ics.periodic_config(n, 32, dt), (x, y, vx, vy, np.ones(n)))
    x, y, vx, vy, u = flow(n, 5)
    for alpha, beta in ((0.0, 0.0), (0.0, 2.0), (1.0, 0.0), (1e-60, 1e50), (-1.0, -0.5)):
        conf = ics.periodic_config(n, 32, 1e-4)
        conf.ViscosityAlpha, conf.ViscosityBeta = alpha, beta
        check(oracle, conf, (x, y, vx, vy, u))
    check(oracle, ics.periodic_config(n, 32, 1e-4), (x, y, vx, vy, np.where(r.random(n) < 0.5, 0.0, u)))  # c = 0


@pytest.mark.parametrize("n,k,kernel", [(333, 32, "Monahan"), (3001, 21, "Wendtland"), (16384, 32, "Monahan"), (2500, 9, "Monahan"),
                                        (5000, 65, "Monahan"), (1200, 128, "Monahan")])
def test_mixed_force_same_bits_pair_by_pair(gpu, n, k, kernel):
    """The mixed force deals its pairs over the lanes up to 16,384 particles
    and runs one thread per particle beyond: a simulation alone, and as a member
    of a larger ensemble, gives the same bits (per-query search in both, whose
    list order does not depend on the other members)."""
    conf, big = ics.periodic_config(n, k, 1e-4, "Mixed"), ics.periodic_config(20_000, k, 1e-4, "Mixed")
    conf.Kernel = kernel
    arrs = flow(n, 21)
    one, many = S.Simulation(conf, *arrs), S.Ensemble([big, conf], [flow(20_000, 22), arrs])
    for s in (one, many):
        s.SetSearch(False)
        s.Step(3)
    a, b, da, db = one.state(), many.state(), one.derived(), many.derived()
    for key in a:
        assert np.array_equal(a[key], b[key][20_000:]), key
    for key in da:
        assert np.array_equal(da[key], db[key][20_000:]), key


# one past a full pass of 32 particles per resident warp, in the force
# (3,040 or 3,800 warps), in the density (4,864), and past two of them
@pytest.mark.parametrize("n", [97_281, 121_601, 155_649, 182_401, 204_289, 311_297])
def test_full_tiles_and_a_rest(gpu, oracle, n):
    check(oracle, ics.periodic_config(n, 13, 1e-5), flow(n, 14))
