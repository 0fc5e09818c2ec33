"""Frames draw eight disks per warp, clipped at the canvas, and colour pixels
from integer arithmetic: disks across and beyond every edge, canvases smaller
than a disk, disk counts that leave a warp part empty, densities from none to
beyond the last colour, byte for byte against the painter."""
import numpy as np
import pytest

from sphugo_gb300 import ics
from sphugo_gb300 import sim as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (3, 200), (9, 8), (10, 11), (640, 361), (2000, 1500)])
@pytest.mark.parametrize("n", [401, 1000, 4103])
def test_frames_equal_the_painter(gpu, oracle, n, w, h):
    r = np.random.default_rng(n)
    x, y = r.uniform(-0.2, 1.2, n), r.uniform(-0.2, 1.2, n)
    x[::3], y[::3] = 0.5 + r.normal(0, 0.01, len(x[::3])), 0.5 + r.normal(0, 0.01, len(x[::3]))
    x[:40] = np.round(x[:40] * w) / w  # disk centres on pixels
    conf = ics.periodic_config(n, 12, 1e-6)
    conf.HorPeriodicity = conf.VertPeriodicity = S.OPEN
    g = S.Simulation(conf, x, y, np.zeros(n), np.zeros(n), np.ones(n))
    z = r.choice(2**62, size=n, replace=False).astype(np.int64)
    g.SetDrawKeys(z)
    for _ in range(2):
        g.Step(1)
        st, rho = g.state(), g.derived()["rho"]
        want = oracle.render(st["x"], st["y"], rho, conf.ParticleMass, oracle.draw_order(z), w, h)
        assert np.array_equal(g.Frame(w, h), want)
    g.close()
    assert rho.max() / (conf.ParticleMass * n * 10) > 1  # the last colour is reached
