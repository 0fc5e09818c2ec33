"""Transfers through pageable host arrays run in the slots' order, without the
map to the caller's order that arrays in pinned memory need: one kernel and its
copies. Beyond 1,048,576 particles state and derived fields are read out in the
caller's order."""
import numpy as np
import pytest

from sphugo_gb300 import _lib as L
from sphugo_gb300 import ics
from sphugo_gb300 import sim as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1_048_576, 1_048_577])
def test_either_order_reads_the_same(gpu, n):
    x, y, vx, vy, u = ics.uniform_blast(n, 3)
    r = np.random.default_rng(1)
    s = S.Simulation(ics.periodic_config(n, 8, 1e-6, "Mixed"), x, y, vx, vy, u)
    s.Step(1)
    plain = list(s.state().values()) + list(s.derived().values())
    pinned = [np.empty(n) for _ in plain]
    for a in pinned:
        L.check(gpu.sph_host_register(a.ctypes.data, 8 * n))
    L.check(gpu.sph_get_state(s._h, *[L.dptr(a) for a in pinned[:8]]))
    L.check(gpu.sph_get_derived(s._h, *[L.dptr(a) for a in pinned[8:]]))
    for a, b in zip(plain, pinned):
        assert np.array_equal(a, b)
    new = [v + 0.01 * r.random(n) for v in plain[:8]]
    s.set_state(*new)  # pageable
    L.check(gpu.sph_get_state(s._h, *[L.dptr(a) for a in pinned[:8]]))
    for a, b in zip(new, pinned):
        assert np.array_equal(a, b)
    for a in pinned:
        L.check(gpu.sph_host_unregister(a.ctypes.data))
    s.close()


def kernels(f):
    """Names of the kernels that f launches."""
    from torch import profiler
    with profiler.profile(activities=[profiler.ProfilerActivity.CPU, profiler.ProfilerActivity.CUDA]) as p:
        f()
    return [e.name for e in p.events() if "sphgpu" in e.name]


def test_pageable_arrays_need_no_map(gpu):
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    n = 10_000
    s = S.Simulation(ics.periodic_config(n, 32, 1e-5), *ics.uniform_blast(n, 3))
    s.Step(2)
    z = [np.zeros(n) for _ in range(8)]
    p = [L.dptr(a) for a in z]
    calls = {"k_gather_state": lambda: L.check(gpu.sph_get_state(s._h, *p)),
             "k_gather_derived": lambda: L.check(gpu.sph_get_derived(s._h, *p[:3])),
             "k_scatter_state": lambda: L.check(gpu.sph_set_state(s._h, *p))}
    kernels(calls["k_gather_state"])  # (a process's first profile may be empty)
    if not kernels(calls["k_gather_state"]):
        pytest.skip("the profiler records no kernels here")
    for name, call in calls.items():
        ran = kernels(call)
        if not ran:
            pytest.skip("the profiler records no kernels here")
        assert len(ran) == 1 and name in ran[0], (name, ran)
