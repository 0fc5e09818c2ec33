"""State and derived fields move in place when the caller's arrays are pinned
(sph_host_alloc, sph_host_register), each array for itself, and through the
staging copies when not: every mixture gives the same values, with arrays left
out as before."""
import ctypes as C

import numpy as np
import pytest

from sphugo_gb300 import _lib as L
from sphugo_gb300 import ics
from sphugo_gb300 import sim as S

pytestmark = pytest.mark.gpu


class Pinned:
    """Arrays of n doubles, some in one block from sph_host_alloc, some registered, some plain."""

    def __init__(self, lib, n, kinds):
        self.lib, self.block, self.reg = lib, C.c_void_p(), []
        L.check(lib.sph_host_alloc(8 * n * len(kinds), C.byref(self.block)))
        raw = np.ctypeslib.as_array(C.cast(self.block, C.POINTER(C.c_double)), (len(kinds), n))
        self.arrays = []
        for i, kind in enumerate(kinds):
            a = raw[i] if kind == "alloc" else np.empty(n)
            if kind == "register":
                L.check(lib.sph_host_register(a.ctypes.data, 8 * n))
                self.reg.append(a)
            self.arrays.append(a)

    def close(self):
        for a in self.reg:
            L.check(self.lib.sph_host_unregister(a.ctypes.data))
        L.check(self.lib.sph_host_free(self.block))


@pytest.mark.parametrize("n", [600, 33_333, 200_001])
@pytest.mark.parametrize("kinds", [["plain"] * 11, ["alloc"] * 11, ["register"] * 11,
                                   ["alloc", "plain", "register"] * 3 + ["plain", "alloc"]])
def test_every_kind_of_host_memory(gpu, n, kinds):
    conf = ics.periodic_config(n, 16, 1e-4, "Exact")
    x, y, _, _, u = ics.uniform_blast(n, 3)
    r = np.random.default_rng(2)
    s = S.Simulation(conf, x, y, r.normal(0, 0.3, n), r.normal(0, 0.3, n), u)
    s.Step(2)  # the slots' order is no longer the caller's
    want = list(s.state().values()) + list(s.derived().values())
    new = [v + 0.125 * r.random(n) for v in want[:8]]
    p = Pinned(gpu, n, kinds)
    h = s._h
    L.check(gpu.sph_get_state(h, *[L.dptr(a) for a in p.arrays[:8]]))
    L.check(gpu.sph_get_derived(h, *[L.dptr(a) for a in p.arrays[8:]]))
    for a, b in zip(p.arrays, want):
        assert np.array_equal(a, b)
    for a, b in zip(p.arrays[:8], new):
        a[:] = b
    L.check(gpu.sph_set_state(h, *[L.dptr(a) for a in p.arrays[:8]]))
    for a, b in zip(s.state().values(), new):
        assert np.array_equal(a, b)
    # arrays left out: zero on the way in, untouched on the way out
    args = [L.dptr(a) for a in p.arrays[:8]]
    L.check(gpu.sph_set_state(h, args[0], args[1], None, args[3], None, args[5], None, None))
    got = list(s.state().values())
    for i, b in enumerate(new):
        assert np.array_equal(got[i], b if i in (0, 1, 3, 5) else np.zeros(n)), i
    p.arrays[2][:] = 7.0
    L.check(gpu.sph_get_state(h, None, args[1], None, args[3], None, None, None, None))
    assert np.array_equal(p.arrays[1], new[1]) and np.all(p.arrays[2] == 7.0)
    L.check(gpu.sph_upload(h, args[0], args[1], None, args[3], args[4]))
    got = list(s.state().values())
    assert np.array_equal(got[0], p.arrays[0]) and np.array_equal(got[4], p.arrays[4]) and not got[2].any() and not got[5].any()
    s.close()
    p.close()
