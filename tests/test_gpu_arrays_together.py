"""System.Step moves and records several swimmer arrays together: the same bits as
the single calls, array by array, whatever happens between the steps."""
import numpy as np
import pytest

from lbswim import lb, swimmers
from lbswim.System import System

pytestmark = pytest.mark.gpu


def build(size, counts, precision):
    lat = lb.Lattice(*size, 0.7, 0.9, precision=precision)
    lat.init_random(5)
    arrays = []
    for i, n in enumerate(counts):
        cp = swimmers.CommonParams()
        cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = 2e-3 - 3e-4 * i, 0.4, 0.05 * i, 1.0, 7 + i
        sw = swimmers.Array(n, cp)
        sw.init_random(lat, 31 + i)
        arrays.append(sw)
    return lat, arrays


def single(lat, arrays, n=1):
    for _ in range(n):
        lat.ZeroForce()
        for sw in arrays:
            sw.AddForces(lat)
        lat.Step()
        lat.CalcHydro()
        for sw in arrays:
            sw.Move(lat)


def state(lat, arrays):
    out = []
    for f in (lat.u, lat.force):
        f.D2H()
        out.append(f.data.copy())
    for sw in arrays:
        sw.D2H()
        out += [sw.r.data.copy(), sw.v.data.copy(), sw.n.data.copy()]
    return out


# below and above the 512 ends that slabs pick from directly, one block and many,
# more arrays than one launch takes
@pytest.mark.parametrize("counts", [(3, 1), (40, 33, 64), (700, 31, 2), (1,) * 8, (5,) * 9,
                                    (64, 0, 7)])
@pytest.mark.parametrize("precision", ["f32", "f16", "f64"])
def test_together_as_apart(counts, precision):
    size = (26, 17, 40)
    lat, arrays = build(size, counts, precision)
    ref, ref_arrays = build(size, counts, precision)
    system = System(lat)
    for sw in arrays:
        system.AddThing(sw)

    def check():
        a, b = state(lat, arrays), state(ref, ref_arrays)
        assert all(np.array_equal(x, y) for x, y in zip(a, b))

    system.Step(3)
    single(ref, ref_arrays, 3)
    check()
    system.Step()
    single(ref, ref_arrays)
    for s in (arrays, ref_arrays):  # read back only: the prepared records hold
        s[0].D2H()
    system.Step()
    single(ref, ref_arrays)
    for s in (arrays, ref_arrays):  # an upload and a new parameter: they do not
        s[-1].r.data[:] = np.mod(s[-1].r.data + 1.25, 16)
        s[-1].r.H2D()
        s[0].common.P = 5e-3
    system.Step(2)
    single(ref, ref_arrays, 2)
    check()
    arrays[0].Move(lat)  # a move of its own
    ref_arrays[0].Move(ref)
    system.Step()
    single(ref, ref_arrays)
    check()
    twice = System(lat)  # the same array twice moves twice
    for sw in (arrays[0], arrays[0]):
        twice.AddThing(sw)
    twice.Step(2)
    single(ref, [ref_arrays[0], ref_arrays[0]], 2)
    check()
