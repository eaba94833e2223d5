"""Programs that write swimmer fields on the device, through the pointers the library
hands out, between system steps: the next step spreads forces at what they wrote."""
import ctypes as C

import numpy as np
import pytest

from lbswim import _lib, lb, swimmers
from lbswim.System import System

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


class _Field:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (3, n), "typestr": "<f8", "data": (ptr, False),
                                         "version": 3}


def device_field(sw, field):
    ptr = C.c_void_p()
    _lib.check(_lib.lib.lbswim_swimmers_device_ptr(sw._h, field, C.byref(ptr)))
    return torch.as_tensor(_Field(ptr.value, sw.num), device="cuda")


def build(counts, precision):
    lat = lb.Lattice(20, 17, 40, 0.7, 0.9, precision=precision)
    lat.init_random(5)
    arrays = []
    for i, n in enumerate(counts):
        cp = swimmers.CommonParams()
        cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = 2e-3 - 3e-4 * i, 0.4, 0.05 * i, 1.0, 7 + i
        sw = swimmers.Array(n, cp)
        sw.init_random(lat, 31 + i)
        arrays.append(sw)
    return lat, arrays


# records are made ahead for one array of an FP64 lattice (of up to 32 swimmers) and for
# one to eight of the others
@pytest.mark.parametrize("counts,precision", [((1,), "f64"), ((32,), "f64"), ((40,), "f64"),
                                              ((5,), "f32"), ((400,), "f32"), ((3, 40, 9), "f32"),
                                              ((300, 2), "bf16")])
@pytest.mark.parametrize("field", [0, 2])  # positions, orientations
@pytest.mark.parametrize("early", [True, False])
def test_writes_between_system_steps(counts, precision, field, early):
    """(One lattice after the other: calls on the second would end what the first keeps.)"""
    got = []
    for steps in (system_steps, single):
        lat, arrays = build(counts, precision)
        view = device_field(arrays[-1], field) if early else None
        steps(lat, arrays, 2)
        torch.cuda.synchronize()
        if not early:
            view = device_field(arrays[-1], field)
        view.copy_(view.roll(1, 0) if field else (view + 3.5).remainder(16.0))
        torch.cuda.synchronize()
        steps(lat, arrays, 1)
        torch.cuda.synchronize()
        view.copy_(view.roll(1, 0) if field else (view + 3.5).remainder(16.0))
        torch.cuda.synchronize()
        steps(lat, arrays, 2)
        got.append((lat, arrays))
    same(*got[0], *got[1])


def system_steps(lat, arrays, n):
    system = System(lat)
    for sw in arrays:
        system.AddThing(sw)
    system.Step(n)


def single(lat, arrays, n):
    for _ in range(n):
        lat.ZeroForce()
        for sw in arrays:
            sw.AddForces(lat)
        lat.Step()
        lat.CalcHydro()
        for sw in arrays:
            sw.Move(lat)


def same(lat, arrays, ref, ref_arrays):
    for a, b in ((lat.u, ref.u), (lat.force, ref.force)):
        a.D2H()
        b.D2H()
        assert np.array_equal(a.data, b.data)
    for a, b in zip(arrays, ref_arrays):
        a.D2H()
        b.D2H()
        assert np.array_equal(a.r.data, b.r.data) and np.array_equal(a.n.data, b.n.data)


# What follows an FP64 system step ends the records made ahead, on both sides of the 32
# swimmers up to which they are made
@pytest.mark.parametrize("n", [1, 32, 33])
@pytest.mark.parametrize("exact", [False, True])
def test_f64_calls_between_system_steps(n, exact):
    def upload(_, s):
        s.D2H()
        s.r.data[:] = np.mod(s.r.data + 1.25, 16)
        s.r.H2D()

    def params(_, s):
        s.common.P = 5e-3

    def mode(on):
        return lambda la, _: la.set_compat(_lib.COMPAT_INIT_SXZ |
                                           (_lib.COMPAT_EXACT_F64 if on else 0))

    between = [upload, params, lambda la, s: s.Move(la), lambda la, s: s.AddForces(la),
               lambda la, s: s.D2H(), lambda la, s: la.ZeroForce()]
    if exact:
        between += [mode(True), upload, mode(False)]
    got = []
    for steps in (system_steps, single):
        lat, (sw,) = build((n,), "f64")
        seen = []
        for f in between:
            steps(lat, [sw], 2)
            f(lat, sw)
            steps(lat, [sw], 1)
            lat.force.D2H()
            seen.append(lat.force.data.copy())
        got.append((lat, sw, seen))
    (lat, sw, seen), (ref, rsw, want) = got
    assert all(np.array_equal(x, y) for x, y in zip(seen, want))
    same(lat, [sw], ref, [rsw])


@pytest.mark.parametrize("first", [0, 10])
def test_f64_step_of_a_one_tile_lattice(first):
    """Thirty swimmers on 4 x 8 x 32 sites, more than the tile's bucket rule admits: System.Step
    gives the bits of the single calls, whatever smaller array the lattice has seen."""
    def make():
        lat = lb.Lattice(4, 8, 32, 0.7, 0.9)
        lat.init_random(5)
        out = []
        for n in (first, 30):
            cp = swimmers.CommonParams()
            cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = 2e-3, 0.4, 0.0, 1.0, 7
            sw = swimmers.Array(n, cp) if n else None
            if sw:
                sw.init_random(lat, 31 + n)
            out.append(sw)
        return lat, out
    lat, (small, sw) = make()
    ref, (rsmall, rsw) = make()
    if first:
        lat.ZeroForce()
        small.AddForces(lat)  # the lattice has buckets from here on
    system = System(lat)
    system.AddThing(sw)
    system.Step(4)
    single(ref, [rsw], 4)
    same(lat, [sw], ref, [rsw])
