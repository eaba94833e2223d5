"""FP64 moves of particles whose position is not a number: their velocity is not one
either, and their neighbours in the block move as ever."""
import ctypes as C

import numpy as np
import pytest

from lbswim import _lib, lb, swimmers, tracers

pytestmark = pytest.mark.gpu


def write(ptr_of, h, field, values):
    ptr = C.c_void_p()
    _lib.check(ptr_of(h, field, C.byref(ptr)))
    buf = np.ascontiguousarray(values)
    _lib.check(_lib.lib.lbswim_memcpy_h2d(ptr, buf.ctypes.data_as(C.c_void_p), buf.nbytes))


@pytest.mark.parametrize("n", [1, 21, 17000])  # one block or many, both block shapes
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_velocity_of_a_lost_point(n, bad, axis):
    size = (9, 12, 33)
    rng = np.random.default_rng([n, axis])
    lat = lb.Lattice(*size, 0.8, 0.8)
    lat.u[:] = 0.05 * rng.standard_normal((3,) + size)
    lat.u.H2D()
    r = rng.random((3, n)) * np.array(size)[:, None]
    lost = np.zeros(n, bool)
    lost[::5] = True
    hit = r.copy()
    hit[axis, lost] = bad

    out = []
    for pos in (hit, r):
        tr = tracers.Array(n)
        tr.r[:] = r
        tr.H2D()
        # in work order, which is the user's before the first move
        write(_lib.lib.lbswim_tracers_device_ptr, tr._h, 0, pos)
        tr.Move(lat)
        tr.D2H()
        sw = swimmers.Array(n, params())
        sw.r[:] = r
        sw.n[:] = np.array([[0.6], [0.0], [0.8]])
        sw.H2D()
        write(_lib.lib.lbswim_swimmers_device_ptr, sw._h, 0, pos)
        sw.Move(lat)
        sw.D2H()
        out.append((tr.v.data.copy(), tr.s.data.copy(), sw.v.data.copy(), sw.n.data.copy()))
    for got, want in zip(*out):
        assert np.all(np.isnan(got[:, lost]))
        assert np.array_equal(got[:, ~lost], want[:, ~lost])


def params():
    cp = swimmers.CommonParams()
    cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = 1e-3, 0.4, 0.0, 2.0, 5
    return cp
