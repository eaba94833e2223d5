"""Host buffers of the caller's that a kernel cannot take as they are: page-locked memory at
an odd address goes through copies."""
import ctypes as C

import numpy as np
import pytest

from lbswim import _lib, lb, swimmers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 100, 5000])  # written by a kernel up to 4096 swimmers
@pytest.mark.parametrize("shift", [0, 8, 4, 1])
@pytest.mark.parametrize("fields", [(0, 1, 2), (1,), (0, 2)])
def test_swimmers_into_any_address(n, shift, fields):
    lat = lb.Lattice(12, 8, 33, 0.8, 0.8)
    cp = swimmers.CommonParams()
    cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = 1e-3, 0.3, 0.0, 1.0, 1
    sw = swimmers.Array(n, cp)
    sw.init_random(lat, 3)
    sw.Move(lat)
    want = []
    for a in (sw.r, sw.v, sw.n):
        a.D2H()
        want.append(a.data.copy())
    room = 24 * n + 16
    blocks = [_lib._PinnedBlock(room) for _ in range(3)]
    ptrs = [b.ptr.value + shift for b in blocks]
    for p in ptrs:
        C.memset(p - shift, 0x55, room)
    args = [C.cast(C.c_void_p(p if f in fields else None), C.POINTER(C.c_double))
            for f, p in enumerate(ptrs)]
    _lib.check(_lib.lib.lbswim_swimmers_d2h_all(sw._h, *args))
    for f, p in enumerate(ptrs):
        raw = np.frombuffer(C.string_at(p - shift, room), np.uint8)
        mid = raw[shift:shift + 24 * n]
        if f in fields:
            assert mid.tobytes() == want[f].tobytes()
        else:
            assert np.all(mid == 0x55)
        assert np.all(raw[:shift] == 0x55) and np.all(raw[shift + 24 * n:] == 0x55)
