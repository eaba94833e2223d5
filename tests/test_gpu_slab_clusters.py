"""Swimmers in a cluster on reduced-precision lattices: slabs with more ends than shared
memory holds, listed or not, give the sums of the others: whatever the slab shape, in the
step and in the force field, alone and in a batch."""
import numpy as np
import pytest

from lbswim import _lib, lb, swimmers
from lbswim.ensemble import Ensemble
from lbswim.System import System
from test_gpu_force_elements import spread_with_bound

pytestmark = pytest.mark.gpu


def build(size, n, box, tile=0, precision="f32", compat=0):
    lat = lb.Lattice(*size, 0.7, 0.9, precision=precision)
    lat.tile = tile
    lat.set_compat(_lib.COMPAT_INIT_SXZ | compat)
    lat.init_random(11)
    cp = swimmers.CommonParams()
    cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = 1e-3, 0.3, 0.1, 0.0, 3
    sw = swimmers.Array(n, cp)
    sw.init_random(lat, 21)
    sw.D2H()
    rng = np.random.default_rng(n)
    box = np.minimum(np.array(box, float), size)
    r = np.mod(np.array(size)[:, None] - 1.0 + box[:, None] * (rng.random((3, n)) - 0.5),
               np.array(size, float)[:, None])
    sw.r[:] = r
    sw.H2D()
    system = System(lat)
    system.AddThing(sw)
    return lat, system, sw


def state(lat, sw):
    out = []
    for f in (lat.u, lat.rho, lat.fOld, lat.force):
        f.D2H()
        out.append(f.data.copy())
    sw.D2H()
    return out + [sw.r.data.copy(), sw.n.data.copy()]


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


# ends a slab picks itself (up to 512 in all), lists (up to 1024) and does not (more); sums
# in 64 bits (more than 65,535 contributions to a site); short axes
CASES = [((40, 24, 64), 128, 3.0), ((40, 24, 64), 140, 3.0), ((40, 24, 64), 250, 6.0),
         ((40, 24, 64), 500, 6.0), ((70, 40, 96), 1500, 9.0), ((3, 2, 40), 300, 40.0),
         ((64, 64, 64), 40000, 30.0), ((5, 3, 7), 3000, 9.0)]


@pytest.mark.parametrize("size,n,box", CASES)
@pytest.mark.parametrize("precision", ["f32", "bf16"])
def test_clusters_in_either_shape(size, n, box, precision):
    got = []
    for tile, compat in ((0, 0), (1, 0), (0, _lib.COMPAT_WIDE_INDEX), (0, _lib.COMPAT_BULK_COPY)):
        if compat == _lib.COMPAT_BULK_COPY and size[2] % 32:
            continue
        lat, system, sw = build(size, n, [box] * 3, tile, precision, compat)
        system.Step(3)
        got.append(state(lat, sw))
    assert all(same(g, got[0]) for g in got[1:])


@pytest.mark.parametrize("size,n,box", CASES[:6])
def test_clustered_force(size, n, box):
    lat, system, sw = build(size, n, [box] * 3)
    lat.ZeroForce()
    sw.AddForces(lat)
    lat.force.D2H()
    r, nv = sw.r.data, sw.n.data
    force, _ = spread_with_bound(size, [(r - nv * 0.3, -1e-3 * nv), (r, 1e-3 * nv)])
    one, _ = spread_with_bound(size, [(r, np.full_like(r, 1e-3)), (r - nv * 0.3, np.full_like(r, 1e-3))])
    # FP32: a weight is off by 2^-23 or so, a contribution by a unit of the fixed-point sums,
    # 2^-22 of the largest force
    tol = 8 * 2.0 ** -23 * one.astype(float) + 64 * n * 2.0 ** -31 * 1e-3 + 64 * 2.0 ** -22 * 1e-3
    assert np.all(np.abs(lat.force.data.reshape(3, -1) - force) <= tol)


def test_clusters_in_a_batch():
    members = [((40, 24, 64), 500, 6.0), ((70, 9, 33), 40, 9.0), ((40, 24, 64), 140, 3.0)]
    batch = [build(s, n, [b] * 3, m % 2) for m, (s, n, b) in enumerate(members)]
    ens = Ensemble([(lat, sw, None) for lat, _, sw in batch])
    ens.Step(4)
    for m, (s, n, b) in enumerate(members):
        alone, system, sw = build(s, n, [b] * 3, m % 2)
        system.Step(4)
        assert same(state(batch[m][0], batch[m][2]), state(alone, sw))
