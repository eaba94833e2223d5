"""FP64 force spreading: every way a force tile sums its ends (integers, in units
made coarser for crowded tiles and folded stencils; FP64 in end order for full
buckets, forces out of the integers' range and dense suspensions) against sums in
extended precision."""
import numpy as np
import pytest

from lbswim import _lib, lb, swimmers

pytestmark = pytest.mark.gpu
X = np.longdouble


def weights(r):
    """Stencil nodes [4, n] and Peskin weights [4, n] of one coordinate."""
    x0 = np.ceil(r - 2)
    node = x0 + np.arange(4)[:, None]
    x = np.abs(r.astype(X) - node.astype(X))
    inner = (3 - 2 * x + np.sqrt(np.maximum(1 + 4 * x - 4 * x * x, 0))) / 8
    outer = (5 - 2 * x - np.sqrt(np.maximum(-7 + 12 * x - 4 * x * x, 0))) / 8
    return node.astype(np.int64), np.where(x < 1, inner, np.where(x < 2, outer, 0))


def spread(force, count, size, r, F):
    idx, w = zip(*[weights(r[d]) for d in range(3)])
    for i in range(4):
        for j in range(4):
            for k in range(4):
                s = np.ravel_multi_index([idx[0][i] % size[0], idx[1][j] % size[1],
                                          idx[2][k] % size[2]], size)
                wt = w[0][i] * w[1][j] * w[2][k]
                for c in range(3):
                    np.add.at(force[c], s, wt * F[c])
                np.add.at(count, s, 1)


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("size,n,box", [
    ((4, 8, 32), 1, 1.0), ((9, 17, 65), 40, 1.0), ((16, 16, 40), 1200, 1.0),
    ((8, 16, 64), 100, 0.1),    # 100 to 200 ends in one tile: coarser units
    ((8, 16, 64), 190, 0.02),   # more than a bucket holds
    ((8, 8, 32), 400, 1.0),     # too dense for buckets
    ((1, 5, 7), 6, 1.0), ((3, 2, 40), 9, 1.0), ((2, 3, 2), 60, 1.0), ((5, 1, 1), 30, 1.0)])
def test_force_of_two_arrays(size, n, box, exact):
    rng = np.random.default_rng([n, size[2]])
    lat = lb.Lattice(*size, 0.8, 0.8)
    if exact:
        lat.set_compat(_lib.COMPAT_INIT_SXZ | _lib.COMPAT_EXACT_F64)
    N = size[0] * size[1] * size[2]
    force = np.zeros((3, N), X)
    count = np.zeros(N)
    lat.ZeroForce()
    arrays, largest = [], 0.0
    for P in (1e-3, 0.7):
        cp = swimmers.CommonParams()
        cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = P, 0.3, 0.0, 1.0, 1
        sw = swimmers.Array(n, cp)
        sw.r[:] = rng.random((3, n)) * (box * np.array(size)[:, None])
        sw.r[:, 0] = 0.0  # on a node, at the box's corner
        nv = rng.standard_normal((3, n))
        sw.n[:] = nv / np.linalg.norm(nv, axis=0)
        sw.H2D()
        sw.AddForces(lat)
        arrays.append(sw)
        nv = sw.n.data
        spread(force, count, size, sw.r.data - nv * 0.3, -P * nv.astype(X))
        spread(force, count, size, sw.r.data, P * nv.astype(X))
        largest = max(largest, P)
    lat.force.D2H()
    # an FP64 weight is off by at most 2^-54, a contribution (three weights of
    # at most 1/2 and a force) by less than 2^-54 of the force, the addition of
    # one more by another 2^-53
    tol = (count + 1) * 2.0 ** -52 * largest
    assert np.all(np.abs(lat.force.data.reshape(3, N) - force) <= tol)


@pytest.mark.parametrize("P", [0.0, -2.0, 1e-290, 1e-305, 1e290, 1e305])
def test_force_scales(P):
    size, n = (6, 9, 33), 25
    rng = np.random.default_rng(7)
    lat = lb.Lattice(*size, 0.8, 0.8)
    cp = swimmers.CommonParams()
    cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = P, 0.5, 0.0, 1.0, 1
    sw = swimmers.Array(n, cp)
    sw.r[:] = rng.random((3, n)) * np.array(size)[:, None]
    sw.n[:] = rng.standard_normal((3, n))
    sw.H2D()
    for _ in range(3):  # the words for the largest force alternate
        lat.ZeroForce()
        sw.AddForces(lat)
    lat.force.D2H()
    N = size[0] * size[1] * size[2]
    force, count = np.zeros((3, N), X), np.zeros(N)
    spread(force, count, size, sw.r.data - sw.n.data * 0.5, -X(P) * sw.n.data)
    spread(force, count, size, sw.r.data, X(P) * sw.n.data)
    largest = float(np.abs(X(P) * sw.n.data).max())
    tol = (count + 1) * 2.0 ** -52 * largest
    assert np.all(np.abs(lat.force.data.reshape(3, N) - force) <= tol)


@pytest.mark.parametrize("size", [(75, 60, 50), (77, 60, 50)])  # 304 and 320 tiles
@pytest.mark.parametrize("n,box", [(40, 1.0), (4000, 1.0), (100, 0.02), (190, 0.01)])
def test_force_of_either_block_size(size, n, box):
    rng = np.random.default_rng([n, size[0]])
    lat = lb.Lattice(*size, 0.8, 0.8)
    cp = swimmers.CommonParams()
    cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = 0.3, 0.4, 0.0, 1.0, 1
    sw = swimmers.Array(n, cp)
    sw.r[:] = rng.random((3, n)) * (box * np.array(size)[:, None])
    nv = rng.standard_normal((3, n))
    sw.n[:] = nv / np.linalg.norm(nv, axis=0)
    sw.H2D()
    lat.ZeroForce()
    sw.AddForces(lat)
    sw.AddForces(lat)
    lat.force.D2H()
    N = size[0] * size[1] * size[2]
    force, count = np.zeros((3, N), X), np.zeros(N)
    nv = sw.n.data
    spread(force, count, size, sw.r.data - nv * 0.4, -0.3 * nv.astype(X))
    spread(force, count, size, sw.r.data, 0.3 * nv.astype(X))
    # as above, twice
    tol = (2 * count + 1) * 2.0 ** -52 * 0.3
    assert np.all(np.abs(lat.force.data.reshape(3, N) - 2 * force) <= tol)
