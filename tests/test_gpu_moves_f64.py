"""FP64 particle moves: velocities interpolated in integers (and in FP64 where
those do not fit: values of every size, zeros) against sums in extended precision,
and the new positions and orientations."""
import numpy as np
import pytest

from lbswim import _lib, lb, swimmers, tracers

pytestmark = pytest.mark.gpu
X = np.longdouble
EPS = 2.0 ** -52


def interp(u, size, r):
    """u [3, nx, ny, nz] at r [3, n], and the largest |u| of each point's stencil."""
    idx, w = [], []
    for d in range(3):
        x0 = np.ceil(r[d] - 2)
        node = x0 + np.arange(4)[:, None]
        x = np.abs(r[d].astype(X) - node.astype(X))
        inner = (3 - 2 * x + np.sqrt(np.maximum(1 + 4 * x - 4 * x * x, 0))) / 8
        outer = (5 - 2 * x - np.sqrt(np.maximum(-7 + 12 * x - 4 * x * x, 0))) / 8
        w.append(np.where(x < 1, inner, np.where(x < 2, outer, 0)))
        idx.append(node.astype(np.int64) % size[d])
    v, top = np.zeros(r.shape, X), np.zeros(r.shape)
    for i in range(4):
        for j in range(4):
            for k in range(4):
                at = u[:, idx[0][i], idx[1][j], idx[2][k]]
                v += w[0][i] * w[1][j] * w[2][k] * at
                top = np.maximum(top, np.abs(at))
    return v, top


def field(rng, size, kind):
    u = 0.05 * rng.standard_normal((3,) + size)
    if kind == "rest":
        u[:] = 0.0
    if kind == "mixed":  # zeros, and neighbours that differ by up to 2^80
        u *= 2.0 ** -rng.integers(0, 80, u.shape)
        u[rng.random(u.shape) < 0.3] = 0.0
    if kind == "tiny":
        u *= 2.0 ** -1000
    if kind == "small":
        u[0] *= 1e-12
        u[2] *= 1e-200
    return u


# the weights are off by at most 2^-54 each (three of them, the others summing to
# one over their axis) and the 64 products and additions by half a last bit of
# partial sums below the largest velocity
TOL = (3 * 4 * 2.0 ** -54 + 70 * 2.0 ** -53)


@pytest.mark.parametrize("kind", ["plain", "rest", "mixed", "tiny", "small"])
# one point a block or many, and both block shapes
@pytest.mark.parametrize("size,n", [((8, 9, 33), 130), ((16, 5, 7), 64), ((1, 2, 3), 33),
                                    ((4, 1, 40), 1), ((12, 16, 40), 17001)])
@pytest.mark.parametrize("compat", [0, _lib.COMPAT_WIDE_INDEX, _lib.COMPAT_EXACT_F64])
def test_moves(kind, size, n, compat):
    rng = np.random.default_rng([n, len(kind)])
    lat = lb.Lattice(*size, 0.8, 0.8)
    lat.set_compat(_lib.COMPAT_INIT_SXZ | compat)
    u = field(rng, size, kind)
    lat.u[:] = u
    lat.u.H2D()
    box = np.array(size, dtype=np.float64)[:, None]
    r = rng.random((3, n)) * box
    r[:, 0] = 0.0
    if n > 3:
        r[:, 1] = np.nextafter(box[:, 0], 0)
        r[:, 2] = np.floor(r[:, 2])
        r[:, 3] = 1e-17
    tr = tracers.Array(n)
    tr.r[:] = r
    tr.H2D()
    tr.Move(lat)
    tr.D2H()
    v, top = interp(u, size, r)
    assert np.all(np.abs(tr.v.data - v) <= TOL * top)
    assert np.array_equal(tr.s.data, tr.v.data)
    assert np.array_equal(tr.r.data, np.mod((r + tr.v.data) + box, box))

    cp = swimmers.CommonParams()
    cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = 1e-3, 0.4, 0.0, 2.0, 5
    sw = swimmers.Array(n, cp)
    nv = rng.standard_normal((3, n))
    nv /= np.linalg.norm(nv, axis=0)
    sw.r[:] = r
    sw.n[:] = nv
    sw.H2D()
    sw.Move(lat)
    sw.D2H()
    want = 2e-3 * nv.astype(X) + v
    assert np.all(np.abs(sw.v.data - want) <= TOL * top + 2 * EPS * np.abs(want) + EPS * 2e-3)
    assert np.array_equal(sw.r.data, np.mod((r + sw.v.data) + box, box))
    vr, topr = interp(u, size, r - nv * 0.4)
    turned = nv + (v - vr) / X(0.4)
    want = turned / np.sqrt((turned * turned).sum(0))
    # the turn's error, and a last bit or so each for the sum, the norm and the division
    tol = 2 * TOL * (top + topr).max(0) / 0.4 + 8 * EPS
    assert np.all(np.abs(sw.n.data - want) <= tol)
    assert lat.status() == 0
