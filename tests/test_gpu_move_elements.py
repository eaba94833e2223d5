"""FP64 interpolation point by point: where the largest velocity of a stencil has hardly
any weight, the small ones that make the result keep their digits."""
import numpy as np
import pytest

from lbswim import _lib, lb, swimmers, tracers
from test_gpu_force_f64 import X, weights

pytestmark = pytest.mark.gpu


def interp(u, size, r):
    """u [3, nx, ny, nz] at r [3, n], and what FP64 arithmetic may be off by: a weight by 2^-53
    (its distance is one rounding off, and it is formed from terms of order one), the 64
    products and sums by a last bit of the sum of the terms' sizes each."""
    idx, w = zip(*[weights(r[d]) for d in range(3)])
    v, tol = np.zeros(r.shape, X), np.zeros(r.shape)
    for i in range(4):
        for j in range(4):
            for k in range(4):
                at = u[:, idx[0][i] % size[0], idx[1][j] % size[1], idx[2][k] % size[2]]
                a, b, c = w[0][i], w[1][j], w[2][k]
                v += a * b * c * at
                tol += (np.abs(at) * ((a * b + b * c + a * c) * 2.0 ** -53 +
                                      a * b * c * 70 * 2.0 ** -53)).astype(float)
    return v, tol


@pytest.mark.parametrize("kind", ["spikes", "decay", "smooth", "steps"])
@pytest.mark.parametrize("n", [1, 500, 17001])
@pytest.mark.parametrize("compat", [0, _lib.COMPAT_WIDE_INDEX])
def test_every_velocity(kind, n, compat):
    size = (12, 16, 40)
    rng = np.random.default_rng([n, len(kind)])
    u = 0.05 * rng.standard_normal((3,) + size)
    if kind == "spikes":   # a node here and there, the others at rest or nearly
        u *= np.where(rng.random(u.shape) < 0.03, 1.0, 0.0)
        u[2] += 1e-13 * rng.standard_normal(size)
    if kind == "decay":    # a factor of up to 2^8 from node to node
        d = np.stack(np.meshgrid(*[np.arange(s) for s in size], indexing="ij")).sum(0)
        u *= 2.0 ** -(8.0 * np.minimum(d, 68 - d))
    if kind == "smooth":
        x = np.stack(np.meshgrid(*[np.arange(s) * 2 * np.pi / s for s in size], indexing="ij"))
        u = 0.05 * np.stack([np.sin(x[1]), np.sin(x[2] + 0.3), np.cos(x[0]) * np.sin(x[1])])
    if kind == "steps":
        u *= 2.0 ** -rng.integers(0, 30, u.shape)
    lat = lb.Lattice(*size, 0.8, 0.8)
    lat.set_compat(_lib.COMPAT_INIT_SXZ | compat)
    lat.u[:] = u
    lat.u.H2D()
    box = np.array(size, dtype=np.float64)[:, None]
    r = rng.random((3, n)) * box
    r[:, ::2] = np.floor(r[:, ::2]) + 2.0 ** -rng.integers(1, 12, r[:, ::2].shape)
    tr = tracers.Array(n)
    tr.r[:] = r
    tr.H2D()
    tr.Move(lat)
    tr.D2H()
    v, tol = interp(u, size, r)
    assert np.all(np.abs(tr.v.data - v) <= tol)
    cp = swimmers.CommonParams()
    cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = 0.0, 0.4, 0.0, 0.0, 5  # swept along only
    sw = swimmers.Array(n, cp)
    sw.r[:] = r
    sw.n[:] = np.array([[0.6], [0.0], [0.8]])
    sw.H2D()
    sw.Move(lat)
    sw.D2H()
    assert np.all(np.abs(sw.v.data - v) <= tol)
