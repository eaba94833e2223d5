"""FP64 force spreading element by element: small forces beside large ones, axes that
the swimmers hardly point along, and the far corners of stencils keep their digits."""
import numpy as np
import pytest

from lbswim import lb, swimmers
from test_gpu_force_f64 import X, weights

pytestmark = pytest.mark.gpu


def spread_with_bound(size, ends):
    """The force, and what FP64 arithmetic may be off by, for ends (r, F) in order: a weight
    is off by at most 2^-53 (its distance is one rounding off, and it is formed from terms of
    order one), products and sums by a last bit each; and 2^-72 of the component's largest
    force a contribution, for sums in a unit that all sites of a tile share."""
    N = size[0] * size[1] * size[2]
    force, tol, mag = np.zeros((3, N), X), np.zeros((3, N)), np.zeros((3, N))
    for r, F in ends:
        idx, w = zip(*[weights(r[d]) for d in range(3)])
        for i in range(4):
            for j in range(4):
                for k in range(4):
                    s = np.ravel_multi_index([idx[0][i] % size[0], idx[1][j] % size[1],
                                              idx[2][k] % size[2]], size)
                    a, b, c = w[0][i], w[1][j], w[2][k]
                    for d in range(3):
                        np.add.at(force[d], s, a * b * c * F[d])
                        np.add.at(mag[d], s, np.abs(a * b * c * F[d]).astype(float))
                        np.add.at(tol[d], s, (np.abs(F[d]) * (a * b + b * c + a * c)
                                              ).astype(float) * 2.0 ** -53 +
                                  2.0 ** -72 * np.abs(F[d]).max())
    return force, tol + mag * 2.0 ** -50 + 1e-320


# direct ends, buckets, more than a chunk and than eight chunks of ends in a tile, folded
# stencils
@pytest.mark.parametrize("size,n,box", [((9, 17, 65), 1, 1.0), ((9, 17, 65), 30, 1.0),
                                        ((16, 16, 40), 300, 1.0), ((8, 16, 64), 100, 0.1),
                                        ((3, 2, 40), 9, 1.0), ((1, 5, 70), 60, 1.0),
                                        ((75, 60, 50), 2000, 1.0), ((77, 60, 50), 2000, 1.0)])
@pytest.mark.parametrize("kind", ["aligned", "mixed", "corner"])
def test_every_element(size, n, box, kind):
    rng = np.random.default_rng([n, len(kind), size[0]])
    r = rng.random((3, n)) * (box * np.array(size)[:, None])
    nv = rng.standard_normal((3, n))
    nv /= np.linalg.norm(nv, axis=0)
    if kind == "aligned":  # along x, but for a little
        nv = np.array([[1.0], [1e-9], [1e-13]]) * (1 + 0.1 * nv)
    if kind == "mixed":    # forces of every size
        nv *= 2.0 ** -rng.integers(0, 12, n)
    if kind == "corner":   # stencils that just reach their last nodes
        r = np.floor(r) + 2.0 ** -rng.integers(4, 9, (3, n))
    lat = lb.Lattice(*size, 0.8, 0.8)
    cp = swimmers.CommonParams()
    cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = 1e-3, 0.3, 0.0, 1.0, 1
    sw = swimmers.Array(n, cp)
    sw.r[:] = r
    sw.n[:] = nv
    sw.H2D()
    lat.ZeroForce()
    sw.AddForces(lat)
    lat.force.D2H()
    nv = sw.n.data
    force, tol = spread_with_bound(size, [(r - nv * 0.3, -1e-3 * nv), (r, 1e-3 * nv)])
    got = lat.force.data.reshape(3, -1)
    assert np.all(np.abs(got - force) <= tol)
