"""FP64 force spreading of swimmers in a cluster: force tiles with more ends than a bucket
holds take their own ends and no others."""
import numpy as np
import pytest

import oracle as O
from gpu_harness import build_gpu, snapshot
from lbswim import _lib, lb, swimmers
from test_gpu_force_elements import spread_with_bound

pytestmark = pytest.mark.gpu


def place(rng, size, n, box, centre):
    r = np.array(centre)[:, None] + np.array(box)[:, None] * (rng.random((3, n)) - 0.5)
    return np.mod(r, np.array(size, float)[:, None])


CASES = [
    # a few past the bucket, several rounds of the chains, both block sizes
    ((16, 16, 64), 140, (1.0, 1.0, 1.0), (8.0, 8.0, 32.0)),
    ((32, 32, 64), 600, (4.0, 6.0, 20.0), (8.0, 8.0, 32.0)),
    ((64, 64, 96), 2500, (6.0, 6.0, 20.0), (0.0, 0.0, 0.0)),   # around the corner
    ((65, 41, 97), 1500, (3.0, 3.0, 3.0), (64.5, 0.0, 96.0)),  # partial last tiles
    ((400, 1, 1), 700, (9.0, 1.0, 1.0), (77.0, 0.5, 0.5)),     # 16 nodes on a site
    ((300, 2, 3), 400, (20.0, 2.0, 3.0), (299.0, 1.0, 1.0))]


@pytest.mark.parametrize("size,n,box,centre", CASES)
def test_clustered_force(size, n, box, centre):
    rng = np.random.default_rng([n, size[0]])
    lat = lb.Lattice(*size, 0.8, 0.8)
    sw, r, nv = array(rng, size, n, box, centre)
    few, r2, nv2 = array(rng, size, 200, size, centre)
    for _ in range(2):  # the chains' heads are left from the first time
        lat.ZeroForce()
        few.AddForces(lat)
        sw.AddForces(lat)
    lat.force.D2H()
    force, tol = spread_with_bound(size, [(r - nv * 0.3, -1e-3 * nv), (r, 1e-3 * nv)])
    f2, t2 = spread_with_bound(size, [(r2 - nv2 * 0.3, -1e-3 * nv2), (r2, 1e-3 * nv2)])
    got = lat.force.data.reshape(3, -1)
    # the two arrays' forces are added in FP64
    assert np.all(np.abs(got - (force + f2)) <= tol + t2 + 2.0 ** -53 * np.abs(got))


def array(rng, size, n, box, centre):
    cp = swimmers.CommonParams()
    cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = 1e-3, 0.3, 0.0, 1.0, 1
    sw = swimmers.Array(n, cp)
    r = place(rng, size, n, box, centre)
    nv = rng.standard_normal((3, n))
    nv /= np.linalg.norm(nv, axis=0)
    sw.r[:] = r
    sw.n[:] = nv
    sw.H2D()
    return sw, r, sw.n.data.copy()


@pytest.mark.parametrize("size,n,box,centre", CASES[:3])
def test_clustered_exact(size, n, box, centre):
    """Exact mode adds a tile's ends in end order, the oracle's bits."""
    case = O.random_case(size, n, 10, seed=4, u_amp=0.01, alpha=0.0)
    case["swimmers"]["r"] = place(np.random.default_rng(n), size, n, box, centre)
    orc = O.make_system(case)
    lat, sw, tr, system = build_gpu(case, "f64",
                                    compat=_lib.COMPAT_INIT_SXZ | _lib.COMPAT_EXACT_F64)
    for _ in range(2):
        orc.step(1)
        system.Step(1)
        o, g = orc.snapshot(), snapshot(lat, sw, tr)
        assert all(np.array_equal(g[k], o[k]) for k in ("force", "f", "sw_r"))


def test_not_a_number_in_a_cluster():
    """One swimmer whose orientation is not a number among a full tile's: NaN where its
    stencils reach, the others' forces elsewhere."""
    torch = pytest.importorskip("torch")
    from test_gpu_device_writes import device_field
    size, n = (32, 32, 64), 500
    rng = np.random.default_rng(3)
    lat = lb.Lattice(*size, 0.8, 0.8)
    sw, r, nv = array(rng, size, n, (4.0, 6.0, 20.0), (8.0, 8.0, 32.0))
    device_field(sw, 2)[:, 7] = float("nan")
    torch.cuda.synchronize()
    lat.ZeroForce()
    sw.AddForces(lat)
    lat.force.D2H()
    got = lat.force.data.reshape(3, -1)
    keep = np.arange(n) != 7
    r, nv = r[:, keep], nv[:, keep]
    force, tol = spread_with_bound(size, [(r - nv * 0.3, -1e-3 * nv), (r, 1e-3 * nv)])
    # FP64 in end order there: a last bit of the sum for each of up to 1000 ends
    ok = np.abs(got - force) <= tol + 1000 * 2.0 ** -53 * 1e-3
    bad = np.isnan(got)
    assert np.all(ok | bad) and 64 <= bad[0].sum() <= 128
