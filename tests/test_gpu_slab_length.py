"""The step's slab length (x planes per slab) follows the lattice and the number
of pending ends; the results do not depend on it: the two slab shapes, several
arrays, and batched members give the same bits."""
import numpy as np
import pytest

from lbswim import lb, swimmers
from lbswim.ensemble import Ensemble
from lbswim.System import System

pytestmark = pytest.mark.gpu


def build(size, counts, tile, precision="f32"):
    lat = lb.Lattice(*size, 0.7, 0.9, precision=precision)
    lat.tile = tile
    lat.init_random(11)
    system, arrays = System(lat), []
    for i, n in enumerate(counts):
        cp = swimmers.CommonParams()
        cp.P, cp.l, cp.alpha, cp.mobility, cp.seed = 1e-3 * (i + 1), 0.5, 0.1, 1.0, 3 + i
        sw = swimmers.Array(n, cp)
        sw.init_random(lat, 21 + i)
        system.AddThing(sw)
        arrays.append(sw)
    return lat, system, arrays


def state(lat, arrays):
    out = []
    for f in (lat.u, lat.rho, lat.fOld):
        f.D2H()
        out.append(f.data.copy())
    for sw in arrays:
        sw.D2H()
        out += [sw.r.data.copy(), sw.n.data.copy()]
    return out


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


# lengths from one plane to the longest (60), even and uneven last slabs, slabs
# whose ends do not fit shared memory, axes shorter than a stencil
@pytest.mark.parametrize("size", [(1, 9, 33), (3, 8, 32), (24, 24, 24), (61, 17, 40),
                                  (130, 40, 33), (250, 8, 16)])
@pytest.mark.parametrize("density", [1 / 500, 1 / 20])
@pytest.mark.parametrize("precision", ["f32", "bf16"])
def test_slab_shapes_give_the_same_bits(size, density, precision):
    n = max(1, int(size[0] * size[1] * size[2] * density))
    got = []
    for tile in (0, 1):
        lat, system, arrays = build(size, (n, 1), tile, precision)
        system.Step(3)
        lat.force.D2H()
        got.append(state(lat, arrays) + [lat.force.data.copy()])
    assert same(*got)
    # the slab shape changes between AddForces and Step: the ends are listed again
    lat, system, arrays = build(size, (n, 1), 0, precision)
    system.Step(2)
    lat.ZeroForce()
    for sw in arrays:
        sw.AddForces(lat)
    lat.tile = 1
    lat.Step()
    lat.CalcHydro()
    for sw in arrays:
        sw.Move(lat)
    assert same(state(lat, arrays), got[0])


@pytest.mark.parametrize("members", [1, 3, 40])
def test_batched_members_give_the_same_bits(members):
    sizes = [(24, 16, 40), (70, 9, 33), (16, 16, 16)]
    batch = [build(sizes[m % 3], (5 + 40 * (m % 3),), m % 2) for m in range(members)]
    ens = Ensemble([(lat, arrays[0], None) for lat, _, arrays in batch])
    ens.Step(2)
    ens.Step(3)
    for m in range(min(members, 6)):
        lat, _, arrays = batch[m]
        lat.force.D2H()
        force = lat.force.data.copy()
        alone, system, arrays1 = build(sizes[m % 3], (5 + 40 * (m % 3),), m % 2)
        system.Step(5)
        alone.force.D2H()
        assert np.array_equal(force, alone.force.data)
        assert same(state(lat, arrays), state(alone, arrays1))
        system.Step()  # a member goes on alone
        System.Step(_with(lat, arrays))
        assert same(state(lat, arrays), state(alone, arrays1))


def _with(lat, arrays):
    system = System(lat)
    for sw in arrays:
        system.AddThing(sw)
    return system


def test_priority_stream_gives_the_same_bits():
    """Tracers at a lower priority than the lattice's stream: slabs of another length
    (13 planes in place of 26)."""
    torch = pytest.importorskip("torch")
    from lbswim import tracers
    got = []
    for priority in (0, -5):
        for n in (15578, 1):
            lat, system, arrays = build((52, 271, 283), (n,), 0)
            stream = torch.cuda.Stream(priority=priority)
            lat.set_stream(stream.cuda_stream)
            tr = tracers.Array(500)
            tr.init_random(lat, 5)
            system.AddThing(tr)
            system.Step(4)
            lat.join()
            tr.D2H()
            got.append(state(lat, arrays) + [tr.r.data.copy()])
            del system, tr, arrays, lat
    assert same(got[0], got[2]) and same(got[1], got[3])
