"""FP64 Step and CalcHydro at the edges of their integer arithmetic: sites that
fit it, sites that do not (and take FP64), mixed within warps, against the
collision in extended precision."""
import numpy as np
import pytest

from lbswim import _lib, lb

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52
C = np.array([[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1],
              [1, 1, 1], [1, 1, -1], [1, -1, 1], [1, -1, -1], [-1, 1, 1], [-1, 1, -1],
              [-1, -1, 1], [-1, -1, -1]])
X = np.longdouble
W = np.array([X(2) / 9] + [X(1) / 9] * 6 + [X(1) / 72] * 8)


def moments(f, F):
    rho = f.sum(0)
    j = np.tensordot(C.T.astype(X), f, 1)
    return rho, j, (j + F / 2) / rho


def collide(f, F, ts, tb):
    """lb.cu:121-203 in extended precision, f [15, n], F [3, n]."""
    rho, j, u = moments(f, F)
    usq, uF = (u * u).sum(0), (u * F).sum(0)
    ws, wb = 1 / (X(ts) + X(0.5)), 1 / (X(tb) + X(0.5))
    Q = [[C[:, a] * C[:, b] - X(a == b) / 3 for b in range(3)] for a in range(3)]
    S = [[np.tensordot(Q[a][b], f, 1) for b in range(3)] for a in range(3)]
    tr = S[0][0] + S[1][1] + S[2][2]
    new = tr - wb * (tr - rho * usq) + 2 * wb * tb * uF
    out = rho + 3 * np.tensordot(C.astype(X), j + F, 1)
    for a in range(3):
        for b in range(3):
            d = X(a == b)
            s = S[a][b] - d * tr / 3
            s = s - ws * (s - rho * (u[a] * u[b] - usq * d))
            s = s + 2 * ws * ts * (u[a] * F[b] + F[a] * u[b] - 2 * uF * d) + d * new / 3
            out = out + X(4.5) * Q[a][b][:, None] * s
    return W[:, None] * out


def state(rng, n, kind):
    """f [15, n] and F [3, n] near an equilibrium, every 7th site unlike it as `kind` says."""
    rho = 0.5 + rng.random(n)
    u = 0.1 * rng.uniform(-1, 1, (3, n))
    F = 1e-3 * rng.uniform(-1, 1, (3, n))
    odd = np.arange(n) % 7 == 3
    if kind == "fast":
        u[:, odd] = 0.45 * rng.choice([-1, 1], (3, odd.sum()))
    if kind == "force":
        F[:, odd] = rng.uniform(-0.1, 0.1, (3, odd.sum()))
        F[:, np.arange(n) % 7 == 5] = 1e-30
    if kind == "scales":
        rho *= 2.0 ** rng.integers(-900, 900, n)
        F *= rho
    cu = np.tensordot(C, u, 1)
    f = W[:, None].astype(float) * rho * (1 + 3 * cu + 4.5 * cu ** 2 - 1.5 * (u * u).sum(0))
    f *= 1 + 1e-2 * rng.uniform(-1, 1, f.shape)
    if kind == "populations":
        p = rng.integers(0, 15, odd.sum())
        f[p, np.nonzero(odd)[0]] *= rng.choice([0.0, -1.0, 1e-3, 5.0, 2.0 ** -7], odd.sum())
    return f, F


@pytest.mark.parametrize("size", [(3, 5, 33), (4, 1, 1), (2, 43, 3), (9, 16, 8)])
@pytest.mark.parametrize("taus", [(0.8, 0.8), (0.01, 1.9), (1e7, 0.6), (0.0, 0.3)])
@pytest.mark.parametrize("kind", ["plain", "fast", "force", "scales", "populations"])
@pytest.mark.parametrize("forced", [True, False])
def test_step_and_calc_hydro(size, taus, kind, forced):
    n = size[0] * size[1] * size[2]
    f, F = state(np.random.default_rng([n, len(kind)]), n, kind)
    lat = lb.Lattice(*size, *taus)
    lat.fOld[:] = f.reshape((15,) + size)
    lat.fOld.H2D()
    lat.ZeroForce()
    if forced:
        lat.force[:] = F.reshape((3,) + size)
        lat.force.H2D()
    else:
        F = 0 * F
    fx, Fx = f.astype(X), F.astype(X)

    # 15 terms a moment: its error is at most 15 EPS / 2 of the sum of their
    # magnitudes; a population takes at most 1.2 of each moment, twice for the
    # relaxation, so 32 EPS of the sum hold it, and 16 EPS the density and momentum
    scale = np.abs(f).sum(0) + 3 * np.abs(F).sum(0)
    lat.CalcHydro()
    lat.rho.D2H()
    lat.u.D2H()
    rho, _, u = moments(fx, Fx)
    assert np.all(np.abs(lat.rho.data.reshape(-1) - rho) <= 16 * EPS * scale)
    tol = (16 * EPS * scale + 16 * EPS * scale * np.abs(u)) / np.abs(rho)
    assert np.all(np.abs(lat.u.data.reshape(3, -1) - u) <= tol)

    lat.Step()
    lat.fOld.D2H()
    got = lat.fOld.data
    want = collide(fx, Fx, *taus).reshape((15,) + size)
    # products of velocities: their errors scale with rho u^2
    usq = 1 + (u * u).sum(0).astype(float)
    tol = (32 * EPS * scale * usq).reshape(size)
    for p in range(15):
        back = np.roll(got[p], shift=tuple(-C[p]), axis=(0, 1, 2))
        assert np.all(np.abs(back - want[p]) <= tol), p


def test_momentum_of_every_magnitude():
    # u = j / rho from a momentum of 1 to 2^50 last bits of an axis population
    n = 1 + 2 * 51 * 5
    lat = lb.Lattice(1, 1, n, 0.7, 0.7)
    f = np.repeat(W.astype(float)[:, None], n, 1)
    ulp = 2.0 ** -56  # of 1/9
    for m in range(51):
        for i, q in enumerate((1, 3, 5, 7, 2)):
            s = 1 + 2 * (5 * m + i)
            f[1 + 2 * (i % 3), s] += q * 2.0 ** m * ulp / 8
            f[1 + 2 * (i % 3), s + 1] -= q * 2.0 ** m * ulp / 8
    lat.fOld[:] = f.reshape(15, 1, 1, n)
    lat.fOld.H2D()
    lat.ZeroForce()
    lat.CalcHydro()
    lat.u.D2H()
    _, _, u = moments(f.astype(X), np.zeros((3, n), X))
    # the momentum is exact: two roundings are left, and the reciprocal's
    got = lat.u.data.reshape(3, n)
    assert np.all(np.abs(got - u) <= 2 * EPS * np.abs(u))


def test_rest_keeps_small_forces_and_nonfinite_sites_stay_local():
    size = (4, 6, 40)
    lat = lb.Lattice(*size, 0.7, 0.7)
    lat.fOld[:] = W.astype(float)[:, None, None, None]
    lat.fOld.H2D()
    lat.force[:] = 1e-25
    lat.force.H2D()
    lat.CalcHydro()
    lat.u.D2H()
    assert np.all(np.abs(lat.u.data - 0.5e-25) <= 4 * EPS * 0.5e-25)
    assert lat.status() == 0
    lat.fOld.data[3, 1, 2, 3] = np.nan
    lat.fOld.H2D()
    lat.Step()
    lat.CalcHydro()
    lat.rho.D2H()
    bad = np.argwhere(~np.isfinite(lat.rho.data[0]))
    near = {tuple((np.array([1, 2, 3]) + c) % size) for c in C}
    assert {tuple(b) for b in bad} == near
    assert lat.status(clear=True) == _lib.STATUS_NONFINITE
