"""Exact FP64 mode on states where leaving out a zero, or a sign, could show: zeros
of both signs, subnormals, infinities and NaN, bit for bit against the reference's
dense loops in numpy (each operation rounded on its own)."""
import numpy as np
import pytest

from lbswim import _lib, lb

pytestmark = pytest.mark.gpu


def dense_step(P, f, F):
    """lb.cu:72-218 on f [15, n], F [3, n], before streaming; and rho, u."""
    mode = np.zeros((15, f.shape[1]))
    for m in range(15):
        for p in range(15):
            mode[m] = mode[m] + f[p] * P.mm[m][p]
    rho, u = mode[0].copy(), np.empty_like(F)
    usq, uF = np.zeros(f.shape[1]), np.zeros(f.shape[1])
    ws, wb = 1.0 / (P.tau_s + 0.5), 1.0 / (P.tau_b + 0.5)
    for a in range(3):
        u[a] = (mode[1 + a] + 0.5 * F[a]) / mode[0]
        mode[1 + a] = mode[1 + a] + F[a]
        usq = usq + u[a] * u[a]
        uF = uF + u[a] * F[a]
    at = [[4, 5, 6], [5, 7, 8], [6, 8, 9]]
    S = [[mode[at[a][b]].copy() for b in range(3)] for a in range(3)]
    tr = np.zeros(f.shape[1])
    for a in range(3):
        tr = tr + S[a][a]
    for a in range(3):
        S[a][a] = S[a][a] - tr / 3.0
    tr = tr - wb * (tr - mode[0] * usq)
    tr = tr + ((2.0 * wb) * P.tau_b) * uF
    for a in range(3):
        for b in range(3):
            d = 1.0 if a == b else 0.0
            S[a][b] = S[a][b] - ws * (S[a][b] - mode[0] * (u[a] * u[b] - usq * d))
            S[a][b] = S[a][b] + ((2.0 * ws) * P.tau_s) * (
                (u[a] * F[b] + F[a] * u[b]) - (2.0 * uF) * d)
        S[a][a] = S[a][a] + tr / 3.0
    for m, (a, b) in zip(range(4, 10), ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))):
        mode[m] = S[a][b]
    mode[10:] = 0.0
    out = np.zeros_like(f)
    for p in range(15):
        for m in range(15):
            out[p] = out[p] + mode[m] * P.mmi[p][m]
    return out, rho, u


@pytest.mark.parametrize("size", [(3, 5, 33), (1, 2, 3)])
@pytest.mark.parametrize("forced", [False, True])
def test_odd_values_keep_the_reference_bits(size, forced):
    n = size[0] * size[1] * size[2]
    rng = np.random.default_rng(n)
    f = rng.random((15, n)) * 0.1 + 0.01
    odd = rng.integers(0, 15, n)
    values = np.array([0.0, -0.0, -0.01, 5e-324, 1e-310, 1e300, np.inf, -np.inf, np.nan])
    pick = rng.integers(0, len(values) + 6, n)
    for s in range(n):
        if pick[s] < len(values):
            f[odd[s], s] = values[pick[s]]
    f[:, 0] = -0.0  # nothing but zeros
    F = 1e-3 * rng.standard_normal((3, n)) if forced else np.zeros((3, n))
    lat = lb.Lattice(*size, 0.8, 1.1)
    lat.set_compat(_lib.COMPAT_INIT_SXZ | _lib.COMPAT_EXACT_F64)
    lat.fOld[:] = f.reshape((15,) + size)
    lat.fOld.H2D()
    lat.ZeroForce()
    if forced:
        lat.force[:] = F.reshape((3,) + size)
        lat.force.H2D()
    with np.errstate(all="ignore"):
        out, rho, u = dense_step(lat.params.impl, f, F)
    lat.CalcHydro()
    lat.rho.D2H()
    lat.u.D2H()
    np.testing.assert_array_equal(lat.rho.data.reshape(-1), rho)
    np.testing.assert_array_equal(lat.u.data.reshape(3, n), u)
    lat.Step()
    lat.fOld.D2H()
    want = np.empty((15,) + size)
    for p in range(15):
        c = [int(v) for v in lat.params.impl.ci[p]]
        want[p] = np.roll(out[p].reshape(size), shift=c, axis=(0, 1, 2))
    got = lat.fOld.data
    np.testing.assert_array_equal(got, want)
    finite = np.isfinite(want)
    assert np.array_equal(np.signbit(got[finite]), np.signbit(want[finite]))
