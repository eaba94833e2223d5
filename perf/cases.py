"""Performance cases of the coupled lattice-Boltzmann step.

Each case is work that a program using this package has it do, through the
public entry points: coupled runs with swimmers and tracers (one step and a
read-back at a time as in the README loop, or many steps in one call), runs of
the fluid alone under a body force, batched ensembles, and the upload /
initialise / checkpoint path.  The densities of the coupled cases are those of
the benchmark's 256^3 workload (one swimmer per 256 sites, one tracer per 16).

``listed()`` gives the fixed cases and ``draw(rng)`` more of the same ranges;
``prepare`` builds a case's objects from a seed, ``run`` does one pass and
returns what it computed, ``work`` counts the bytes and operations a pass cannot
do without, and ``exact`` computes the same pass in 64 bits with plain torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir,
                                "gpu-swimmers_gb300"))
from lbswim import _lib, lb, swimmers, tracers  # noqa: E402
from lbswim.System import System  # noqa: E402
from lbswim.ensemble import Ensemble  # noqa: E402

F_BYTES = {"f64": 8, "f32": 4, "bf16": 2, "f16": 2}
MEMBER_SHAPES = ((16, 16, 16), (24, 24, 24), (32, 32, 32), (48, 48, 48), (64, 64, 64),
                 (32, 32, 64), (48, 48, 96))


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def coupled(size, precision, steps, nsw, ntr, arrays=1, readback=False, bits=False, tau=0.8,
            alpha=0.01, history=True, noise=1e-3, grid=False):
    """A coupled run.  readback: steps one at a time with the swimmers read back
    after each; bits: FP64 in the reference's operation order; history: the
    tracers' displacements and velocities are read back beside their positions;
    grid: tracers at the integer grid points; arrays: swimmer arrays, each with
    its own parameters."""
    return {"path": "coupled", "nx": size[0], "ny": size[1], "nz": size[2],
            "precision": precision, "steps": steps, "swimmers": nsw, "tracers": ntr,
            "arrays": arrays, "readback": readback, "bits": bits, "tau": tau, "alpha": alpha,
            "history": history, "noise": noise, "grid": grid}


def fluid(size, precision, steps, tau):
    return {"path": "fluid", "nx": size[0], "ny": size[1], "nz": size[2], "precision": precision,
            "steps": steps, "tau": tau}


def listed():
    return [
        # the README program: one swimmer, 4096 tracers, Step() then D2H() each step
        dict(coupled((16, 16, 16), "f64", 10, 1, 4096, readback=True, tau=0.25, noise=0.0,
                     grid=True), name="readme_f64"),
        # a small suspension in reduced precision, watched step by step
        dict(coupled((24, 24, 24), "f32", 20, 54, 864, readback=True), name="small_f32"),
        # an odd-sized box in the default precision
        dict(coupled((65, 47, 90), "f64", 10, 1074, 17184, alpha=0.05), name="ragged_f64"),
        # an odd-sized box in FP32
        dict(coupled((100, 75, 130), "f32", 20, 3809, 60938), name="ragged_f32"),
        # the benchmark's suspension in FP64 (the reference's precision, the default)
        dict(coupled((256, 256, 256), "f64", 4, 65536, 1048576), name="bulk_f64"),
        # ... and in FP32
        dict(coupled((256, 256, 256), "f32", 20, 65536, 1048576, history=False),
             name="bulk_f32"),
        # the precision study's form: 16-bit storage, swimmers in arrays of their own parameters
        dict(coupled((192, 200, 208), "bf16", 10, 31200, 124800, arrays=4), name="arrays_bf16"),
        # reproducing the reference bit for bit
        dict(coupled((64, 64, 64), "f64", 5, 1024, 16384, bits=True), name="bits_f64"),
        # a driven flow without particles, the library's calls one by one
        dict(fluid((160, 192, 176), "f64", 5, 0.6), name="fluid_f64"),
        dict(fluid((200, 256, 224), "f32", 10, 0.7), name="fluid_f32"),
        # a sweep of independent small solves advanced together
        {"name": "ensemble_f32", "path": "ensemble", "members": 96, "steps": 100},
        # a new initial state and a checkpoint of it
        {"name": "restart_f32", "path": "restart", "nx": 128, "ny": 144, "nz": 160,
         "precision": "f32", "tau": 0.8},
    ]


def _size(rng, lo, hi):
    """An axis length, spread over the logarithm of the range; odd ones as likely as not."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("coupled", "coupled", "coupled", "coupled", "fluid", "fluid", "ensemble",
                       "restart"))
    if kind == "ensemble":
        return {"path": "ensemble", "members": rng.randint(8, 96), "steps": rng.randint(40, 100)}
    side = _size(rng, 12, 224)
    size = tuple(max(8, min(240, int(round(side * rng.uniform(0.7, 1.4))))) for _ in range(3))
    sites = size[0] * size[1] * size[2]
    precision = rng.choice(("f64", "f64", "f32", "f32", "bf16", "f16"))
    tau = round(rng.uniform(0.5, 1.5), 3)
    if kind == "fluid":
        return fluid(size, precision, rng.randint(3, 5 if precision == "f64" else 10), tau)
    if kind == "restart":
        return {"path": "restart", "nx": min(160, size[0]), "ny": min(160, size[1]),
                "nz": min(160, size[2]), "precision": precision, "tau": tau}
    density = math.exp(rng.uniform(math.log(1 / 512), math.log(1 / 128)))
    nsw = max(1, int(sites * density))
    ntr = max(1, int(sites * math.exp(rng.uniform(math.log(1 / 64), math.log(1 / 8)))))
    bits = precision == "f64" and sites < 400000 and rng.random() < 0.25
    arrays = rng.choice((1, 1, 1, 3)) if nsw >= 64 else 1
    return coupled(size, precision, rng.randint(2, 4 if sites > 2000000 else 10), nsw, ntr,
                   arrays=arrays, readback=rng.random() < 0.4, bits=bits, tau=tau,
                   alpha=round(rng.uniform(0.0, 0.05), 4), history=ntr < 200000)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _shape(case):
    return (case["nx"], case["ny"], case["nz"])


def _swimmer_groups(case, seed):
    """One dict per swimmer array: its parameters, positions and orientations."""
    rng = np.random.default_rng([seed, 1])
    L = np.array(_shape(case), dtype=np.float64).reshape(3, 1)
    groups = []
    for k in range(case["arrays"]):
        n = case["swimmers"] * (k + 1) // case["arrays"] - case["swimmers"] * k // case["arrays"]
        nv = rng.standard_normal((3, n))
        nv /= np.linalg.norm(nv, axis=0, keepdims=True)
        one = case["arrays"] == 1
        a, hydro = 0.1, 1.5
        groups.append({
            "n": n, "r": rng.random((3, n)) * L, "nvec": nv,
            "P": 1e-3 if one else float(rng.uniform(5e-4, 2e-3)),
            "alpha": case["alpha"] if one else float(rng.uniform(0.0, 0.05)),
            "l": 0.1 if case["grid"] else 0.5,
            "mobility": (1 / a - 1 / hydro) / (6 * math.pi * case["tau"] / 3),
            "seed": int(rng.integers(1, 2 ** 31))})
    return groups


def _tracer_positions(case, seed):
    n, size = case["tracers"], _shape(case)
    if case["grid"]:  # the integer grid points, from a corner that the seed picks
        i = (np.arange(n) + seed * 7) % (size[0] * size[1] * size[2])
        return np.stack(np.unravel_index(i, size)).astype(np.float64)
    return np.random.default_rng([seed, 2]).random((3, n)) * np.array(size).reshape(3, 1)


def _density(case, seed):
    size = _shape(case)
    if not case["noise"]:
        return np.ones(size)
    return 1.0 + case["noise"] * np.random.default_rng([seed, 3]).random(size)


def _flow(case, seed):
    """(rho, u, force) of the fluid cases: a Taylor-Green-like flow of random
    phases and amplitudes with density noise, and a sinusoidal body force."""
    rng = np.random.default_rng([seed, 4])
    size = _shape(case)
    ax = [np.arange(n) * (2 * np.pi / n) for n in size]
    ph = rng.uniform(0, 2 * np.pi, (3, 3))
    amp = rng.uniform(0.01, 0.03, 3)
    u = np.empty((3,) + size)
    force = np.empty((3,) + size)
    for c in range(3):
        x, y, z = ax[0] + ph[c, 0], ax[1] + ph[c, 1], ax[2] + ph[c, 2]
        u[c] = amp[c] * (np.cos(x)[:, None, None] * np.sin(y)[None, :, None]
                         * np.sin(z)[None, None, :])
        force[c] = 1e-5 * (c + 1) * np.sin(ax[(c + 1) % 3] + ph[c, 0]).reshape(
            [-1 if d == (c + 1) % 3 else 1 for d in range(3)])
    rho = 1.0 + 1e-3 * rng.random(size)
    return rho, u, force


def _member_specs(case, seed):
    """Members of a batched ensemble, sizes and parameters drawn as in the
    benchmark's ensemble."""
    rng = np.random.default_rng([seed, 5])
    # the shapes come from the case alone, so that every seed is the same work
    shapes = np.random.default_rng(case["members"])
    specs = []
    for m in range(case["members"]):
        size = MEMBER_SHAPES[shapes.integers(len(MEMBER_SHAPES))]
        nsw = max(1, min(512, int(math.exp(shapes.uniform(0.0, math.log(512.0))))))
        ntr = int(shapes.integers(1, 4097))
        specs.append(dict(
            coupled(size, "f32", case["steps"], nsw, ntr, tau=float(shapes.uniform(0.6, 1.5)),
                    alpha=float(rng.uniform(0.0, 0.05))),
            P=float(rng.uniform(1e-4, 1e-3)), seed=int(rng.integers(1, 2 ** 31))))
    return specs


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
class _DeviceArray:
    """A device buffer of the lattice as torch sees it."""

    def __init__(self, ptr, shape, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr,
                                         "data": (ptr, False), "version": 3}


def _view(lat, field, shape, typestr):
    ptr, _ = lat.device_ptr(field)
    return torch.as_tensor(_DeviceArray(ptr, shape, typestr, lat), device="cuda")


def _hydro(lat):
    """rho and u on the device: [N] and [3, N] doubles of an FP64 lattice, packed
    {ux, uy, uz, rho - rho0} floats of the others."""
    n = lat.addr.n
    if lat.precision == "f64":
        return {"rho": _view(lat, _lib.FIELD_RHO, (n,), "<f8"),
                "u": _view(lat, _lib.FIELD_U, (3, n), "<f8")}
    h = _view(lat, _lib.FIELD_U, (n, 4), "<f4")
    return {"rho": h[:, 3], "u": h[:, :3]}


def _distributions(lat):
    """fOld on the device: [15, N] doubles, or the blocks [N / 32][15][32] of a
    reduced-precision lattice."""
    n = lat.addr.n
    if lat.precision == "f64":
        return _view(lat, _lib.FIELD_FOLD, (15, n), "<f8")
    shape = (-(-n // 32), 15, 32)
    if lat.precision == "f32":
        return _view(lat, _lib.FIELD_FOLD, shape, "<f4")
    kind = torch.bfloat16 if lat.precision == "bf16" else torch.float16
    return _view(lat, _lib.FIELD_FOLD, shape, "<i2").view(kind)


def _lattice(case, rho, u=None):
    lat = lb.Lattice(*_shape(case), case["tau"], case["tau"], precision=case["precision"])
    if case.get("bits"):
        lat.set_compat(_lib.COMPAT_INIT_SXZ | _lib.COMPAT_EXACT_F64)
    lat.rho[:] = rho
    lat.rho.H2D()
    if u is not None:
        lat.u[:] = u
    lat.u.H2D()
    lat.ZeroForce()
    return lat


def _coupled_system(case, seed, P=None):
    lat = _lattice(case, _density(case, seed))
    system = System(lat)
    arrays = []
    for g in _swimmer_groups(case, seed):
        cp = swimmers.CommonParams()
        cp.P, cp.l, cp.alpha, cp.mobility = P or g["P"], g["l"], g["alpha"], g["mobility"]
        cp.seed = g["seed"]
        sw = swimmers.Array(g["n"], cp)
        sw.r[:] = g["r"]
        sw.n[:] = g["nvec"]
        sw.H2D()
        system.AddThing(sw)
        arrays.append(sw)
    tr = tracers.Array(case["tracers"])
    tr.r[:] = _tracer_positions(case, seed)
    tr.H2D()
    system.AddThing(tr)
    lat.InitFromHydro()
    return {"case": case, "lat": lat, "system": system, "swimmers": arrays, "tracers": tr}


def prepare(case, seed):
    if case["path"] == "coupled":
        return _coupled_system(case, seed)
    if case["path"] == "fluid":
        rho, u, force = _flow(case, seed)
        lat = _lattice(case, rho, u)
        lat.force[:] = force
        lat.force.H2D()
        lat.InitFromHydro()
        return {"case": case, "lat": lat}
    if case["path"] == "restart":
        rho, u, _ = _flow(case, seed)
        lat = _lattice(case, rho, u)
        lat.fOld  # the host copy of a program that writes checkpoints
        return {"case": case, "lat": lat}
    parts = [_coupled_system(s, s["seed"], P=s["P"]) for s in _member_specs(case, seed)]
    ens = Ensemble([(p["lat"], p["swimmers"][0], p["tracers"]) for p in parts])
    ens.autotune()
    return {"case": case, "parts": parts, "ensemble": ens}


def _swimmer_outputs(sw, precision):
    # the velocities of a reduced-precision lattice carry FP32 values
    v = sw.v.data if precision == "f64" else sw.v.data.astype(np.float32)
    return {"r": sw.r.data, "v": v, "n": sw.n.data}


def _run_coupled(state):
    case, system = state["case"], state["system"]
    if case["readback"]:
        for _ in range(case["steps"]):
            system.Step()
            for sw in state["swimmers"]:
                sw.D2H()
    else:
        system.Step(case["steps"])
        for sw in state["swimmers"]:
            sw.D2H()
    precision, tr = case["precision"], state["tracers"]
    out = {"swimmers": [_swimmer_outputs(sw, precision) for sw in state["swimmers"]]}
    if case["history"]:
        tr.D2H()
        wide = precision == "f64"
        out["tracers"] = {"r": tr.r.data, "s": tr.s.data if wide else tr.s.data.astype(np.float32),
                          "v": tr.v.data if wide else tr.v.data.astype(np.float32)}
    else:
        tr.r.D2H()
        out["tracers"] = {"r": tr.r.data}
    out.update(_hydro(state["lat"]))
    return out


def run(state):
    case = state["case"]
    if case["path"] == "coupled":
        return _run_coupled(state)
    if case["path"] == "fluid":
        lat = state["lat"]
        for _ in range(case["steps"]):
            lat.Step()
            lat.CalcHydro()
        return dict(_hydro(lat), f=_distributions(lat))
    if case["path"] == "restart":
        lat = state["lat"]
        lat.rho.H2D()
        lat.u.H2D()
        lat.InitFromHydro()
        lat.fOld.D2H()
        return {"f": lat.fOld.data}
    state["ensemble"].Step(case["steps"])
    r, n, u = [], [], []
    for p in state["parts"]:
        sw = p["swimmers"][0]
        sw.D2H()
        r.append(sw.r.data)
        n.append(sw.n.data)
        u.append(_hydro(p["lat"])["u"])
    return {"r": np.concatenate(r, axis=1), "n": np.concatenate(n, axis=1), "u": torch.cat(u)}


# ---------------------------------------------------------------------------
# work: what a pass cannot do without
# ---------------------------------------------------------------------------
SITE_FLOPS = 240  # collision and moments of one site
PARTICLE_FLOPS = 64 * 8  # one 4^3 stencil


def _coupled_work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    fb = F_BYTES[case["precision"]]
    hb = 8 if case["precision"] == "f64" else 4
    # per step: f read and written, rho and u written; r, n (or s) read and
    # written and v written per particle
    step = n * (30 * fb + 4 * hb) + 120 * (case["swimmers"] + case["tracers"])
    flops = n * SITE_FLOPS + PARTICLE_FLOPS * (4 * case["swimmers"] + case["tracers"])
    back = 72 * case["swimmers"] * (case["steps"] if case["readback"] else 1)
    back += (72 if case["history"] else 24) * case["tracers"]
    return {"bytes": step * case["steps"] + back, "flops": flops * case["steps"]}


def work(case):
    if case["path"] == "coupled":
        return _coupled_work(case)
    if case["path"] == "ensemble":
        parts = [_coupled_work(s) for s in _member_specs(case, 1)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = case["nx"] * case["ny"] * case["nz"]
    fb, hb = F_BYTES[case["precision"]], 8 if case["precision"] == "f64" else 4
    if case["path"] == "fluid":
        return {"bytes": case["steps"] * n * (30 * fb + 3 * hb + 4 * hb),
                "flops": case["steps"] * n * SITE_FLOPS}
    # restart: rho and u come in, f goes out, in 64 bits; f written and read on the way
    return {"bytes": n * (32 + 120 + 30 * fb), "flops": n * 60}


# ---------------------------------------------------------------------------
# exact: the same pass in 64 bits with plain torch
# ---------------------------------------------------------------------------
C = torch.tensor([[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1],
                  [1, 1, 1], [1, 1, -1], [1, -1, 1], [1, -1, -1], [-1, 1, 1], [-1, 1, -1],
                  [-1, -1, 1], [-1, -1, -1]], dtype=torch.float64)
W = torch.tensor([2 / 9] + [1 / 9] * 6 + [1 / 72] * 8, dtype=torch.float64)
PAIRS = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))


class _Fluid64:
    """D3Q15 MRT fluid: f [15, nx, ny, nz], rho, u, force [3, nx, ny, nz]."""

    def __init__(self, size, tau, rho, u, sxz_from_xy):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.size, self.tau = size, tau
        self.rho = torch.as_tensor(rho, dtype=torch.float64, device=self.dev).clone()
        u = torch.zeros((3,) + size, dtype=torch.float64) if u is None else torch.as_tensor(u)
        self.u = u.to(self.dev, torch.float64).clone()
        self.force = torch.zeros((3,) + size, dtype=torch.float64, device=self.dev)
        j = self.rho * self.u
        S = {p: j[p[0]] * self.u[p[1]] for p in PAIRS}
        if sxz_from_xy:  # the reference's InitFromHydro takes S_xz from u_x u_y
            S[(0, 2)] = S[(0, 1)]
        self.f = self._project(self.rho, j, S)

    def _project(self, rho, j, S):
        tr = S[(0, 0)] + S[(1, 1)] + S[(2, 2)]
        f = torch.empty((15,) + self.size, dtype=torch.float64, device=self.dev)
        for p in range(15):
            c = [int(v) for v in C[p]]
            acc = rho - 1.5 * tr
            for a in range(3):
                if c[a]:
                    acc = acc + (3 * c[a]) * j[a]
            for a, b in PAIRS:
                if c[a] * c[b]:
                    acc = acc + (4.5 * c[a] * c[b] * (1 if a == b else 2)) * S[(a, b)]
            f[p] = float(W[p]) * acc
        return f

    def _sum(self, weights):
        out = torch.zeros(self.size, dtype=torch.float64, device=self.dev)
        for p, w in enumerate(weights):
            if w:
                out += self.f[p] * w
        return out

    def step(self):
        c = [[int(v) for v in row] for row in C]
        rho = self._sum([1] * 15)
        j = torch.stack([self._sum([c[p][a] for p in range(15)]) for a in range(3)])
        S = {(a, b): self._sum([c[p][a] * c[p][b] for p in range(15)]) - (rho / 3 if a == b else 0)
             for a, b in PAIRS}
        F, t = self.force, self.tau
        u = (j + 0.5 * F) / rho
        usq = (u * u).sum(0)
        uF = (u * F).sum(0)
        om = 1 / (t + 0.5)
        tr = S[(0, 0)] + S[(1, 1)] + S[(2, 2)]
        new = tr - om * (tr - rho * usq) + 2 * om * t * uF
        for a, b in PAIRS:
            s = S[(a, b)] - tr / 3 if a == b else S[(a, b)]
            eq = u[a] * u[b] - (usq if a == b else 0)
            s = s - om * (s - rho * eq)
            s = s + 2 * om * t * (u[a] * F[b] + F[a] * u[b] - (2 * uF if a == b else 0))
            S[(a, b)] = s + new / 3 if a == b else s
        g = self._project(rho, j + F, S)
        for p in range(15):
            self.f[p] = torch.roll(g[p], shifts=c[p], dims=(0, 1, 2))

    def calc_hydro(self):
        c = [[int(v) for v in row] for row in C]
        self.rho = self._sum([1] * 15)
        for a in range(3):
            self.u[a] = (self._sum([c[p][a] for p in range(15)]) + 0.5 * self.force[a]) / self.rho

    # -- particles: Peskin 4-point delta -------------------------------------
    def _nodes(self, r):
        """Site index [n] and weight [n] of each of the 64 nodes of positions r [3, n]."""
        idx, w = [], []
        for d in range(3):
            x0 = torch.ceil(r[d] - 2)
            node = x0[None] + torch.arange(4, device=self.dev, dtype=torch.float64)[:, None]
            x = (r[d] - node).abs()
            inner = 3 - 2 * x + torch.sqrt((1 + 4 * x - 4 * x * x).clamp(min=0))
            outer = 5 - 2 * x - torch.sqrt((-7 + 12 * x - 4 * x * x).clamp(min=0))
            w.append(torch.where(x < 1, inner, torch.where(x < 2, outer, 0 * x)) / 8)
            idx.append(torch.remainder(node, self.size[d]).to(torch.int64))
        for i in range(4):
            for j in range(4):
                wij = w[0][i] * w[1][j]
                row = (idx[0][i] * self.size[1] + idx[1][j]) * self.size[2]
                for k in range(4):
                    yield row + idx[2][k], wij * w[2][k]

    def interp(self, r):
        u = self.u.reshape(3, -1)
        v = torch.zeros_like(r)
        for s, w in self._nodes(r):
            v += w * u[:, s]
        return v

    def spread(self, r, F):
        force = self.force.view(3, -1)
        for s, w in self._nodes(r):
            force.index_add_(1, s, w * F)


def _philox(seed, ids, step, block):
    """Philox4x32-10 (Salmon et al. 2011): four words for counter (id, step, block)."""
    m32 = np.uint64(0xffffffff)
    one = np.ones_like(ids, dtype=np.uint64)
    c = [ids.astype(np.uint64), one * np.uint64(step & 0xffffffff), one * np.uint64(step >> 32),
         one * np.uint64(block)]
    k0, k1 = seed & 0xffffffff, seed >> 32
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & m32,
             (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xffffffff, (k1 + 0xBB67AE85) & 0xffffffff
    return c


def _normals(seed, ids, step):
    g = []
    for block in (1, 2):
        x = _philox(seed, ids, step, block)
        a, b = (((x[i] << np.uint64(21)) + (x[i + 1] >> np.uint64(11)) + np.uint64(1)).astype(
            np.float64) * 2.0 ** -53 for i in (0, 2))
        radius = np.sqrt(-2 * np.log(a))
        g += [radius * np.cos(2 * np.pi * b), radius * np.sin(2 * np.pi * b)]
    return np.stack(g[:3])


class _Particles64:
    def __init__(self, case, seed, fluid64, P=None):
        self.fluid = fluid64
        dev = fluid64.dev
        self.box = torch.tensor(fluid64.size, dtype=torch.float64, device=dev).reshape(3, 1)
        self.groups = _swimmer_groups(case, seed)
        for g in self.groups:
            g["P"] = P or g["P"]
            g["r"] = torch.as_tensor(g["r"], device=dev)
            g["nvec"] = torch.as_tensor(g["nvec"], device=dev)
        self.r = torch.as_tensor(_tracer_positions(case, seed), device=dev).clone()
        self.s = torch.zeros_like(self.r)
        self.v = torch.zeros_like(self.r)
        self.moves = 0

    def add_forces(self):
        self.fluid.force.zero_()
        for g in self.groups:
            self.fluid.spread(g["r"] - g["nvec"] * g["l"], -g["P"] * g["nvec"])
            self.fluid.spread(g["r"], g["P"] * g["nvec"])

    def move(self):
        for g in self.groups:
            r, n = g["r"], g["nvec"]
            v = self.fluid.interp(r)
            turned = n + (v - self.fluid.interp(r - n * g["l"])) / g["l"]
            g["v"] = g["mobility"] * g["P"] * n + v
            g["r"] = torch.remainder(r + g["v"], self.box)
            ids = np.arange(g["n"])
            uniform = ((_philox(g["seed"], ids, self.moves, 0)[0] >> np.uint64(8))
                       + np.uint64(1)).astype(np.float64) * 2.0 ** -24
            tumble = np.nonzero(uniform < g["alpha"])[0]
            if tumble.size:
                turned[:, torch.as_tensor(tumble, device=n.device)] = torch.as_tensor(
                    _normals(g["seed"], tumble, self.moves), device=n.device)
            g["nvec"] = turned / turned.norm(dim=0, keepdim=True)
        self.v = self.fluid.interp(self.r)
        self.r = torch.remainder(self.r + self.v, self.box)
        self.s = self.s + self.v
        self.moves += 1


def _exact_coupled(case, seed, P=None):
    fl = _Fluid64(_shape(case), case["tau"], _density(case, seed), None, False)
    parts = _Particles64(case, seed, fl, P)
    rho0 = float(np.float32(fl.rho.mean().item()))
    for _ in range(case["steps"]):
        parts.add_forces()
        fl.step()
        fl.calc_hydro()
        parts.move()
    return fl, parts, rho0


def _hydro64(fl, precision, rho0):
    rho, u = fl.rho.reshape(-1), fl.u.reshape(3, -1)
    return {"rho": rho, "u": u} if precision == "f64" else {"rho": rho - rho0, "u": u.T}


def exact(case, seed):
    if case["path"] == "coupled":
        fl, parts, rho0 = _exact_coupled(case, seed)
        out = {"swimmers": [{"r": g["r"], "v": g["v"], "n": g["nvec"]} for g in parts.groups],
               "tracers": {"r": parts.r}}
        if case["history"]:
            out["tracers"].update(s=parts.s, v=parts.v)
        out.update(_hydro64(fl, case["precision"], rho0))
        return out
    if case["path"] == "ensemble":
        r, n, u = [], [], []
        for s in _member_specs(case, seed):
            fl, parts, rho0 = _exact_coupled(s, s["seed"], P=s["P"])
            r.append(parts.groups[0]["r"])
            n.append(parts.groups[0]["nvec"])
            u.append(fl.u.reshape(3, -1).T)
        return {"r": torch.cat(r, 1), "n": torch.cat(n, 1), "u": torch.cat(u)}
    rho, u, force = _flow(case, seed)
    fl = _Fluid64(_shape(case), case["tau"], rho, u, True)
    if case["path"] == "restart":
        return {"f": fl.f}
    rho0 = float(np.float32(rho.mean()))
    fl.force = torch.as_tensor(force, device=fl.dev)
    for _ in range(case["steps"]):
        fl.step()
        fl.calc_hydro()
    out = _hydro64(fl, case["precision"], rho0)
    f = fl.f.reshape(15, -1)
    if case["precision"] == "f64":
        return dict(out, f=f)
    # deviations from w rho0 (over w in the 16-bit formats) in blocks of 32 sites
    w = W.to(f.device)[:, None]
    f = f - w * rho0
    if case["precision"] != "f32":
        f = f / w
    f = torch.nn.functional.pad(f, (0, -f.shape[1] % 32))
    return dict(out, f=f.reshape(15, -1, 32).permute(1, 0, 2))
