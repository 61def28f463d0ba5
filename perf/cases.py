"""The work that users have this framework do, as timed cases.

A case is a dict of plain values.  ``prepare`` builds what a user's program holds before
the call (the potential with its tables on the device, positions in GPU memory), ``run`` is
one pass through the public entry points, ``work`` says what that pass cannot do without and
``exact`` gives the same results from plain FP64 torch code that shares nothing with the
package.

Potentials
  halo      Multipole of an NFW halo, even l up to lmax (triaxial), a few dozen nodes
  lopsided  the same with every l (a halo with a satellite's wake)
  galaxy    halo + Miyamoto-Nagai disk + Hernquist bulge
  milkyway  halo lmax + Miyamoto-Nagai + DiskAnsatz + an NFW satellite moving on a (1000, 4)
            track + 16 Evolving Multipole snapshots (time dependent)
  disk      CylSpline of a barred disk, 32 x 32 nodes, m = 0, +-2, +-4, +-6
  barred    disk + halo
Positions follow the mass: Hernquist spheres around halos, exponential disks around disks,
all inside the radial grids of the tables.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import agama_gpu_b200 as agb
from agama_gpu_b200 import integrate
from agama_gpu_b200.autograd import potential_and_force
from agama_gpu_b200.coefs import CylSplineCoefs, MultipoleCoefs

G = 4.30091727067736e-06            # kpc (km/s)^2 / Msol
MUL0 = 3.5449077018110318           # 2 sqrt(pi): the angular factor of m = 0 terms
MUL1 = 5.0132565706694072           # and of the others, as the coefficient format has it
SNAPS, LMAX_SNAP, NODES_SNAP = 16, 16, 50
MN = dict(mass=5e10, scaleRadius=3.0, scaleHeight=0.3)
BULGE = dict(mass=1e10, scaleRadius=0.7)
ANSATZ = dict(surfaceDensity=1e9, scaleRadius=3.0, scaleHeight=0.3)
SATELLITE = dict(mass=1.5e11, scaleRadius=10.0)
CYL = dict(n_R=32, n_z=32, size=200.0, mmax=6)


def listed():
    return [
        # one orbit stepped by a program of the user's own: one force per call, all latency
        dict(name="point_force", kind="eval", tree="galaxy", lmax=8, nodes=50, n=1,
             call="force", precision="fp64"),
        # a thousand tracers with their tidal tensors (Jacobi radii, frequency maps)
        dict(name="tracer_tides", kind="eval", tree="galaxy", lmax=16, nodes=64, n=1000,
             call="evalDeriv", precision="fp64"),
        # a catalogue of clusters in the full time-dependent Milky Way model
        dict(name="clusters_milkyway", kind="eval", tree="milkyway", lmax=32, nodes=100, n=10007,
             call="eval", precision="fp64"),
        # a halo snapshot's forces: the reference's plain Multipole configuration
        dict(name="halo_force", kind="eval", tree="halo", lmax=8, nodes=50, n=100000,
             call="force", precision="fp64"),
        # density of a lopsided halo at the particles of a simulation
        dict(name="lopsided_density", kind="eval", tree="lopsided", lmax=20, nodes=64, n=500000,
             call="density", precision="fp64"),
        # forces on a barred disk's particles
        dict(name="disk_force", kind="eval", tree="disk", lmax=0, nodes=32, n=1000000,
             call="force", precision="fp64"),
        # the time-dependent Milky Way model at a million particles, full precision
        dict(name="milkyway_fp64", kind="eval", tree="milkyway", lmax=32, nodes=100, n=1048589,
             call="eval", precision="fp64"),
        # the same at the benchmark's 4M points, mixed precision
        dict(name="milkyway_mixed", kind="eval", tree="milkyway", lmax=32, nodes=100, n=4000000,
             call="eval", precision="mixed"),
        # many galaxies of uneven sizes in one launch (a semi-analytic model's step)
        dict(name="many_halos", kind="batch", units=48, lmax=32, nodes=120, n=200000,
             call="force", precision="mixed"),
        # a population of orbits, static potential
        dict(name="orbits", kind="orbits", tree="galaxy", lmax=8, nodes=50, n=20000, steps=32,
             precision="fp64"),
        # a stream fit: leapfrog forwards and its adjoint with the tables' gradient
        dict(name="stream_adjoint", kind="adjoint", tree="galaxy", lmax=16, nodes=64, n=131072,
             steps=8, precision="mixed"),
        # a potential fit to measured accelerations: gradients for positions and node tables
        dict(name="node_fit", kind="fit", tree="halo", lmax=12, nodes=50, n=200003,
             precision="fp64"),
    ]


def draw(rng):
    """One more case: sizes over the ranges of the listed ones (log-uniform), any tree,
    call and precision that go together; costs stay below the largest listed case's."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["eval"] * 6 + ["batch", "orbits", "adjoint", "fit"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "batch":
        return dict(kind=kind, units=rng.randint(3, 48), lmax=rng.randint(4, 32),
                    nodes=rng.randint(40, 120), n=size(3000, 200000),
                    call=rng.choice(["force", "eval"]), precision=prec)
    if kind == "orbits":
        return dict(kind=kind, tree=rng.choice(["galaxy", "halo"]), lmax=rng.randint(2, 16),
                    nodes=rng.randint(30, 100), n=size(100, 60000), steps=rng.choice([16, 32, 48]),
                    precision=prec)
    if kind == "adjoint":
        return dict(kind=kind, tree=rng.choice(["galaxy", "halo"]), lmax=rng.randint(4, 16),
                    nodes=rng.randint(40, 80), n=size(5000, 150000), steps=rng.randint(4, 8),
                    precision=prec)
    if kind == "fit":
        return dict(kind=kind, tree=rng.choice(["halo", "galaxy"]), lmax=rng.randint(4, 16),
                    nodes=rng.randint(30, 80), n=size(2000, 250000), precision="fp64")
    tree = rng.choice(["halo", "lopsided", "galaxy", "milkyway", "disk", "barred"])
    call = rng.choice(["force", "force", "eval", "eval", "potential", "evalDeriv", "density"])
    if call == "density" and tree in ("disk", "barred"):
        call = "force"
    case = dict(kind=kind, tree=tree, lmax=rng.randint(2, 32), nodes=rng.randint(30, 120),
                n=size(1, 4000000), call=call, precision=prec)
    if tree == "disk":
        case["lmax"], case["nodes"] = 0, 32
    cost = _flops_per_point(case) * (2 if prec == "fp64" else 1)
    most = _flops_per_point(listed()[7]) * listed()[7]["n"]
    case["n"] = max(1, min(case["n"], int(0.8 * most / cost)))
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _halo_arrays(lmax, nodes, seed, mass=1e12, rs=20.0, every_l=False, drift=0.0, rmin=1e-2,
                 rmax=1e3):
    """(r, Phi_lm, dPhi_lm/dr, [(l, m)]): an NFW monopole and harmonics of 5 % of it that
    fall as 10^(-l/2)."""
    rng = np.random.default_rng(seed)
    r = np.exp(np.linspace(math.log(rmin), math.log(rmax), nodes))
    labels = [(l, m) for l in range(lmax + 1) for m in range(-l, l + 1)]
    p0 = -G * mass * np.log1p(r / rs) / r
    d0 = G * mass * (np.log1p(r / rs) / (r * r) - 1.0 / (r * (r + rs)))
    phi = np.zeros((nodes, len(labels)))
    dphi = np.zeros_like(phi)
    for c, (l, m) in enumerate(labels):
        f = 1.0 if l == 0 else 0.05 * 10.0 ** (-l / 2.0) * rng.normal() * (1.0 + drift)
        if l % 2 == 0 or every_l:
            phi[:, c], dphi[:, c] = p0 * f, d0 * f
    return r, phi, dphi, labels


def _halo(arrays):
    r, phi, dphi, labels = arrays
    return agb.MultipolePotentialGPU(MultipoleCoefs(r, phi, dphi, labels, {"type": "Multipole"}))


def _main_halo(case, seed):
    lopsided = case.get("tree") == "lopsided"
    return _halo_arrays(case["lmax"], case["nodes"], seed, every_l=lopsided)


def _snapshot(i, seed):
    return _halo_arrays(LMAX_SNAP, NODES_SNAP, seed + 100, mass=2e11, rs=12.0,
                        drift=0.5 * i / (SNAPS - 1))


def _snap_times():
    return np.linspace(0.0, 1.5, SNAPS)


def _track(seed):
    """(1000, 4) rows [t, x, y, z]: an inclined circular orbit at 50 kpc."""
    inc = np.random.default_rng(seed + 3).uniform(0.2, 0.6)
    t = np.linspace(0.0, 2.0, 1000)
    w = 2.0 * math.pi / 1.5
    return np.stack([t, 50.0 * np.cos(w * t), 50.0 * np.sin(w * t) * math.cos(inc),
                     50.0 * np.sin(w * t) * math.sin(inc)], axis=1)


def _epoch(seed):
    """The index of the track's row whose time the call asks for (inside the snapshots)."""
    return int(np.random.default_rng(seed + 9).integers(20, 740))


def _bar_arrays(seed):
    """(R, z, {m: Phi_m}): a Miyamoto-Nagai m = 0 and a bar in m = +-2, +-4, +-6."""
    rng = np.random.default_rng(seed + 1)
    R = np.sinh(np.linspace(0.0, math.asinh(CYL["size"]), CYL["n_R"]))
    z = np.sinh(np.linspace(-math.asinh(CYL["size"]), math.asinh(CYL["size"]), CYL["n_z"]))
    RR, ZZ = np.meshgrid(R, z, indexing="ij")
    p0 = -G * MN["mass"] / np.sqrt(RR ** 2 + (MN["scaleRadius"]
                                              + np.sqrt(ZZ ** 2 + MN["scaleHeight"] ** 2)) ** 2)
    phi = {0: p0}
    for m, a in zip(range(2, CYL["mmax"] + 1, 2), (0.1, 0.03, 0.01)):
        ph = rng.uniform(0.0, 2.0 * math.pi)
        phi[m] = a * np.exp(-RR / 4.0) * p0 * math.cos(ph)
        phi[-m] = a * np.exp(-RR / 4.0) * p0 * math.sin(ph)
    return R, z, phi


def _disk():
    return agb.MiyamotoNagaiPotentialGPU(**MN)


def _potential(case, seed):
    tree = case["tree"]
    if tree in ("halo", "lopsided"):
        pot = _halo(_main_halo(case, seed))
    elif tree == "galaxy":
        pot = _halo(_main_halo(case, seed)) + _disk() + agb.HernquistPotentialGPU(**BULGE)
    elif tree == "milkyway":
        pot = agb.CompositePotentialGPU([
            _halo(_main_halo(case, seed)), _disk(), agb.DiskAnsatzPotentialGPU(**ANSATZ),
            agb.ShiftedPotentialGPU(agb.NFWPotentialGPU(**SATELLITE), _track(seed)),
            agb.EvolvingPotentialGPU([_halo(_snapshot(i, seed)) for i in range(SNAPS)],
                                     _snap_times())])
    else:
        R, z, phi = _bar_arrays(seed)
        pot = agb.CylSplinePotentialGPU(CylSplineCoefs(R, z, phi, {"type": "CylSpline"}))
        if tree == "barred":
            pot = pot + _halo(_main_halo(case, seed))
    return pot.set_precision(case["precision"])


def _device():
    return torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() \
        else torch.device("cpu")


def _uniform(gen, *shape):
    return torch.rand(*shape, generator=gen, dtype=torch.float64, device=gen.device)


def _sphere(n, gen, a=10.0, rmin=0.02, rmax=300.0):
    """Isotropic Hernquist sphere of scale a, from rmin to rmax."""
    lo, hi = (rmin / (rmin + a)) ** 2, (rmax / (rmax + a)) ** 2
    su = torch.sqrt(lo + (hi - lo) * _uniform(gen, n))
    u = torch.randn(n, 3, generator=gen, dtype=torch.float64, device=gen.device)
    return u / u.norm(dim=1, keepdim=True) * (a * su / (1.0 - su))[:, None]


def _disk_points(n, gen):
    """Exponential disk: R ~ Gamma(2, 3 kpc), z ~ Laplace(0.3 kpc)."""
    R = -3.0 * torch.log((1.0 - _uniform(gen, n)) * (1.0 - _uniform(gen, n))) + 1e-3
    v = _uniform(gen, n) - 0.5
    z = -0.3 * torch.sign(v) * torch.log1p(-2.0 * v.abs())
    ph = 2.0 * math.pi * _uniform(gen, n)
    return torch.stack([R * torch.cos(ph), R * torch.sin(ph), z], dim=1)


def _generator(seed):
    # always drawn on the CPU: the same inputs whatever computes on them
    g = torch.Generator()
    g.manual_seed(1000003 * (seed + 1))
    return g


def _points(case, seed):
    gen = _generator(seed)
    if case.get("tree") in ("disk", "barred"):
        return _disk_points(case["n"], gen)
    return _sphere(case["n"], gen)


def _unit_specs(case, seed):
    """Uneven units: lmax, nodes, scale and particle count of each (the layout is the
    case's, the harmonics are the seed's)."""
    rng = np.random.default_rng([case["units"], case["lmax"], case["nodes"], case["n"]])
    out = []
    for u in range(case["units"]):
        out.append(dict(lmax=int(rng.integers(2, case["lmax"] + 1)),
                        nodes=int(rng.integers(30, case["nodes"] + 1)),
                        mass=float(10 ** rng.uniform(10, 12)), rs=float(rng.uniform(2.0, 30.0)),
                        seed=seed + 1000 + u,
                        n=int(math.exp(rng.uniform(math.log(1000), math.log(case["n"]))))))
    return out


def _unit_arrays(spec):
    return _halo_arrays(spec["lmax"], spec["nodes"], spec["seed"], spec["mass"], spec["rs"])


def _unit_points(specs, seed):
    gen = _generator(seed)
    return [_sphere(s["n"], gen, a=s["rs"]) for s in specs]


def _orbit_state(case, seed):
    """Positions of a sphere at 2-60 kpc and near-circular velocities."""
    gen = _generator(seed)
    x = _sphere(case["n"], gen, a=15.0, rmin=2.0, rmax=60.0)
    axis = torch.randn(case["n"], 3, generator=gen, dtype=torch.float64)
    t = torch.linalg.cross(axis, x)
    t = t / t.norm(dim=1, keepdim=True)
    v = t * (180.0 + 40.0 * torch.randn(case["n"], 1, generator=gen, dtype=torch.float64))
    target = x + torch.randn(case["n"], 3, generator=gen, dtype=torch.float64)
    return x, v, target


DT = 1e-3 / 0.977792221             # 1 Myr in kpc / (km/s)


def prepare(case, seed):
    dev = _device()
    kind = case["kind"]
    if kind == "batch":
        specs = _unit_specs(case, seed)
        pots = [_halo(_unit_arrays(s)) for s in specs]
        batch = agb.BatchedPotentialGPU(pots, [s["n"] for s in specs], precision=case["precision"])
        return dict(case=case, pot=batch, x=torch.cat(_unit_points(specs, seed)).to(dev))
    pot = _potential(case, seed)
    if kind in ("orbits", "adjoint"):
        x, v, target = (a.to(dev) for a in _orbit_state(case, seed))
        return dict(case=case, pot=pot, x=x, v=v, target=target,
                    integ=integrate.Leapfrog(pot, DT, precision=case["precision"]))
    x = _points(case, seed).to(dev)
    if kind == "fit":
        gen = _generator(seed + 17)
        return dict(case=case, pot=pot, x=x.requires_grad_(True), nodes=pot.node_parameters(),
                    g_phi=torch.randn(case["n"], generator=gen, dtype=torch.float64).to(dev),
                    g_force=torch.randn(case["n"], 3, generator=gen, dtype=torch.float64).to(dev))
    return dict(case=case, pot=pot, x=x, t=float(_track(seed)[_epoch(seed), 0]))


def run(state):
    case, pot, x = state["case"], state["pot"], state["x"]
    kind = case["kind"]
    if kind == "orbits":
        xT, vT, _ = state["integ"].run(x, state["v"], case["steps"],
                                       checkpoint_every=case["steps"])
        return {"x": xT, "v": vT}
    if kind == "adjoint":
        # every step's positions are kept, as the integrator picks when they fit
        xT, vT, kept = state["integ"].run(x, state["v"], case["steps"], checkpoint_every=None)
        lx, lv, tables = state["integ"].adjoint(kept, case["steps"], 2.0 * (xT - state["target"]),
                                                torch.zeros_like(vT), table_grads=True)
        halo = next(k for k in tables if not isinstance(k, tuple))
        return {"x": xT, "v": vT, "dx": lx, "dv": lv, "dtable": tables[halo],
                "dconst": tables[("const", halo)]}
    if kind == "fit":
        phi, force = potential_and_force(pot, x)
        grads = torch.autograd.grad((phi, force), [x] + state["nodes"],
                                    grad_outputs=(state["g_phi"], state["g_force"]))
        return {"phi": phi.detach(), "force": force.detach(), "dx": grads[0],
                "dphi_nodes": grads[1], "ddphi_nodes": grads[2]}
    t = state.get("t", 0.0)
    if case["call"] == "eval":
        return pot.eval(x, pot=True, acc=True, t=t)
    return getattr(pot, case["call"])(x, t=t)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _harmonics(lmax, every_l=False):
    return sum(2 * l + 1 for l in range(0, lmax + 1, 1 if every_l else 2))


# multiply-adds a harmonic needs per point (radial quintic with the derivatives asked for,
# its Legendre function and the sums), times two
_PER_HARMONIC = {"potential": 16, "force": 30, "eval": 30, "evalDeriv": 50, "density": 34}


def _flops_per_point(case):
    call = case.get("call", "force")
    per = _PER_HARMONIC[call]
    tree = case.get("tree", "halo")
    f = 60.0
    if tree != "disk":
        f += per * _harmonics(case["lmax"], tree == "lopsided")
    if tree in ("disk", "barred"):
        f += 7 * (150 if call == "evalDeriv" else 90)
    if tree == "galaxy":
        f += 80
    if tree == "milkyway":
        f += 2 * per * _harmonics(LMAX_SNAP) + 150
    return f


def work(case):
    """Bytes: positions in, results out, tables once.  Flops: multiply-adds of the sums."""
    n, kind = case["n"], case["kind"]
    table = 8 * 6 * case["nodes"] * _harmonics(case["lmax"], case.get("tree") == "lopsided")
    if kind == "batch":
        sizes = _unit_specs(case, 0)
        total = sum(s["n"] for s in sizes)
        flops = sum(s["n"] * _flops_per_point(dict(case, lmax=s["lmax"])) for s in sizes)
        out = 24 if case["call"] == "force" else 32
        return {"bytes": total * (24 + out) + case["units"] * table // 4, "flops": flops}
    if kind == "orbits":
        f = _flops_per_point(case) * n * (case["steps"] + 1)
        return {"bytes": n * 96 * case["steps"] + table, "flops": f}
    if kind == "adjoint":
        f = _flops_per_point(case) * n * (case["steps"] + 1)
        return {"bytes": n * (96 + 96) * case["steps"] + 2 * table, "flops": 3.0 * f}
    if kind == "fit":
        return {"bytes": n * (24 + 32 + 32 + 24) + 2 * table, "flops": 3.0 * n * _flops_per_point(case)}
    out = {"potential": 8, "force": 24, "eval": 32, "evalDeriv": 80, "density": 8}[case["call"]]
    if case["tree"] == "milkyway":
        table += 2 * 8 * 6 * NODES_SNAP * _harmonics(LMAX_SNAP)
    if case["tree"] in ("disk", "barred"):
        table += 7 * CYL["n_R"] * CYL["n_z"] * 32
    return {"bytes": n * (24 + out) + table, "flops": n * _flops_per_point(case)}


# ---------------------------------------------------------------------------
# the same in plain FP64 torch
# ---------------------------------------------------------------------------
def _node_columns(arrays):
    """The non-zero harmonics, ordered by (|m|, l, cos before sin), and their (l, m)."""
    _, phi, dphi, labels = arrays
    keep = [c for c, (l, m) in enumerate(labels) if l == 0 or np.any(phi[:, c] != 0.0)]
    keep.sort(key=lambda c: (abs(labels[c][1]), labels[c][0], labels[c][1] < 0))
    return keep, [labels[c] for c in keep]


def _inverse_centre(p0, d0, r):
    """1/Phi_00(0) of the core the format puts inside the first node of such tables:
    Phi = U (r/r_1)^2 + W with the node's value and slope (differentiable in both)."""
    inv = 1.0 / (p0[0] - 0.5 * r[0] * d0[0])
    return torch.zeros_like(inv) if bool((p0 * inv >= 1.0).any()) else inv


class _Tables:
    """Quintic splines of one Multipole in log r: column 0 holds log(1/W - 1/Phi_00), the
    others the ratios Phi_lm / Phi_00.  nodes: differentiable (Phi, dPhi/dr) node tables."""

    def __init__(self, arrays, dev, nodes=None):
        r = torch.from_numpy(arrays[0]).to(dev)
        cols, self.lm = _node_columns(arrays)
        if nodes is None:
            nodes = [torch.from_numpy(np.ascontiguousarray(a[:, cols])).to(dev) for a in arrays[1:3]]
        phi, dphi = nodes
        lr = torch.log(r)
        self.lo, self.step, self.n = float(lr[0]), float((lr[-1] - lr[0]) / (len(r) - 1)), len(r) - 1
        p0, d0 = phi[:, :1], dphi[:, :1] * r[:, None]
        inv = _inverse_centre(phi[:, 0], dphi[:, 0], r)
        self.inv = inv.detach().clone() if not inv.requires_grad else inv
        ratio = phi[:, 1:] / p0
        f = torch.cat([torch.log(self.inv - 1.0 / p0), ratio], 1)
        m = torch.cat([d0 / (p0 * (self.inv * p0 - 1.0)),
                       (dphi[:, 1:] * r[:, None] - ratio * d0) / p0], 1) * self.step
        # second derivatives: a continuous third one, a vanishing fourth one at the ends
        n = len(r)
        A = torch.zeros(n, n, dtype=torch.float64, device=dev)
        i = torch.arange(1, n - 1, device=dev)
        A[i, i - 1], A[i, i], A[i, i + 1] = -3.0, 18.0, -3.0
        A[0, 0], A[0, 1], A[-1, -1], A[-1, -2] = 1.5, -1.0, 1.5, -1.0
        dd = f[1:] - f[:-1]
        rhs = torch.cat([(15.0 * dd[0] - 8.0 * m[0] - 7.0 * m[1])[None],
                         60.0 * (dd[1:] - dd[:-1]) - 24.0 * (m[2:] - m[:-2]),
                         (-15.0 * dd[-1] + 7.0 * m[-2] + 8.0 * m[-1])[None]])
        q = torch.linalg.solve(A, rhs)
        m0, m1, q0, q1 = m[:-1], m[1:], q[:-1], q[1:]
        poly = torch.stack([f[:-1], m0, 0.5 * q0,
                            10.0 * dd - 6.0 * m0 - 4.0 * m1 - 1.5 * q0 + 0.5 * q1,
                            -15.0 * dd + 8.0 * m0 + 7.0 * m1 + 1.5 * q0 - q1,
                            6.0 * dd - 3.0 * m0 - 3.0 * m1 + 0.5 * (q1 - q0)], -1)
        self.poly = poly                             # (interval, column, 6)
        self.L = max(l for l, _ in self.lm)

    def leaves(self):
        """The spline coefficients and 1/W as independent variables."""
        self.poly = self.poly.detach().clone().requires_grad_(True)
        self.inv = self.inv.detach().clone().requires_grad_(True)
        return self

    def place(self, x):
        lr = torch.log(x.norm(dim=1))
        k = torch.clamp(((lr.detach() - self.lo) / self.step).long(), 0, self.n - 1)
        return k, (lr - self.lo) / self.step - k

    def phi(self, x, k=None):
        """Phi at x (n, 3); k: the interval when all points share it."""
        r = x.norm(dim=1)
        kk, s = self.place(x)
        S = torch.stack([s ** j for j in range(6)], 0)                    # (6, n)
        if k is None:
            C = torch.einsum("ncj,jn->cn", self.poly[kk], S)
        else:
            C = self.poly[k] @ S
        F = 1.0 / (self.inv - torch.exp(C[0]))
        u, w, c = x[:, 0] / r, x[:, 1] / r, x[:, 2] / r
        # sin^m(theta) (cos, sin)(m phi) as polynomials of x/r, y/r
        re, im = [torch.ones_like(r)], [torch.zeros_like(r)]
        for _ in range(self.L):
            a, b = re[-1], im[-1]
            re.append(a * u - b * w)
            im.append(a * w + b * u)
        at = {lm: i for i, lm in enumerate(self.lm)}
        total = torch.ones_like(r)                    # the monopole: Phi_00 = F
        for m in range(self.L + 1):
            # Legendre functions over sin^m: seed (2m-1)!! with phase and normalisation
            seed = (-1) ** m * math.sqrt((2 * m + 1) / (4.0 * math.pi)
                                         * math.prod((2 * j - 1) / (2 * j) for j in range(1, m + 1)))
            Qp, Q = torch.zeros_like(r), torch.full_like(r, seed * (MUL0 if m == 0 else MUL1))
            even, odd = [], []
            for l in range(m, self.L + 1):
                if l > m:
                    d = l * l - m * m
                    a = math.sqrt((4 * l * l - 1) / d)
                    b = math.sqrt((2 * l + 1) * ((l - 1) ** 2 - m * m) / ((2 * l - 3) * d)) \
                        if l > m + 1 else 0.0
                    Q, Qp = a * c * Q - b * Qp, Q
                if (l, m) in at and l > 0:
                    even.append(C[at[(l, m)]] * Q)
                if m > 0 and (l, -m) in at:
                    odd.append(C[at[(l, -m)]] * Q)
            if even:
                total = total + sum(even[1:], even[0]) * re[m]
            if odd:
                total = total + sum(odd[1:], odd[0]) * im[m]
        return F * total


def _slopes(x, f, clamped):
    """Slopes at the nodes of the cubic spline along axis 0: natural ends, or a zero first
    slope where `clamped`."""
    n = len(x)
    h = np.diff(x)
    A, b = np.zeros((n, n)), np.zeros_like(f)
    for i in range(1, n - 1):
        A[i, i - 1], A[i, i + 1] = 1.0 / h[i - 1], 1.0 / h[i]
        A[i, i] = 2.0 * (A[i, i - 1] + A[i, i + 1])
        b[i] = 3.0 * ((f[i] - f[i - 1]) / h[i - 1] ** 2 + (f[i + 1] - f[i]) / h[i] ** 2)
    A[0, 0], A[0, 1], b[0] = 2.0, 1.0, 3.0 * (f[1] - f[0]) / h[0]
    if clamped:
        A[0, 0], A[0, 1], b[0] = 1.0, 0.0, 0.0
    A[-1, -1], A[-1, -2], b[-1] = 2.0, 1.0, 3.0 * (f[-1] - f[-2]) / h[-1]
    return np.linalg.solve(A, b)


class _Bar:
    """Bicubic Hermite interpolation of log(-Phi_0) and Phi_m / Phi_0 in asinh(R/s), asinh(z/s)."""

    def __init__(self, arrays, dev):
        R, z, phi = arrays
        # the scale: mass over central potential, the mass from a fit of exterior
        # multipoles to the grid's border (the format's own angular basis)
        Rb = np.concatenate([np.repeat(R[:-1], 2), np.full(len(z), R[-1])])
        zb = np.concatenate([np.tile([z[-1], z[0]], len(R) - 1), z])
        pb = np.concatenate([phi[0][:-1][:, [-1, 0]].reshape(-1), phi[0][-1]])
        rb = np.hypot(Rb, zb)
        ct, r0 = zb / rb, min(R[-1], np.abs(z).max())
        basis, older, old, cur = [np.ones_like(ct), ct], 0.0 * ct, np.ones_like(ct), ct
        for l in range(2, 9):
            new = (ct * (2 * l - 1) * cur - (l - 1) * older) / l
            basis.append(new)
            older, old, cur = old, cur, new
        M = np.stack([P * math.sqrt((2 * l + 1) / (4.0 * math.pi)) * MUL0 * (rb / r0) ** -(l + 1)
                      for l, P in enumerate(basis)], 1)
        W = np.linalg.lstsq(M, pb, rcond=None)[0]
        self.scale = W[0] * r0 * MUL0 / phi[0][0, (len(z) + 1) // 2]
        lR, lz = np.arcsinh(R / self.scale), np.arcsinh(z / self.scale)
        self.ms, nodes = sorted(phi, key=lambda m: (abs(m), m < 0)), []
        for m in self.ms:
            f = np.log(-phi[0]) if m == 0 else phi[m] / phi[0]
            fz = _slopes(lz, f.T, False).T
            nodes.append(np.stack([f, _slopes(lR, f, True), fz, _slopes(lR, fz, True)], -1))
        self.nodes = torch.from_numpy(np.stack(nodes)).to(dev)        # (harmonic, R, z, 4)
        self.lR, self.lz = torch.from_numpy(lR).to(dev), torch.from_numpy(lz).to(dev)

    def phi(self, x, k=None):
        R = torch.sqrt(x[:, 0] ** 2 + x[:, 1] ** 2)
        a, b = torch.asinh(R / self.scale), torch.asinh(x[:, 2] / self.scale)

        def axis(v, g):
            i = torch.clamp(torch.searchsorted(g, v.detach(), right=True) - 1, 0, len(g) - 2)
            h = g[i + 1] - g[i]
            t = (v - g[i]) / h
            return i, [(1 + 2 * t) * (1 - t) ** 2, t * t * (3 - 2 * t)], \
                [t * (1 - t) ** 2 * h, -t * t * (1 - t) * h]
        i, vR, sR = axis(a, self.lR)
        j, vz, sz = axis(b, self.lz)
        f = torch.zeros(len(self.ms), len(x), dtype=torch.float64, device=x.device)
        for p in range(2):
            for q in range(2):
                nd = self.nodes[:, i + p, j + q]                       # (harmonic, n, 4)
                f = f + nd[..., 0] * (vR[p] * vz[q]) + nd[..., 1] * (sR[p] * vz[q]) \
                    + nd[..., 2] * (vR[p] * sz[q]) + nd[..., 3] * (sR[p] * sz[q])
        c, s = x[:, 0] / R, x[:, 1] / R
        trig = {0: (torch.ones_like(R), torch.zeros_like(R))}
        for m in range(1, max(self.ms) + 1):
            e, o = trig[m - 1]
            trig[m] = (e * c - o * s, e * s + o * c)
        total = torch.ones_like(R)
        for h, m in enumerate(self.ms[1:], 1):
            total = total + f[h] * trig[abs(m)][0 if m > 0 else 1]
        return -torch.exp(f[0]) * total


def _mn(x, k=None):
    R2, z = x[:, 0] ** 2 + x[:, 1] ** 2, x[:, 2]
    h = MN["scaleRadius"] + torch.sqrt(z * z + MN["scaleHeight"] ** 2)
    return -G * MN["mass"] / torch.sqrt(R2 + h * h)


def _hernquist(x, k=None):
    return -G * BULGE["mass"] / (x.norm(dim=1) + BULGE["scaleRadius"])


def _ansatz(x, k=None):
    h = ANSATZ["scaleHeight"]
    u = x[:, 2].abs() / h
    return 4.0 * math.pi * G * ANSATZ["surfaceDensity"] \
        * torch.exp(-x.norm(dim=1) / ANSATZ["scaleRadius"]) * 0.5 * h * (torch.expm1(-u) + u)


def _leaves(case, seed, dev):
    """[(Phi function, weight, its Multipole tables or None, its CylSpline or None)]"""
    tree, out = case["tree"], []
    if tree != "disk":
        tab = _Tables(_main_halo(case, seed), dev)
        out.append((tab.phi, 1.0, tab, None))
    if tree in ("galaxy", "milkyway"):
        out.append((_mn, 1.0, None, None))
    if tree == "galaxy":
        out.append((_hernquist, 1.0, None, None))
    if tree in ("disk", "barred"):
        bar = _Bar(_bar_arrays(seed), dev)
        out.append((bar.phi, 1.0, None, bar))
    if tree == "milkyway":
        row = _track(seed)[_epoch(seed)]
        at = torch.from_numpy(row[1:]).to(dev)

        def satellite(x, k=None):
            r = (x - at).norm(dim=1)
            return -G * SATELLITE["mass"] * torch.log1p(r / SATELLITE["scaleRadius"]) / r
        out += [(_ansatz, 1.0, None, None), (satellite, 1.0, None, None)]
        ts = _snap_times()
        i = int(np.searchsorted(ts, row[0], side="right")) - 1
        w = (row[0] - ts[i]) / (ts[i + 1] - ts[i])
        for j, weight in ((i, 1.0 - w), (i + 1, w)):
            if weight:
                tab = _Tables(_snapshot(j, seed), dev)
                out.append((tab.phi, weight, tab, None))
    return out


_ORDER = ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (0, 2))


def _derivatives(fun, x, k, second):
    """Phi, grad Phi and (second) the six second derivatives at x."""
    x = x.detach().requires_grad_(True)
    phi = fun(x, k)
    g, = torch.autograd.grad(phi.sum(), x, create_graph=second)
    if not second:
        return phi.detach(), g, None
    rows = [torch.autograd.grad(g[:, i].sum(), x, retain_graph=i < 2)[0] for i in range(3)]
    return phi.detach(), g.detach(), torch.stack([rows[i][:, j] for i, j in _ORDER], 1)


def _sum_leaves(leaves, x, second=False):
    n, dev = len(x), x.device
    phi = torch.zeros(n, dtype=torch.float64, device=dev)
    grad = torch.zeros(n, 3, dtype=torch.float64, device=dev)
    hess = torch.zeros(n, 6, dtype=torch.float64, device=dev) if second else None
    for fun, weight, tab, bar in leaves:
        chunks = []
        if tab is not None:          # points of one interval together
            k, _ = tab.place(x)
            order = torch.argsort(k)
            counts = torch.bincount(k, minlength=tab.n).tolist()
            at = 0
            for kk, c in enumerate(counts):
                for p in range(at, at + c, 32768):
                    chunks.append((order[p:min(p + 32768, at + c)], kk))
                at += c
        else:
            everything = torch.arange(n, device=dev)
            chunks = [(everything[p:p + 262144], None) for p in range(0, n, 262144)]
        for idx, kk in chunks:
            p, g, h = _derivatives(fun, x[idx], kk, second)
            if bar is not None and second:
                # the CylSpline Hessian of the format leaves out the terms of
                # dPhi/dphi with the second derivatives of phi
                X, Y = x[idx, 0], x[idx, 1]
                q = (X * g[:, 1] - Y * g[:, 0]) / (X * X + Y * Y) ** 2
                h[:, 0] -= 2.0 * q * X * Y
                h[:, 1] += 2.0 * q * X * Y
                h[:, 3] -= q * (Y * Y - X * X)
            phi[idx] += weight * p
            grad[idx] += weight * g
            if second:
                hess[idx] += weight * h
    return phi, grad, hess


def _call_result(call, phi, grad, hess):
    if call == "potential":
        return phi
    if call == "force":
        return -grad
    if call == "eval":
        return phi, -grad
    if call == "density":
        return (hess[:, 0] + hess[:, 1] + hess[:, 2]) / (4.0 * 3.141592653589793 * G)
    return phi, -grad, -hess


def _force_of(leaves, x):
    """Force with its graph (x requires grad)."""
    phi = sum(w * f(x) for f, w, _, _ in leaves)
    return -torch.autograd.grad(phi.sum(), x, create_graph=True)[0]


def _exact_orbits(case, seed, dev):
    leaves = _leaves(case, seed, dev)
    x, v, _ = (a.to(dev) for a in _orbit_state(case, seed))
    F = -_sum_leaves(leaves, x)[1]
    for _ in range(case["steps"]):
        v = v + 0.5 * DT * F
        x = x + DT * v
        F = -_sum_leaves(leaves, x)[1]
        v = v + 0.5 * DT * F
    return {"x": x, "v": v}


def _exact_adjoint(case, seed, dev):
    leaves = _leaves(case, seed, dev)
    tab = leaves[0][2].leaves()
    parts = {k: [] for k in ("x", "v", "dx", "dv")}
    gpoly, ginv = torch.zeros_like(tab.poly), torch.zeros_like(tab.inv)
    X, V, T = (a.to(dev) for a in _orbit_state(case, seed))
    for p in range(0, case["n"], 8192):
        x0 = X[p:p + 8192].clone().requires_grad_(True)
        v0 = V[p:p + 8192].clone().requires_grad_(True)
        x, v = x0, v0
        F = _force_of(leaves, x)
        for _ in range(case["steps"]):
            v = v + 0.5 * DT * F
            x = x + DT * v
            F = _force_of(leaves, x)
            v = v + 0.5 * DT * F
        loss = ((x - T[p:p + 8192]) ** 2).sum()
        dx, dv, gp, gi = torch.autograd.grad(loss, [x0, v0, tab.poly, tab.inv])
        gpoly += gp
        ginv += gi
        for key, a in (("x", x.detach()), ("v", v.detach()), ("dx", dx), ("dv", dv)):
            parts[key].append(a)
        del x, v, F, loss
    out = {key: torch.cat(a) for key, a in parts.items()}
    out["dtable"] = gpoly.permute(1, 0, 2).contiguous()
    out["dconst"] = torch.cat([ginv.reshape(1), torch.zeros(7, dtype=torch.float64, device=dev)])
    return out


def _exact_fit(case, seed, dev):
    arrays = _main_halo(case, seed)
    cols, _ = _node_columns(arrays)
    nodes = [torch.from_numpy(np.ascontiguousarray(a[:, cols])).to(dev).requires_grad_(True)
             for a in arrays[1:3]]
    tab = _Tables(arrays, dev, nodes)
    build = (tab.poly, tab.inv)
    tab.leaves()
    leaves = [(tab.phi, 1.0, tab, None)] + _leaves(dict(case, lmax=0), seed, dev)[1:]
    x, gen = _points(case, seed).to(dev), _generator(seed + 17)
    g_phi = torch.randn(case["n"], generator=gen, dtype=torch.float64).to(dev)
    g_force = torch.randn(case["n"], 3, generator=gen, dtype=torch.float64).to(dev)
    parts = {"phi": [], "force": [], "dx": []}
    gpoly, ginv = torch.zeros_like(tab.poly), torch.zeros_like(tab.inv)
    for p in range(0, case["n"], 16384):
        q = x[p:p + 16384].clone().requires_grad_(True)
        phi = sum(w * f(q) for f, w, _, _ in leaves)
        F = -torch.autograd.grad(phi.sum(), q, create_graph=True)[0]
        loss = (phi * g_phi[p:p + 16384]).sum() + (F * g_force[p:p + 16384]).sum()
        dx, gp, gi = torch.autograd.grad(loss, [q, tab.poly, tab.inv])
        gpoly += gp
        ginv += gi
        for key, a in (("phi", phi.detach()), ("force", F.detach()), ("dx", dx)):
            parts[key].append(a)
        del phi, F, loss
    out = {key: torch.cat(a) for key, a in parts.items()}
    out["dphi_nodes"], out["ddphi_nodes"] = torch.autograd.grad(build, nodes,
                                                                grad_outputs=(gpoly, ginv))
    return out


def exact(case, seed):
    dev = _device()
    kind = case["kind"]
    if kind == "orbits":
        return _exact_orbits(case, seed, dev)
    if kind == "adjoint":
        return _exact_adjoint(case, seed, dev)
    if kind == "fit":
        return _exact_fit(case, seed, dev)
    second = case["call"] in ("evalDeriv", "density")
    if kind == "batch":
        specs, parts = _unit_specs(case, seed), []
        for s, x in zip(specs, _unit_points(specs, seed)):
            tab = _Tables(_unit_arrays(s), dev)
            parts.append(_sum_leaves([(tab.phi, 1.0, tab, None)], x.to(dev)))
        phi, grad = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
        return _call_result(case["call"], phi, grad, None)
    x = _points(case, seed).to(dev)
    return _call_result(case["call"], *_sum_leaves(_leaves(case, seed, dev), x, second))
