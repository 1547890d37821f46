"""What the framework's speed is measured on: calls that a user's program makes, through
the public Python entry points of pinq_b200 (KSHamiltonian, CellBatch, propagate,
DipolePropagation), over the range of cells, orbital counts and precisions in use.

A case is a dict of plain values:

  op         apply | batch | propagate | scf | cn | ortho | mlwf | adjoint
  nx ny nz   grid;  spacing  grid spacing (bohr), the cell is orthorhombic
  orbitals   M;  ld  leading dimension of the block (>= M)
  atoms      atoms with s + p Gaussian projectors;  sites  diamond | random | shell
  precision  fp64 (complex128) | mixed (complex64 storage)
  field      amplitude of the vector potential (atomic units, along x)
  steps      time steps of an adjoint case;  every  its checkpoint interval
  cells mix  number of cells of a batch, and the seed of their sizes

Inputs depend on the seed: thermal displacements of the atoms (and their potential and
projector tables) and the orbitals' random plane-wave coefficients.
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "inq-wannier-fork_b200"))

import pinq_b200 as pb  # noqa: E402
from pinq_b200.adjoint import DipolePropagation  # noqa: E402
from pinq_b200.batch import CellBatch  # noqa: E402
from pinq_b200.propagate import propagate  # noqa: E402

SPACING = 0.320625        # 10.26 / 32, the silicon-like cells
FINE = 30.0 / 144         # the 240-atom cage
RADIUS, SIGMA = 3.0, 1.0  # projector spheres
EKB = (1.5, -0.7, -0.7, -0.7)
DT = 0.05
LDA = 2
CUBIC = (16, 18, 20, 24, 30, 32, 36, 40, 48, 60, 64, 72, 80, 96, 128, 144)
BOXES = ((18, 24, 20), (24, 24, 48), (32, 32, 48), (36, 48, 60), (64, 64, 96))


def _case(name, op, n, orbitals, atoms, precision, **more):
    nx, ny, nz = (n, n, n) if isinstance(n, int) else n
    c = dict(name=name, op=op, nx=nx, ny=ny, nz=nz, spacing=SPACING, orbitals=orbitals, ld=orbitals, atoms=atoms,
             sites="random", precision=precision, field=0.0, steps=0, every=0, cells=0, mix=0)
    c.update(more)
    return c


def listed():
    return [
        # a molecule in a small box: a few launches on a nearly empty GPU, a partly filled orbital group
        _case("apply_4atom_fp64", "apply", 24, 10, 4, "fp64"),
        # the 64-atom supercell with all its 128 occupied states: the ordinary H|psi> of a
        # ground-state or propagation loop, in both precisions
        _case("apply_64atom_mixed", "apply", 64, 128, 64, "mixed", sites="diamond"),
        _case("apply_64atom_fp64", "apply", 64, 128, 64, "fp64", sites="diamond"),
        # a block whose rows are not 16-byte aligned (odd orbital count), with a field, on a
        # grid that is no power of two
        _case("apply_odd_mixed", "apply", 60, 37, 28, "mixed", field=0.05),
        # the large cell: 240 atoms, one GPU's share (64) of its 480 states
        _case("apply_240atom_mixed", "apply", 144, 64, 240, "mixed", spacing=FINE, sites="shell"),
        # sixteen uneven cells at once: high-throughput screening
        _case("batch_16cells_mixed", "batch", 48, 64, 16, "mixed", cells=16, mix=0),
        # a step of the time loop as a user runs it: ETRS, density, energy, dipole
        _case("propagate_64atom_mixed", "propagate", 64, 128, 64, "mixed", sites="diamond", field=0.02),
        # real-time TDDFT with the LDA potential following the density
        _case("scf_27atom_fp64", "scf", 48, 40, 27, "fp64", field=0.01),
        # the implicit propagator, to its default convergence
        _case("cn_16atom_mixed", "cn", 40, 24, 16, "mixed", field=0.01),
        # orthonormalisation of a block of guess or propagated states
        _case("ortho_128states_fp64", "ortho", 64, 128, 0, "fp64"),
        # Wannier centres after a time step
        _case("mlwf_64states_fp64", "mlwf", 48, 64, 0, "fp64"),
        # gradients of the final dipole with respect to the pulse and the potential
        _case("adjoint_8atom_mixed", "adjoint", 32, 16, 8, "mixed", sites="diamond", field=0.01, steps=20, every=10),
    ]


# ------------------------------------------------------------------ drawn cases
_APPLIES = {"apply": 1, "batch": 8, "propagate": 11, "scf": 24, "cn": 60, "ortho": 8, "mlwf": 30, "adjoint": 32}


def _cost(c):
    """Orbital-grid-point applications of H (complex64) of about the same time."""
    n = c["nx"] * c["ny"] * c["nz"]
    w = n * c["orbitals"] * _APPLIES[c["op"]] * max(1, c["steps"]) * (2 if c["precision"] == "fp64" else 1)
    if c["op"] in ("ortho", "mlwf"):
        w *= max(1.0, c["orbitals"] / 128.0)
    return w


_MOST = 64 ** 3 * 128 * 11  # the listed propagation step


def draw(rng):
    op = rng.choice(["apply"] * 5 + ["batch", "propagate", "scf", "cn", "ortho", "mlwf", "adjoint"])
    while True:
        precision = rng.choice(["mixed", "fp64"])
        if rng.random() < 0.2:
            n = rng.choice(BOXES)
        else:
            size = math.exp(rng.uniform(math.log(16), math.log(144)))
            n = min(CUBIC, key=lambda k: abs(math.log(k / size)))
            n = (n, n, n)
        most_m = 300 if op == "apply" else 160
        least_m = 4 if op == "mlwf" else 1
        m = int(round(math.exp(rng.uniform(math.log(least_m), math.log(most_m)))))
        fine = max(n) > 96
        if fine and op not in ("apply", "ortho"):
            continue
        spacing = FINE if fine else SPACING
        volume = n[0] * n[1] * n[2] * spacing ** 3
        if op == "mlwf" and m > 0.02 * volume:
            continue
        atoms = 0 if op in ("ortho", "mlwf") else max(1, min(240, int(rng.uniform(0.2, 1.0) * 0.0074 * volume)))
        c = _case("", op, n, m, atoms, precision, spacing=spacing)
        del c["name"]
        if op == "apply":
            c["ld"] = m + rng.choice([0, 0, 0, 1, 3, 8])
        if op in ("apply", "propagate", "scf", "cn", "adjoint"):
            c["field"] = rng.choice([0.0, round(rng.uniform(0.002, 0.05), 4)])
        if op == "adjoint":
            c["steps"] = rng.randint(3, 24)
            c["every"] = rng.randint(2, 12)
            c["field"] = max(c["field"], 0.002)
        if op == "batch":
            c["nx"] = c["ny"] = c["nz"] = 48
            c["orbitals"] = c["ld"] = 64
            c["cells"], c["mix"], c["atoms"] = rng.randint(3, 16), rng.randint(1, 10 ** 6), 16
        if _cost(c) <= _MOST:
            return c


# ------------------------------------------------------------------ systems
def _random_sites(rng, edges, count, apart=2.0):
    """count points of a periodic box, at least `apart` from one another."""
    sites = np.zeros((0, 3))
    while len(sites) < count:
        p = rng.uniform(0.0, 1.0, 3) * edges
        d = sites - p
        d -= edges * np.round(d / edges)
        if not len(sites) or (d * d).sum(1).min() > apart * apart:
            sites = np.concatenate([sites, p[None]])
    return sites


def _positions(c, rng):
    edges = np.array([c["nx"], c["ny"], c["nz"]]) * c["spacing"]
    if c["sites"] == "diamond":
        reps = round((c["atoms"] / 8) ** (1 / 3))
        base = np.array([[0, 0, 0], [0, 2, 2], [2, 0, 2], [2, 2, 0], [1, 1, 1], [1, 3, 3], [3, 1, 3], [3, 3, 1]]) / 4.0
        cells = np.stack(np.meshgrid(*[np.arange(reps)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
        sites = ((cells + base).reshape(-1, 3)) / reps * edges
    elif c["sites"] == "shell":
        k = np.arange(c["atoms"]) + 0.5
        z = 1.0 - 2.0 * k / c["atoms"]
        r, phi = np.sqrt(1.0 - z * z), k * np.pi * (3.0 - np.sqrt(5.0))
        sites = edges / 2 + 6.7 * np.stack([r * np.cos(phi), r * np.sin(phi), z], 1)
    else:
        return _random_sites(rng, edges, c["atoms"])
    return sites + rng.normal(0.0, 0.05, sites.shape)  # thermal displacements


def _projectors(c, sites):
    """The separable s + p tables a pseudopotential code hands over: per atom the grid points
    within RADIUS (periodic images included), their position relative to the atom in lattice
    units, the projectors' values there and their energies."""
    nr = np.array([c["nx"], c["ny"], c["nz"]])
    h = c["spacing"]
    w = int(RADIUS / h) + 2
    o = np.stack(np.meshgrid(*[np.arange(-w, w + 1)] * 3, indexing="ij"), -1).reshape(-1, 3)
    coords, rel, beta = [], [], []
    for p in sites:
        i = np.round(p / h).astype(int) + o
        r = i * h - p
        keep = (r * r).sum(1) <= RADIUS * RADIUS
        i, r = i[keep], r[keep]
        f = (r / (nr * h)).astype(np.float32)
        x = f.astype(np.float64) * (nr * h)
        g = np.exp(-(x * x).sum(1) / (2 * SIGMA * SIGMA))
        y0, y1 = 0.5 / math.sqrt(math.pi), math.sqrt(3.0 / (4.0 * math.pi))
        coords.append(i % nr)
        rel.append(f)
        beta.append(np.stack([y0 * g, y1 * x[:, 1] * g, y1 * x[:, 2] * g, y1 * x[:, 0] * g]))
    n, smax = len(sites), max(len(f) for f in rel)
    kb = dict(counts=np.array([len(f) for f in rel], np.int32), coords=-np.ones((n, smax, 3), np.int32),
              relpos=np.zeros((n, smax, 3), np.float32), beta=np.zeros((n, 4, smax)),
              coeff=np.tile(np.array(EKB), (n, 1)), smax=smax, L=4)
    for a in range(n):
        k = len(rel[a])
        kb["coords"][a, :k], kb["relpos"][a, :k], kb["beta"][a, :, :k] = coords[a], rel[a], beta[a]
    return kb


def _sym(n):
    i = np.arange(n)
    return np.where(i >= (n + 1) // 2, i - n, i)


def _potential(c, sites):
    """Periodic sum of Gaussian wells on the atoms, [N] (FP64, host)."""
    if not len(sites):
        return np.zeros(c["nx"] * c["ny"] * c["nz"])
    axes = []
    for d, n in enumerate((c["nx"], c["ny"], c["nz"])):
        edge = n * c["spacing"]
        x = np.arange(n) * c["spacing"] - sites[:, d:d + 1]
        axes.append(torch.as_tensor(sum(np.exp(-(x + k * edge) ** 2 / (2 * 0.8 ** 2)) for k in (-2, -1, 0, 1, 2)),
                                    device="cuda"))
    xy = (axes[0][:, :, None] * axes[1][:, None, :]).reshape(len(sites), -1)
    return (-4.0 * (xy.T @ axes[2])).reshape(-1).cpu().numpy()


def _plane_waves(c, seed, ecut=25.0):
    """M normalised orbitals of random complex plane-wave coefficients below ecut, [N, ld]."""
    nr, m, h = (c["nx"], c["ny"], c["nz"]), c["orbitals"], c["spacing"]
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    kx, ky, kz = (torch.as_tensor(2 * np.pi * _sym(n) / (n * h), device="cuda") for n in nr)
    inside = 0.5 * (kx[:, None, None] ** 2 + ky[None, :, None] ** 2 + kz[None, None, :] ** 2) <= ecut
    dtype = torch.complex128 if c["precision"] == "fp64" else torch.complex64
    n = nr[0] * nr[1] * nr[2]
    out = torch.zeros((n, c["ld"]), dtype=dtype, device="cuda")
    for m0 in range(0, m, 8):
        k = min(8, m - m0)
        z = torch.randn((k,) + nr, generator=g, device="cuda", dtype=dtype) * inside
        x = torch.fft.ifftn(z, dim=(1, 2, 3)).reshape(k, n)
        out[:, m0:m0 + k] = (x / (x.norm(dim=1, keepdim=True) * math.sqrt(h ** 3))).T
    return out[:, :m]


def _gaussians(c, seed):
    """M orthonormal localised states on random sites, mixed as a time step mixes them."""
    rng = np.random.default_rng(seed)
    nr, m, h = (c["nx"], c["ny"], c["nz"]), c["orbitals"], c["spacing"]
    edges = np.array(nr) * h
    sites = _random_sites(rng, edges, m)
    ax = []
    for d, n in enumerate(nr):
        x = np.arange(n) * h - sites[:, d:d + 1]
        x -= edges[d] * np.round(x / edges[d])
        ax.append(torch.as_tensor(np.exp(-x * x / 2), device="cuda"))
    psi = torch.einsum("ma,mb,mc->abcm", *ax).reshape(-1, m) + 0j
    s, v = torch.linalg.eigh(psi.conj().T @ psi * h ** 3)
    psi = psi @ (v * s.rsqrt()) @ v.conj().T
    g = torch.as_tensor(rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m)), device="cuda") * (0.1 / math.sqrt(m))
    psi = psi @ torch.linalg.matrix_exp(g - g.conj().T)
    return psi.to(torch.complex128 if c["precision"] == "fp64" else torch.complex64).contiguous()


def _cells(c):
    """The sizes of a batch: cubic cells of 24 to 48 points, 8 to 64 orbitals, 2 to 16 atoms."""
    r = random.Random(c["mix"])
    out = []
    for _ in range(c["cells"]):
        n = r.choice([24, 32, 40, 48])
        out.append(_case("", "apply", n, 8 * r.randint(1, 8), min(r.randint(2, 16), n // 3), c["precision"]))
    return out


def _inputs(c, seed):
    """The user's data, made from the seed: atoms' tables, potential (host) and orbitals (GPU)."""
    rng = np.random.default_rng(seed)
    if c["op"] == "mlwf":
        return dict(V=None, kb=None, psi=_gaussians(c, seed))
    sites = _positions(c, rng) if c["atoms"] else np.zeros((0, 3))
    s = dict(V=_potential(c, sites), kb=_projectors(c, sites) if c["atoms"] else None, psi=_plane_waves(c, seed + 1))
    s["amplitudes"] = c["field"] * rng.normal(size=max(2, c["steps"]))
    return s


def _lattice(c):
    return np.diag([c["nx"] * c["spacing"], c["ny"] * c["spacing"], c["nz"] * c["spacing"]])


def _ham(c, s):
    h = pb.KSHamiltonian(_lattice(c), (c["nx"], c["ny"], c["nz"]), c["precision"])
    if s["V"] is not None:
        h.set_scalar_potential(s["V"])
    if s["kb"] is not None:
        h.set_projectors(s["kb"])
    if c["op"] in ("propagate", "scf", "cn", "adjoint"):
        h.set_fourier_sphere_mask(True)  # 1/2 G_max^2 dt / 2 is beyond the series' stable range otherwise
    return h


def _pulse(c):
    return lambda t: np.array([c["field"] * math.cos(0.3 * t), 0.0, 0.0])


def _occ(c):
    return np.full(c["orbitals"], 2.0)


# ------------------------------------------------------------------ the measured calls
def prepare(case, seed):
    c = case
    if c["op"] == "batch":
        cells = _cells(c)
        ins = [_inputs(k, 1000 * seed + i) for i, k in enumerate(cells)]
        hams = [_ham(k, s) for k, s in zip(cells, ins)]
        return dict(c=c, hams=hams, batch=CellBatch(hams), psis=[s["psi"] for s in ins],
                    outs=[torch.empty_like(s["psi"]) for s in ins])
    s = _inputs(c, seed)
    h = _ham(c, s)
    s.update(c=c, ham=h)
    if c["op"] == "apply":
        h.set_uniform_vector_potential(_pulse(c)(0.0))
        s["out"] = torch.empty((h.N, c["ld"]), dtype=h.dtype, device="cuda")[:, :c["orbitals"]]
    if c["op"] in ("scf", "cn"):
        s["kA"] = [h.cart_to_cov(_pulse(c)(t)) for t in (0.0, DT)]
    if c["op"] == "scf":
        s["occ"] = torch.as_tensor(_occ(c), device="cuda")
        s["vion"] = torch.as_tensor(s["V"], device="cuda")
        s["rho"] = h.density(s["psi"], s["occ"])
        h.ks_potential(s["rho"], s["vion"], LDA)
    if c["op"] == "mlwf":
        s["work"] = torch.empty_like(s["psi"])
    if c["op"] == "adjoint":
        s["prop"] = DipolePropagation(h, s["psi"], _occ(c), DT, every=c["every"])
    return s


def run(state):
    s = state
    c = s["c"]
    op = c["op"]
    if op == "apply":
        return s["ham"].apply(s["psi"], s["out"])
    if op == "batch":
        return s["batch"].apply(s["psis"], s["outs"])
    h, psi = s["ham"], s["psi"]
    if op == "propagate":
        r = propagate(h, psi, _occ(c), DT, 1, vector_potential=_pulse(c))
        return dict(psi=psi, energy=np.array(r.total_energy), dipole=np.array(r.dipole))
    if op == "scf":
        _, en = h.etrs_scf_step_(psi, s["rho"], DT, s["kA"][0], s["kA"][1], s["occ"], s["vion"], LDA)
        return dict(psi=psi, rho=s["rho"], energies=np.array([en[k] for k in ("external", "hartree", "xc", "nvxc")]))
    if op == "cn":
        h.crank_nicolson_step_(psi, DT, s["kA"][0], s["kA"][1])
        return psi
    if op == "ortho":
        return h.orthonormalize_(psi)
    if op == "mlwf":
        s["work"].copy_(psi)  # each pass starts from the states as the time step left them
        centres, spreads, _ = h.mlwf_step_(s["work"])
        return dict(psi=s["work"], centres=centres, spreads=spreads)
    dipole = s["prop"].forward(s["amplitudes"])
    ga, gv = s["prop"].backward()
    return dict(dipole=dipole, pulse=ga, potential=gv)


def _apply_work(c, b):
    """H once: the block read and written, the potential and the projector tables read; the
    flops of the two FFTs, the products with kinetic energy and potential, the projectors."""
    n, m = c["nx"] * c["ny"] * c["nz"], c["orbitals"]
    entries = c["atoms"] * 4.0 / 3.0 * math.pi * RADIUS ** 3 / c["spacing"] ** 3
    return dict(bytes=2 * n * m * b + n * b / 2 + entries * 4 * b / 2,
                flops=m * (n * (10 * math.log2(n) + 10) + entries * (2 * 16 + 2 * 8)))


def work(case):
    """Each H application of a step reads and writes its block once (a block does not stay
    on the chip); the other work counts its inputs and outputs once."""
    c = case
    b = 16 if c["precision"] == "fp64" else 8
    n, m = c["nx"] * c["ny"] * c["nz"], c["orbitals"]
    if c["op"] == "batch":
        each = [_apply_work(k, b) for k in _cells(c)]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    if c["op"] == "ortho":  # overlap (Hermitian) and rotation (triangular)
        return dict(bytes=2 * n * m * b, flops=8.0 * n * m * m)
    if c["op"] == "mlwf":  # three weighted Gram matrices, one dense rotation
        return dict(bytes=2 * n * m * b, flops=4 * 8.0 * n * m * m)
    a = _apply_work(c, b)
    # propagate: 8 in the step, 2 energies; scf: 4 + 4 per iteration (at least 2); cn: at
    # least one sweep of 5 steps with 2 each; adjoint: 8 forward, 8 backward a step
    applies = dict(apply=1, propagate=10, scf=12, cn=11, adjoint=16 * c["steps"])[c["op"]]
    return {k: applies * v for k, v in a.items()}


def tolerance(case):
    """About four times the difference of two correct evaluations at this precision."""
    fp64 = {"apply": 1e-14, "batch": 1e-14, "propagate": 1e-14, "scf": 1e-13, "cn": 1e-12, "ortho": 2e-14,
            "mlwf": 1e-11, "adjoint": 1e-12}
    mixed = {"apply": 4e-6, "batch": 2e-6, "propagate": 2e-6, "scf": 4e-6, "cn": 2e-6, "ortho": 4e-7, "mlwf": 2e-5,
             "adjoint": 2e-5}
    return {"rel": (fp64 if case["precision"] == "fp64" else mixed)[case["op"]]}


# ------------------------------------------------------------------ 64-bit reference in plain torch
class _Plain:
    """H of one case in complex128 with torch: psi [N, M]."""

    def __init__(self, c, s):
        self.nr, self.h = (c["nx"], c["ny"], c["nz"]), c["spacing"]
        self.n = self.nr[0] * self.nr[1] * self.nr[2]
        self.dv = self.h ** 3
        self.v = torch.as_tensor(s["V"], device="cuda")
        self.mask = c["op"] in ("propagate", "scf", "cn", "adjoint")
        sy = [torch.as_tensor(_sym(n).astype(np.float64), device="cuda") for n in self.nr]
        frac = [a / n for a, n in zip(sy, self.nr)]
        # |n / N|^2 <= 1/4, in whole numbers: points lie exactly on the sphere
        sq = [(torch.as_tensor(_sym(n), device="cuda") * (self.n // n)) ** 2 for n in self.nr]
        self.inside = 4 * (sq[0][:, None, None] + sq[1][None, :, None] + sq[2][None, None, :]) <= self.n ** 2
        self.g = torch.stack(torch.meshgrid(*[2 * math.pi / self.h * f for f in frac], indexing="ij"))
        self.r = torch.stack(torch.meshgrid(*[self.h * a for a in sy], indexing="ij")).reshape(3, -1)
        self.kb = []
        if s["kb"] is not None:
            edges = torch.tensor([n * self.h for n in self.nr], dtype=torch.float64, device="cuda")
            for a, k in enumerate(s["kb"]["counts"]):
                i = s["kb"]["coords"][a, :k].astype(np.int64)
                at = torch.as_tensor((i[:, 0] * self.nr[1] + i[:, 1]) * self.nr[2] + i[:, 2], device="cuda")
                rel = torch.as_tensor(s["kb"]["relpos"][a, :k].astype(np.float64), device="cuda") * edges
                self.kb.append((at, rel, torch.as_tensor(s["kb"]["beta"][a, :, :k], device="cuda"),
                                torch.as_tensor(s["kb"]["coeff"][a], device="cuda")))

    def kinetic(self, ka):
        t = 0.5 * ((self.g + ka[:, None, None, None]) ** 2).sum(0)
        return torch.where(self.inside, t, 0.5 * (ka * ka).sum()) if self.mask else t

    def apply(self, psi, ka, v=None):
        v = self.v if v is None else v
        t = self.kinetic(ka)
        out = []
        for m0 in range(0, psi.shape[1], 16):
            x = psi[:, m0:m0 + 16]
            f = torch.fft.fftn(x.reshape(self.nr + (-1,)), dim=(0, 1, 2))
            y = torch.fft.ifftn(t[..., None] * f, dim=(0, 1, 2)).reshape(self.n, -1) + v[:, None] * x
            for at, rel, beta, coeff in self.kb:
                phase = torch.exp(1j * (rel @ ka))
                p = (self.dv * coeff)[:, None] * ((beta * phase) @ x[at])
                y = y.index_add(0, at, (beta * phase.conj()).T.contiguous() @ p)
            out.append(y)
        return torch.cat(out, 1)

    def series(self, psi, ka, f, v=None):
        """sum_k (f H)^k / k! psi, k <= 4, for each factor of f."""
        sums, y, c = [psi.clone() for _ in f], psi, [1.0 for _ in f]
        for k in range(1, 5):
            y = self.apply(y, ka, v)
            c = [a * b / k for a, b in zip(c, f)]
            sums = [s + a * y for s, a in zip(sums, c)]
        return sums

    def etrs(self, psi, k0, k1, v=None):
        psi = self.series(psi, k0, [0.5j * DT], v)[0]
        return self.series(psi, k1, [0.5j * DT], v)[0]

    def density(self, psi):
        return 2.0 * (psi.real ** 2 + psi.imag ** 2).sum(1)

    def dipole(self, rho):
        return self.dv * (self.r * rho).sum(1)

    def energy(self, psi, ka):
        hp = self.apply(psi, ka)
        return (2.0 * ((hp.conj() * psi).sum(0).real / (psi.abs() ** 2).sum(0))).sum()

    def ks_potential(self, rho):
        """vion + V_H + the Slater and Perdew-Zunger LDA potential, and the four energies."""
        g2 = (self.g ** 2).sum(0)
        f = torch.fft.fftn(rho.reshape(self.nr) + 0j)
        vh = torch.fft.ifftn(torch.where(g2 < 1e-6, 0.0, 4 * math.pi / g2.clamp_min(1e-6)) * f).real.reshape(-1)
        n = rho.clamp_min(1e-15)
        ex = -0.75 * (3 / math.pi) ** (1 / 3) * n ** (1 / 3)
        rs = (3 / (4 * math.pi * n)) ** (1 / 3)
        den = 1 + 1.0529 * rs.sqrt() + 0.3334 * rs
        ec1, dc1 = -0.1423 / den, 0.1423 * (0.5 * 1.0529 / rs.sqrt() + 0.3334) / den ** 2
        ec2 = 0.0311 * rs.log() - 0.048 + 0.0020 * rs * rs.log() - 0.0116 * rs
        dc2 = 0.0311 / rs + 0.0020 * (rs.log() + 1) - 0.0116
        ec, dc = torch.where(rs >= 1, ec1, ec2), torch.where(rs >= 1, dc1, dc2)
        exc, vxc = ex + ec, 4 / 3 * ex + ec - rs / 3 * dc
        exc, vxc = (torch.where(rho >= 1e-15, a, 0.0) for a in (exc, vxc))
        en = torch.stack([(rho * self.v).sum(), 0.5 * (rho * vh).sum(), (exc * rho).sum(), (rho * vxc).sum()]) * self.dv
        return self.v + vh + vxc, en


def _vec(x):
    return torch.as_tensor(x, dtype=torch.float64, device="cuda")


def _exact_scf(h, psi, k0, k1):
    rho = h.density(psi)
    v, en = h.ks_potential(rho)
    save, psi = h.series(psi, k0, [0.5j * DT, 1j * DT], v)
    rho = h.density(psi)
    v, en = h.ks_potential(rho)
    for _ in range(5):
        psi = h.series(save, k1, [0.5j * DT], v)[0]
        new = h.density(psi)
        delta = h.dv * (new - rho).abs().sum()
        rho = new
        v, en = h.ks_potential(rho)
        if delta < 5e-5:
            break
    return dict(psi=psi, rho=rho, energies=en)


def _exact_cn(h, psi, k0, k1):
    rhs = psi - 0.5j * DT * h.apply(psi, k0)
    for _ in range(300):
        for _ in range(5):
            r = psi + 0.5j * DT * h.apply(psi, k1) - rhs
            w = r + 0.5j * DT * h.apply(r, k1)
            ca = h.dv * (w.abs() ** 2).sum(0)
            cb = 4 * h.dv * (r.conj() * w).sum(0).real
            cc = h.dv * (r.abs() ** 2).sum(0)
            disc = cb * cb - 4 * ca * cc
            sign = torch.where(cb * disc >= 0, 1.0, -1.0)
            root = torch.where(disc >= 0, disc.abs().sqrt() + 0j, -1j * disc.abs().sqrt())
            psi = psi + cc / (-0.5 * (cb + sign * root)) * r
        if cc.max() < 1e-10:
            return psi
    return psi


def _exact_mlwf(c, psi):
    """Centres and spreads at the joint-diagonality optimum next to the given states (their
    rotation is fixed only up to phases, so the states are not compared)."""
    edges = np.array([c["nx"], c["ny"], c["nz"]]) * c["spacing"]
    m = psi.shape[1]
    th = [torch.as_tensor(2 * np.pi * _sym(n) / n, device="cuda") for n in (c["nx"], c["ny"], c["nz"])]
    th = torch.stack(torch.meshgrid(*th, indexing="ij")).reshape(3, -1)
    psi = psi / psi.norm(dim=0)
    a = []
    for d in range(3):
        for w in (torch.cos(th[d]), torch.sin(th[d])):
            a.append((psi.conj().T @ (w[:, None] * psi)).cpu().numpy())
    a = np.array(a)
    even = m + m % 2
    ring = list(range(even))
    for _ in range(200):
        before = np.einsum("kii->ki", a).real.copy()
        for _ in range(even - 1):
            pq = [(ring[i], ring[even - 1 - i]) for i in range(even // 2)]
            p, q = (np.array([x[k] for x in pq if max(x) < m], int) for k in (0, 1))
            h = np.stack([a[:, p, p] - a[:, q, q], a[:, p, q] + a[:, q, p], 1j * (a[:, q, p] - a[:, p, q])], -1)
            g = np.einsum("kir,kis->irs", h, h.conj()).real
            v = np.linalg.eigh(g)[1][:, :, -1]
            x, y, z = (v * np.where(v[:, :1] < 0, -1, 1)).T
            co = np.sqrt((x + 1) / 2)
            s = (y - 1j * z) / (2 * co)
            ap, aq = a[:, p, :].copy(), a[:, q, :].copy()
            a[:, p, :], a[:, q, :] = (co[:, None] * ap + s.conj()[:, None] * aq, -s[:, None] * ap + co[:, None] * aq)
            ap, aq = a[:, :, p].copy(), a[:, :, q].copy()
            a[:, :, p], a[:, :, q] = co * ap + s * aq, -s.conj() * ap + co * aq
            ring = [ring[0], ring[-1]] + ring[1:-1]
        if np.abs(np.einsum("kii->ki", a).real - before).max() < 1e-13:
            break
    d = np.einsum("kii->ki", a).real
    centres = np.stack([np.arctan2(d[2 * k + 1], d[2 * k]) / (2 * np.pi) * edges[k] for k in range(3)], 1)
    spread2 = sum((1 - d[2 * k] ** 2 - d[2 * k + 1] ** 2) * (edges[k] / (2 * np.pi)) ** 2 for k in range(3))
    return dict(psi=None, centres=centres, spreads=np.sqrt(spread2))


def _exact_adjoint(c, h, psi, amplitudes):
    amps = _vec(amplitudes).requires_grad_()
    v = h.v.clone().requires_grad_()
    zero = torch.zeros(2, dtype=torch.float64, device="cuda")
    last = len(amplitudes) - 1
    for n in range(len(amplitudes)):
        psi = h.etrs(psi, torch.cat([amps[n:n + 1], zero]), torch.cat([amps[min(n + 1, last)][None], zero]), v)
    d = h.dipole(h.density(psi))[0]
    ga, gv = torch.autograd.grad(d, (amps, v))
    return dict(dipole=float(d.detach()), pulse=ga, potential=gv)


def exact(case, seed):
    c = case
    if c["op"] == "batch":
        return [exact(k, 1000 * seed + i) for i, k in enumerate(_cells(c))]
    s = _inputs(c, seed)
    psi = s["psi"].to(torch.complex128)
    if c["op"] == "mlwf":
        return _exact_mlwf(c, psi)
    if c["op"] == "ortho":
        u = torch.linalg.cholesky(c["spacing"] ** 3 * (psi.conj().T @ psi), upper=True)
        return torch.linalg.solve_triangular(u, psi, upper=True, left=False)
    # the backward pass of torch keeps every H application's intermediates
    if c["op"] == "adjoint" and psi.numel() * c["steps"] > 4e7:
        return None
    h = _Plain(c, s)
    k0, k1 = _vec(_pulse(c)(0.0)), _vec(_pulse(c)(DT))
    if c["op"] == "apply":
        return h.apply(psi, k0)
    if c["op"] == "propagate":
        out = h.etrs(psi, k0, k1)
        return dict(psi=out, energy=torch.stack([h.energy(psi, k0), h.energy(out, k1)]),
                    dipole=torch.stack([h.dipole(h.density(x)) for x in (psi, out)]))
    if c["op"] == "scf":
        return _exact_scf(h, psi, k0, k1)
    if c["op"] == "cn":
        return _exact_cn(h, psi, k0, k1)
    return _exact_adjoint(c, h, psi, s["amplitudes"])
