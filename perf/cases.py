"""The work that a user of mdpy_gb300 has it do, as cases that can be timed.

Every case goes through the package's public classes, on inputs made from a
seed.  The programs below keep single-precision frames, as mdpy itself does
(its arrays are float32 unless told otherwise), so positions, velocities and
forces are turned into float32 where they are read.

Kinds of programs (`kind`):

* ``md``     the main use: a Langevin or Verlet run between two reports, the
             frame taken over as device tensors on the program's own stream.
* ``log``    a `Simulation` with a `LogDumper`, the frame read as host arrays.
* ``batch``  many small systems of uneven size in one `EnsembleBatch`.
* ``forces`` single points: another program's frame in (host arrays), forces
             and energies out, as a re-scored trajectory or a Monte Carlo
             move does it.
* ``host``   a host-driven loop: each step's frame goes through pinned host
             memory (`mdg_step_host`), as a program with its own biases does.

What a system holds (`coulomb`): ``ewald`` flexible water with the Ewald sum
(LJ + erfc + PME + bonded), with `beads` a solvated chain too; ``bare`` the
terms of mdpy's own constraints (LJ and bare Coulomb over all pairs);
``none`` a Lennard-Jones fluid.
"""
import functools
import math

import numpy as np
import torch

from mdpy_gb300 import batch, constraint as C, systems, unit
from mdpy_gb300.ensemble import Ensemble
from mdpy_gb300.integrator import LangevinIntegrator, VerletIntegrator
from mdpy_gb300.simulation import LogDumper, Simulation
from mdpy_gb300.topology import Topology

EWALD_TOL = 1e-5
TEMPERATURE, FRICTION = 300.0, 1e-3

_BASE = {"kind": "md", "coulomb": "ewald", "atoms": 2700, "aspect": 1.0, "beads": 0, "cutoff": 12.0,
         "switch": 10.0, "order": 4, "integrator": "langevin", "dt": 1.0, "every": 1, "steps": 50}


def listed():
    return [dict(_BASE, **c) for c in (
        # the smallest water box of the tests and the survey (900 waters in
        # 30 A): launches and their order decide
        {"name": "md_2700"},
        # mdpy's own set of constraints on the same box: hard cutoff, bare
        # Coulomb over all pairs
        {"name": "md_bare_2700", "coulomb": "bare", "switch": 0.0, "steps": 10},
        # the benchmark's box: 30,000 waters and a 500-bead chain in 96.5 A
        {"name": "md_chain_88k", "atoms": 90500, "beads": 500},
        # the large box: 333,333 waters in about 215 A
        {"name": "md_1m", "atoms": 999999, "steps": 10},
        # boxes of 1.5k to 12k atoms, one batch
        {"name": "batch_40", "kind": "batch", "atoms": 12000, "boxes": 40, "cutoff": 10.0, "switch": 0.0,
         "steps": 20},
        # single points of a small box, the highest PME order
        {"name": "forces_2k", "kind": "forces", "atoms": 2103, "cutoff": 9.0, "switch": 0.0, "order": 6,
         "steps": 1},
        # single points of a middle-sized box that is no cube
        {"name": "forces_24k", "kind": "forces", "atoms": 24051, "aspect": 1.7, "order": 5, "steps": 1},
        # host-driven steps
        {"name": "host_24k", "kind": "host", "atoms": 24000, "steps": 10},
        # a Lennard-Jones fluid, constant energy
        {"name": "lj_20k", "coulomb": "none", "atoms": 20011, "integrator": "verlet", "dt": 2.0, "steps": 40},
        # a logged run: a row of energies every 10 steps
        {"name": "log_6k", "kind": "log", "atoms": 6003, "cutoff": 10.0, "switch": 8.0, "steps": 40},
        # multiple time steps: the reciprocal force every other step
        {"name": "mts_24k", "atoms": 24300, "cutoff": 10.0, "switch": 0.0, "order": 5, "every": 2, "steps": 20},
    )]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    c = dict(_BASE, cutoff=rng.choice([9.0, 10.0, 11.0, 12.0]), order=rng.choice([4, 4, 5, 6]),
             aspect=round(rng.uniform(1.0, 1.8), 3))
    c["switch"] = rng.choice([0.0, c["cutoff"] - 2.0])
    c["kind"] = rng.choice(["md", "md", "md", "md", "log", "batch", "forces", "forces", "host"])
    if c["kind"] == "md":
        c["coulomb"] = rng.choice(["ewald", "ewald", "ewald", "bare", "none"])
        c["atoms"] = size(2700, 8000 if c["coulomb"] == "bare" else 500000)
        c["integrator"] = rng.choice(["langevin", "langevin", "verlet"])
        if c["coulomb"] == "ewald":
            c["every"] = rng.choice([1, 1, 1, 2, 3])
            c["beads"] = rng.choice([0, 0, 200]) if 20000 < c["atoms"] < 120000 else 0
        if c["coulomb"] == "none":
            c["dt"] = 2.0
        if c["beads"]:
            c["aspect"] = 1.0
        c["steps"] = rng.randint(5, 10 if c["atoms"] > 120000 else 50)
    elif c["kind"] == "batch":
        c.update(atoms=size(3000, 12000), boxes=rng.randint(3, 40), cutoff=9.0, switch=0.0, aspect=1.0,
                 steps=rng.randint(5, 20))
    elif c["kind"] == "log":
        c.update(atoms=size(2700, 60000), steps=10 * rng.randint(2, 5))
    elif c["kind"] == "forces":
        c.update(atoms=size(2000, 200000), steps=1)
    else:
        c.update(atoms=size(2700, 60000), steps=rng.randint(3, 10))
    if c["kind"] != "batch" and c["atoms"] < 12000:
        c["aspect"] = min(c["aspect"], 1.2)  # the shortest edge stays above two cutoffs
        c["cutoff"] = min(c["cutoff"], 9.0) if c["atoms"] < 6000 else c["cutoff"]
        c["switch"] = min(c["switch"], c["cutoff"] - 1.0) if c["switch"] else 0.0
    return c


# ---- the inputs ----------------------------------------------------------------
class Box:
    """One system as plain arrays: what both `prepare` and `exact` start from."""


def water(rng, n_waters, edges, temperature=TEMPERATURE):
    """Flexible waters on a jittered lattice, randomly turned and a little bent
    (as `systems.water_box` sets them up, for any orthorhombic box)."""
    per = np.maximum(1, np.round(edges * (n_waters / np.prod(edges)) ** (1 / 3))).astype(int)
    while np.prod(per) < n_waters:
        per[np.argmax(edges / per)] += 1
    site = rng.permutation(int(np.prod(per)))[:n_waters]
    o = (np.stack(np.unravel_index(site, per), 1) + 0.5) * (edges / per) + rng.uniform(-0.3, 0.3, (n_waters, 3))
    half = math.radians(systems.WATER_THETA0_DEG) / 2
    a = rng.normal(size=(n_waters, 3))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    b = np.cross(a, rng.normal(size=(n_waters, 3)))
    b /= np.linalg.norm(b, axis=1, keepdims=True)
    h1 = systems.WATER_R0 * (math.sin(half) * a + math.cos(half) * b)
    h2 = systems.WATER_R0 * (-math.sin(half) * a + math.cos(half) * b)
    x = np.stack([o, o + h1, o + h2], 1).reshape(-1, 3) + rng.normal(0.0, 0.03, (3 * n_waters, 3))
    s = Box()
    s.edges, s.x = edges, x - edges * np.round(x / edges)
    s.types = ["OT", "HT", "HT"] * n_waters
    s.mass = np.tile([systems.O_MASS, systems.H_MASS, systems.H_MASS], n_waters)
    s.q = np.tile([systems.O_CHARGE, systems.H_CHARGE, systems.H_CHARGE], n_waters)
    base = 3 * np.arange(n_waters)
    s.bonds = np.stack([base, base + 1, base, base + 2], 1).reshape(-1, 2)
    s.angles = np.stack([base + 1, base, base + 2], 1)
    s.dihedrals, s.dprm = np.zeros((0, 4), int), np.zeros((0, 3))
    kcal = unit.KCAL_PER_MOL
    s.lj = {"OT": [systems.O_EPS_KCAL * kcal, systems.O_SIGMA], "HT": [0.0, 1.0]}
    s.bprm = np.tile([systems.BOND_K_KCAL * kcal, systems.WATER_R0], (2 * n_waters, 1))
    s.aprm = np.tile([systems.ANGLE_K_KCAL * kcal, math.radians(systems.WATER_THETA0_DEG), 0.0, 0.0], (n_waters, 1))
    s.partners = np.stack([base + 1, base + 2, base, base + 2, base, base + 1], 1).reshape(-1, 2)
    s.v = systems.maxwell_boltzmann(rng, s.mass, temperature)
    return s


def solvated_chain(case, rng):
    """One chain in water (the first of `systems.chain_in_water`: some of its
    later ones cross themselves), each atom displaced a little."""
    w = systems.chain_in_water((case["atoms"] - case["beads"]) // 3, box_edges(case)[0], case["beads"], seed=0)
    t, p, s = w.topology, w.parameters, Box()
    s.edges, s.types = w.box, t.particle_types
    s.x = w.positions + rng.normal(0.0, 0.03, w.positions.shape)
    s.v = systems.maxwell_boltzmann(rng, t.masses, TEMPERATURE)
    s.mass, s.q = t.masses.reshape(-1), t.charges.reshape(-1)
    s.bonds, s.angles, s.dihedrals, s.dprm = t.bonds, t.angles, t.dihedrals, w.dihedral_parameters
    s.lj = p["nonbonded"]
    first = s.bonds[:, 0] < case["beads"]
    s.bprm = np.where(first[:, None], p["bond"]["CB-CB"], p["bond"]["OT-HT"])
    first = s.angles[:, 0] < case["beads"]
    s.aprm = np.where(first[:, None], p["angle"]["CB-CB-CB"], p["angle"]["HT-OT-HT"])
    s.partners, s.topology = t.bonded_particles, t
    return s


def lj_fluid(rng, n, edges):
    """Argon-like atoms near a jittered lattice at 120 K."""
    per = np.maximum(1, np.ceil(edges * (n / np.prod(edges)) ** (1 / 3))).astype(int)
    site = rng.permutation(int(np.prod(per)))[:n]
    x = (np.stack(np.unravel_index(site, per), 1) + 0.5) * (edges / per) + rng.uniform(-0.2, 0.2, (n, 3))
    s = Box()
    s.edges, s.x = edges, x - edges * np.round(x / edges)
    s.types, s.mass, s.q = ["AR"] * n, np.full(n, 39.948), np.zeros(n)
    s.lj = {"AR": [0.238 * unit.KCAL_PER_MOL, 3.405]}
    s.bonds, s.angles, s.dihedrals = np.zeros((0, 2), int), np.zeros((0, 3), int), np.zeros((0, 4), int)
    s.bprm, s.aprm, s.dprm, s.partners = np.zeros((0, 2)), np.zeros((0, 4)), np.zeros((0, 3)), np.full((n, 1), -1)
    s.v = systems.maxwell_boltzmann(rng, s.mass, 120.0)
    return s


def box_edges(case):
    """Edges of the box: 0.1 atoms per cubic A (0.0208 for the Lennard-Jones
    fluid), the sides `aspect` apart."""
    a = case["aspect"]
    edge = (case["atoms"] / (0.0208 if case["coulomb"] == "none" else 0.1)) ** (1 / 3)
    if case["beads"]:
        edge = (case["atoms"] / 0.1007) ** (1 / 3)
    return edge * np.array([1.0 / a, 1.0, a]) ** 0.5


def grid_of(case, edges):
    """PME grid of about 1 A spacing (of the batch: clipped to 24 to 48)."""
    if case["kind"] == "batch":
        return [min(48, max(24, systems.fft_friendly(int(round(e))))) for e in edges]
    return [systems.fft_friendly(int(math.ceil(e))) for e in edges]


def boxes_of(case, seed):
    """The case's systems (one, but for a batch)."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        lo = min(1500, case["atoms"])
        counts = np.exp(np.random.default_rng(case["boxes"]).uniform(math.log(lo), math.log(case["atoms"]), case["boxes"]))
        cells = [max(case["cutoff"] * 2.02, (3 * round(n / 3) / 0.1) ** (1 / 3)) for n in counts]
        return [water(rng, max(int(0.1 * e ** 3 / 3), 1), np.full(3, e)) for e in cells]
    if case["coulomb"] == "none":
        return [lj_fluid(rng, case["atoms"], box_edges(case))]
    if case["beads"]:
        return [solvated_chain(case, rng)]
    return [water(rng, case["atoms"] // 3, box_edges(case))]


# ---- the programs --------------------------------------------------------------
def bind(case, s, make):
    """An ensemble with the case's constraints, positions and velocities."""
    t = getattr(s, "topology", None) or Topology.from_arrays(
        s.types, s.mass, s.q, bonds=s.bonds, angles=s.angles, dihedrals=s.dihedrals, bonded_particles=s.partners)
    ens = make(t, np.diag(s.edges))
    switch = case["switch"] or None
    if case["coulomb"] == "ewald":
        terms = [C.NonbondedConstraint(s.lj, case["cutoff"], switch, ewald_error=EWALD_TOL),
                 C.PMEConstraint(grid_of(case, s.edges), case["order"], EWALD_TOL, real_space_cutoff=case["cutoff"])]
    elif case["coulomb"] == "bare":
        terms = [C.CharmmNonbondedConstraint(s.lj, case["cutoff"], switch), C.ElectrostaticConstraint()]
    else:
        terms = [C.CharmmNonbondedConstraint(s.lj, case["cutoff"], switch)]
    if len(s.bonds):
        terms += [C.CharmmBondConstraint(None, float_parameters=s.bprm),
                  C.CharmmAngleConstraint(None, float_parameters=s.aprm)]
    if len(s.dihedrals):
        terms.append(C.CharmmDihedralConstraint(None, float_parameters=s.dprm))
    ens.add_constraints(*terms)
    if case["kind"] != "forces":
        ens.state.set_positions(s.x)
        ens.state.set_velocities(s.v)
    return ens


def temperature_of(case):
    return 120.0 if case["coulomb"] == "none" else TEMPERATURE


def prepare(case, seed):
    kind, boxes = case["kind"], boxes_of(case, seed)
    if kind == "batch":
        ens = batch.EnsembleBatch([bind(case, s, batch.member) for s in boxes], device=0)
    else:
        ens = bind(case, boxes[0], functools.partial(Ensemble, device=0))
    st = {"case": case, "ens": ens, "n": sum(len(s.x) for s in boxes)}
    if kind == "forces":
        st["frame"] = boxes[0].x
        return st
    if case["integrator"] == "langevin":
        st["integrator"] = LangevinIntegrator(case["dt"], temperature_of(case), FRICTION, seed=seed,
                                              reciprocal_every=case["every"])
    else:
        st["integrator"] = VerletIntegrator(case["dt"], reciprocal_every=case["every"])
    if kind in ("md", "batch"):
        st["stream"] = torch.cuda.Stream()
        ens.system.set_stream(st["stream"].cuda_stream)
        st["x"] = torch.empty(st["n"], 3, dtype=torch.float64, device="cuda")
        st["v"] = torch.empty_like(st["x"])
    elif kind == "log":
        st["simulation"] = Simulation(ens, st["integrator"])
        st["simulation"].add_dumpers(LogDumper(dump_frequency=10))
    else:  # host: the frames go back and forth between pinned buffers
        ens.system.integrator_config(1, case["dt"], TEMPERATURE, FRICTION, seed)
        st["frames"] = [[torch.empty(st["n"], 3, dtype=torch.float64, pin_memory=True) for _ in range(2)]
                        for _ in range(2)]
        st["frames"][0][0].copy_(torch.from_numpy(boxes[0].x))
        st["frames"][0][1].copy_(torch.from_numpy(boxes[0].v))
        st["energies"] = np.zeros(7)
    return st


def run(state):
    case, ens = state["case"], state["ens"]
    kind = case["kind"]
    if kind == "forces":
        ens.state.set_positions(state["frame"])
        ens.update()
        return {"f": ens.forces.astype(np.float32), "e": np.array(list(ens.energies.values()), np.float32)}
    if kind == "log":
        state["simulation"].integrate(case["steps"])
        return {"x": ens.state.positions.astype(np.float32), "v": ens.state.velocities.astype(np.float32),
                "e": [ens.potential_energy, ens.kinetic_energy]}
    if kind == "host":
        for _ in range(case["steps"]):
            (x, v), (x2, v2) = state["frames"]
            kinetic = ens.system.step_host_ptr(x.data_ptr(), v.data_ptr(), 1, ens.term_mask, x2.data_ptr(),
                                               v2.data_ptr(), state["energies"])
            state["frames"].reverse()
        return {"x": x2.float(), "v": v2.float(), "e": [float(state["energies"].sum()), kinetic]}
    with torch.cuda.stream(state["stream"]):
        state["integrator"].integrate(ens, case["steps"])
        ens.system.get_positions_ptr(state["x"].data_ptr())
        ens.system.get_velocities_ptr(state["v"].data_ptr())
        frame = {"x": state["x"].float(), "v": state["v"].float()}
    if kind == "batch":
        return dict(frame, e=ens.potential_energies.astype(np.float32), k=ens.kinetic_energies.astype(np.float32))
    return dict(frame, e=[ens.potential_energy, ens.kinetic_energy])


def work(case):
    """Pairs inside the cutoff at 60 operations each, the PME grid and the
    bonded terms, per force evaluation; frames once in and once out."""
    sizes = [case["atoms"]]
    if case["kind"] == "batch":  # log-uniform counts between 1,500 and `atoms`
        lo, hi = min(1500, case["atoms"]), case["atoms"]
        sizes = [(hi - lo) / math.log(hi / lo) if hi > lo else hi] * case["boxes"]
    flops = 0.0
    for n in sizes:
        rho = 0.0208 if case["coulomb"] == "none" else 0.1
        flops += n * rho * 2 / 3 * math.pi * case["cutoff"] ** 3 * (60 if case["coulomb"] == "ewald" else 30)
        if case["coulomb"] == "bare":
            flops += n * n / 2 * 25
        if case["coulomb"] == "ewald":
            k3 = n * 10 if case["kind"] != "batch" else min(n * 10, 48 ** 3)
            flops += n * 10 * case["order"] ** 3 + 2 * 2.5 * k3 * math.log2(k3) + 4 * k3
        flops += n * 60
    n = sum(sizes)
    return {"bytes": 96.0 * n, "flops": flops * case["steps"]}


# ---- the same in 64 bits -------------------------------------------------------
KCOUL = 1.0 / (4.0 * math.pi * (8.85418e-12 * 1.66053904e-27 / 1.602176634e-19 ** 2))
KB = 1.38064852e-23 / (1.66053904e-27 * 1e-20 / 1e-30)


class Exact:
    """One system's forces and steps in FP64 with plain torch."""

    SKIN = 1.0

    def __init__(self, case, s, first_atom=0):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.case, self.dev, self.n, self.first = case, dev, len(s.x), first_atom
        put = functools.partial(torch.as_tensor, device=dev)
        self.L = put(np.asarray(s.edges, float))
        self.x, self.v = put(s.x.copy()), put(s.v.copy())
        self.m, self.q = put(s.mass.astype(float)), put(s.q.astype(float))
        names = sorted(s.lj)
        kind = np.searchsorted(names, np.asarray(s.types))
        self.eps = put(np.array([s.lj[k][0] for k in names])[kind])
        self.sig = put(np.array([s.lj[k][1] for k in names])[kind])
        self.skip = put(s.partners.astype(np.int64))
        own = np.repeat(np.arange(self.n), s.partners.shape[1]), s.partners.reshape(-1)
        half = own[0] < own[1]
        self.excl = put(np.stack([own[0][half], own[1][half]], 1).astype(np.int64))
        self.bonds, self.angles, self.dihedrals = (put(np.asarray(v, np.int64)) for v in (s.bonds, s.angles, s.dihedrals))
        self.bprm, self.aprm, self.dprm = (put(np.asarray(v, float)) for v in (s.bprm, s.aprm, s.dprm))
        self.beta = math.sqrt(-math.log(2 * EWALD_TOL)) / case["cutoff"]
        self.K = grid_of(case, s.edges)
        self.built = None

    def near(self, d):
        return d - self.L * torch.round(d / self.L)

    # pairs i < j within cutoff + skin, none of them excluded
    def pairs(self):
        if self.built is not None and float(self.near(self.x - self.built).norm(dim=1).max()) < 0.5 * self.SKIN:
            return self.list
        r = self.case["cutoff"] + self.SKIN
        x = self.x - self.L * torch.floor(self.x / self.L)
        nc = torch.clamp((self.L / r).floor().long(), min=1)
        found = []
        if int(nc.min()) < 3:
            rows = max(1, 40_000_000 // self.n)
            for lo in range(0, self.n, rows):
                d2 = sum((lambda d, e: d - e * torch.round(d / e))(x[lo:lo + rows, None, k] - x[None, :, k], self.L[k]) ** 2
                         for k in range(3))
                i, j = torch.nonzero(d2 < r * r, as_tuple=True)
                found.append(self.ordered(i + lo, j))
        else:
            c = torch.minimum((x / self.L * nc).long(), nc - 1)
            cell = (c[:, 0] * nc[1] + c[:, 1]) * nc[2] + c[:, 2]
            total = int(nc.prod())
            order = torch.argsort(cell)
            count = torch.bincount(cell, minlength=total)
            start, most = torch.cumsum(count, 0) - count, int(count.max())
            slot = torch.arange(self.n, device=self.dev) - start[cell[order]]
            table = torch.full((total, most), -1, dtype=torch.int64, device=self.dev)
            table[cell[order], slot] = order
            at = torch.arange(total, device=self.dev)
            at = torch.stack([at // (nc[1] * nc[2]), at // nc[2] % nc[1], at % nc[2]], 1)
            for code in range(14):  # the cell itself and half of its neighbours
                step = torch.tensor([code // 9, code // 3 % 3, code % 3], device=self.dev) - 1
                to = (at + step) % nc
                to = (to[:, 0] * nc[1] + to[:, 1]) * nc[2] + to[:, 2]
                rows = max(1, 100_000_000 // most ** 2)
                for lo in range(0, total, rows):
                    i, j = table[lo:lo + rows, :, None], table[to[lo:lo + rows]][:, None, :]
                    d = x[i.clamp(min=0)].float() - x[j.clamp(min=0)].float()
                    d = d - (self.L * torch.round(d / self.L)).float()
                    hit = (d.square().sum(-1) < r * r + 0.01) & (i >= 0) & (j >= 0)
                    a, b, e = torch.nonzero(hit, as_tuple=True)
                    i, j = table[a + lo, b], table[to[a + lo], e]
                    found.append(self.ordered(i, j) if code == 13 else self.ordered(torch.minimum(i, j), torch.maximum(i, j)))
        self.list, self.built = torch.cat(found, 1), self.x.clone()
        return self.list

    def ordered(self, i, j):
        keep = (i < j) & (self.skip[i] != j[:, None]).all(1)
        return torch.stack([i[keep], j[keep]])

    def short_range(self, f):
        case, rc = self.case, self.case["cutoff"]
        e_lj = e_c = 0.0
        listed_ = self.pairs()
        for lo in range(0, listed_.shape[1], 50_000_000):
            i, j = listed_[0, lo:lo + 50_000_000], listed_[1, lo:lo + 50_000_000]
            d = self.near(self.x[j] - self.x[i])
            r2 = d.square().sum(1)
            keep = r2 <= rc * rc
            i, j, d, r2 = i[keep], j[keep], d[keep], r2[keep]
            c = 4 * torch.sqrt(self.eps[i] * self.eps[j])
            s6 = ((0.5 * (self.sig[i] + self.sig[j])) ** 2 / r2) ** 3
            e, fr = c * s6 * (s6 - 1), c * s6 * (12 * s6 - 6) / r2
            if case["switch"]:
                rs2, rc2 = case["switch"] ** 2, rc * rc
                rr = torch.clamp(r2, min=rs2)
                sw = (rc2 - rr) ** 2 * (rc2 + 2 * rr - 3 * rs2) / (rc2 - rs2) ** 3
                dsw = 12 * (rc2 - rr) * (rs2 - rr) / (rc2 - rs2) ** 3
                fr, e = fr * sw - e * dsw, e * sw
            e_lj += float(e.sum())
            if case["coulomb"] == "ewald":
                r, qq = r2.sqrt(), KCOUL * self.q[i] * self.q[j]
                e = qq * torch.erfc(self.beta * r) / r
                fr = fr + (e + qq * 2 * self.beta / math.sqrt(math.pi) * torch.exp(-self.beta ** 2 * r2)) / r2
                e_c += float(e.sum())
            w = fr[:, None] * d
            f.index_add_(0, j, w)
            f.index_add_(0, i, -w)
        return e_lj, e_c

    def bare(self, f):
        total, rows = 0.0, max(1, 20_000_000 // self.n)
        skip = torch.zeros(self.n, self.n, dtype=torch.bool, device=self.dev)
        skip[self.excl[:, 0], self.excl[:, 1]] = True
        skip |= skip.T.clone()
        skip.fill_diagonal_(True)
        for lo in range(0, self.n, rows):
            d = self.near(self.x[None] - self.x[lo:lo + rows, None])
            r2 = d.square().sum(-1).masked_fill(skip[lo:lo + rows], math.inf)
            e = KCOUL * self.q[lo:lo + rows, None] * self.q[None] / r2.sqrt()
            total += 0.5 * float(e.sum())
            f[lo:lo + rows] -= ((e / r2)[..., None] * d).sum(1)
        return total

    # B-spline weights of the `order` points that a coordinate touches
    def spline(self, w):
        a, da = [1 - w, w], None
        for n in range(3, self.case["order"] + 1):
            if n == self.case["order"]:
                da = [-a[0]] + [a[k - 1] - a[k] for k in range(1, n - 1)] + [a[n - 2]]
            a = [((w + n - 1 - k) * (a[k - 1] if k else 0) + (k + 1 - w) * (a[k] if k < n - 1 else 0)) / (n - 1)
                 for k in range(n)]
        return torch.stack(a, -1), torch.stack(da, -1)

    def modulus(self, K):
        p = self.case["order"]
        th = self.spline(torch.zeros(1, dtype=torch.float64))[0][0].numpy()
        k = np.arange(p - 1)
        b = np.abs((th[p - 2 - k] * np.exp(2j * np.pi * np.outer(np.arange(K), k) / K)).sum(1)) ** 2
        return np.where(b < 1e-10, 0.5 * (np.roll(b, 1) + np.roll(b, -1)), b)

    def reciprocal(self, f):
        """PME on the case's own grid and order, self, net charge and the
        excluded pairs."""
        if not hasattr(self, "G"):
            m = [np.fft.fftfreq(K, 1.0 / K) / float(e) for K, e in zip(self.K, self.L)]
            m[2] = np.arange(self.K[2] // 2 + 1) / float(self.L[2])
            m2 = m[0][:, None, None] ** 2 + m[1][None, :, None] ** 2 + m[2][None, None] ** 2
            b = [self.modulus(K) for K in self.K]
            m2[0, 0, 0] = 1.0
            G = np.exp(-np.pi ** 2 * m2 / self.beta ** 2) / (np.pi * float(self.L.prod()) * m2)
            G /= b[0][:, None, None] * b[1][None, :, None] * b[2][None, None, :len(m[2])]
            G[0, 0, 0] = 0.0
            self.G = torch.as_tensor(G, device=self.dev)
        p, K = self.case["order"], torch.tensor(self.K, device=self.dev)
        u = (self.x - self.L * torch.floor(self.x / self.L)) / self.L * K
        c = torch.minimum(u.long(), K - 1)
        th, dth = self.spline(u - c)
        at = (c[..., None] - p + 1 + torch.arange(p, device=self.dev)) % K[:, None]
        idx = ((at[:, 0, :, None, None] * K[1] + at[:, 1, None, :, None]) * K[2] + at[:, 2, None, None, :]).reshape(self.n, -1)

        def outer(a, b, d):
            return (a[:, :, None, None] * b[:, None, :, None] * d[:, None, None, :]).reshape(self.n, -1)

        grid = torch.zeros(int(K.prod()), dtype=torch.float64, device=self.dev)
        grid.index_add_(0, idx.reshape(-1), (self.q[:, None] * outer(th[:, 0], th[:, 1], th[:, 2])).reshape(-1))
        F = torch.fft.rfftn(grid.reshape(self.K))
        wgt = torch.full((self.G.shape[2],), 2.0, dtype=torch.float64, device=self.dev)
        wgt[0] = 1.0
        if self.K[2] % 2 == 0:
            wgt[-1] = 1.0
        e = 0.5 * KCOUL * float((wgt * self.G * (F.real ** 2 + F.imag ** 2)).sum())
        phi = torch.fft.irfftn(F * self.G, s=self.K, norm="forward").reshape(-1)[idx]
        for k in range(3):
            w = [th[:, a] if a != k else dth[:, a] for a in range(3)]
            f[:, k] -= KCOUL * self.q * (outer(*w) * phi).sum(1) * (self.K[k] / self.L[k])
        e -= KCOUL * self.beta / math.sqrt(math.pi) * float(self.q.square().sum())
        e -= KCOUL * math.pi * float(self.q.sum()) ** 2 / (2 * self.beta ** 2 * float(self.L.prod()))
        i, j = self.excl[:, 0], self.excl[:, 1]
        d = self.near(self.x[j] - self.x[i])
        r = d.norm(dim=1)
        qq = KCOUL * self.q[i] * self.q[j]
        ex = -qq * torch.erf(self.beta * r) / r
        fr = (ex + qq * 2 * self.beta / math.sqrt(math.pi) * torch.exp(-(self.beta * r) ** 2)) / r ** 2
        f.index_add_(0, j, fr[:, None] * d)
        f.index_add_(0, i, -fr[:, None] * d)
        return e + float(ex.sum())

    def bonded(self, f):
        e = [0.0, 0.0, 0.0]
        with torch.enable_grad():
            for k, (idx, prm) in enumerate(((self.bonds, self.bprm), (self.angles, self.aprm), (self.dihedrals, self.dprm))):
                if not len(idx):
                    continue
                x = self.x[idx].detach().requires_grad_(True)
                if k == 0:
                    r = self.near(x[:, 1] - x[:, 0]).norm(dim=1)
                    v = prm[:, 0] * (r - prm[:, 1]) ** 2
                elif k == 1:
                    a, b = self.near(x[:, 0] - x[:, 1]), self.near(x[:, 2] - x[:, 1])
                    v = prm[:, 0] * (torch.acos((a * b).sum(1) / a.norm(dim=1) / b.norm(dim=1)) - prm[:, 1]) ** 2
                else:
                    b1, b2, b3 = (self.near(x[:, t + 1] - x[:, t]) for t in range(3))
                    m, n = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
                    phi = torch.atan2(b2.norm(dim=1) * (b1 * n).sum(1), (m * n).sum(1))
                    v = prm[:, 0] * (1 + torch.cos(prm[:, 1] * phi - prm[:, 2]))
                v = v.sum()
                (g,) = torch.autograd.grad(v, x)
                f.index_add_(0, idx.reshape(-1), -g.reshape(-1, 3))
                e[k] = float(v.detach())
        return e

    def forces(self, slow=1.0):
        """Forces with the reciprocal part weighted by `slow`, and the seven
        energies."""
        f = torch.zeros_like(self.x)
        e = [0.0] * 7
        e[0], e[1] = self.short_range(f)
        if self.case["coulomb"] == "ewald":
            g = torch.zeros_like(f)
            e[2] = self.reciprocal(g)
            f += slow * g
        elif self.case["coulomb"] == "bare":
            e[1] = self.bare(f)
        e[3:6] = self.bonded(f)
        return f, e

    # Philox4x32-10 (Salmon et al. 2011) and Box-Muller: the thermostat's
    # noise of each atom and step
    def noise(self, step, seed):
        m32 = 0xFFFFFFFF
        atom = torch.arange(self.first, self.first + self.n, device=self.dev)
        c = [atom, torch.full_like(atom, step & m32), torch.full_like(atom, step >> 32), torch.full_like(atom, 0x4C414E47)]
        k = [seed & m32, seed >> 32 & m32]
        for _ in range(10):
            prod = []
            for mult, v in ((0xD2511F53, c[0]), (0xCD9E8D57, c[2])):
                lo = mult * (v & 0xFFFF)
                hi = mult * (v >> 16) + (lo >> 16)
                prod.append((hi >> 16, (hi & 0xFFFF) << 16 | lo & 0xFFFF))
            c = [prod[1][0] ^ c[1] ^ k[0], prod[1][1], prod[0][0] ^ c[3] ^ k[1], prod[0][1]]
            k = [(k[0] + 0x9E3779B9) & m32, (k[1] + 0xBB67AE85) & m32]
        u = [((v >> 8).double() + 0.5) / 2 ** 24 for v in c]
        r0, r1 = torch.sqrt(-2 * torch.log(u[0])), torch.sqrt(-2 * torch.log(u[2]))
        return torch.stack([r0 * torch.cos(2 * math.pi * u[1]), r0 * torch.sin(2 * math.pi * u[1]),
                            r1 * torch.cos(2 * math.pi * u[3])], 1)

    def steps(self, seed):
        """The case's steps: Groenbech-Jensen--Farago Langevin or velocity
        Verlet, the reciprocal force every `every` steps.  The energies are
        the last step's."""
        case, dt, k = self.case, self.case["dt"], self.case["every"]
        g = FRICTION if case["integrator"] == "langevin" else 0.0
        a, b = (1 - 0.5 * g * dt) / (1 + 0.5 * g * dt), 1 / (1 + 0.5 * g * dt)
        m = self.m[:, None]
        f, _ = self.forces(k)
        for n in range(case["steps"]):
            h = 0.5 * dt / m
            beta = torch.zeros_like(f)
            if g:
                beta = torch.sqrt(2 * g * KB * temperature_of(case) * dt * m) * self.noise(n, seed)
            x = self.x + b * (dt * (self.v + h * f) + h * beta)
            v = a * self.v + a * h * f + b / m * beta
            self.x = x
            f, e = self.forces(k if (n + 1) % k == 0 else 0.0)
            self.v = v + h * f
        return e, float(0.5 * (m * self.v ** 2).sum())


def exact(case, seed):
    boxes, first, got = boxes_of(case, seed), 0, []
    with torch.no_grad():
        for s in boxes:
            w = Exact(case, s, first)
            first += w.n
            if case["kind"] == "forces":
                f, e = w.forces()
                return {"f": f.cpu().numpy(), "e": np.array(e)}
            e, kinetic = w.steps(seed)
            got.append((w.near(w.x).cpu(), w.v.cpu(), sum(e), kinetic))
    frame = {"x": torch.cat([g[0] for g in got]).numpy(), "v": torch.cat([g[1] for g in got]).numpy()}
    if case["kind"] == "batch":
        return dict(frame, e=np.array([g[2] for g in got]), k=np.array([g[3] for g in got]))
    return dict(frame, e=[got[0][2], got[0][3]])
