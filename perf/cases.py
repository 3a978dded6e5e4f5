"""The work this framework does, as cases that can be timed and compared.

Three paths, each through the public Python API (`apocharmm_b200.api`):

  forces  one evaluation at new host coordinates: `CharmmContext.setCoordinates`
          (which builds the neighbour list), `calculateForces` with energies and,
          in some cases, the virial, then forces, energies and virial read back;
          what minimisers, restraint scans, energy requests of a server and
          machine-learning loops do
  md      `CudaIntegrator.propagate` of a run that goes on from pass to pass, with
          coordinates and velocities read back after every pass, as a program that
          samples a trajectory does; a pass is one or more list periods of 20 steps
  batch   `Batch.propagate` of many independent systems at once

Systems are TIP3P water and bead chains in water at the density of the package's
own workloads, cutoffs, grids and spline orders as in its configurations and tests.
They are built from a small periodic cell, relaxed here in 64 bits, that is repeated,
shifted as a whole by a random vector, and shaken a little, molecule by molecule;
some waters are left out so that the counts are not round.

The checker (`exact`) restates the force field in 64-bit torch arithmetic: every
pair of atoms for the direct space, autograd for the bonded terms and for the charge
spreading of the reciprocal space.
"""
import dataclasses
import math
import os
import tempfile
import warnings

import numpy as np
import torch

from apocharmm_b200 import api, systems

DENSITY = 0.1003        # atoms per cubic Angstrom of the package's water boxes
KAPPA = 0.34
TIMFAC = 0.0488882129   # AKMA time unit in ps
KBOLTZ = 1.987191e-3
CCELEC = 332.0716
ENERGIES = ("bond", "angle", "ureyb", "dihe", "imdihe", "ewks", "ewse", "ewex", "elec", "vdw")


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest call: a few hundred atoms, bound by launches and copies
        dict(name="forces_water648", path="forces", kind="water", tile=216, tx=1, ty=1, tz=1, drop=0,
             roff=8.0, ron=7.0, rlist=9.0, order=4, spacing=1.0, precise=False, virial=False),
        # an ordinary water box (the size and cutoffs of the 12,480-atom workload)
        dict(name="forces_water12k", path="forces", kind="water", tile=521, tx=2, ty=2, tz=2, drop=8,
             roff=10.0, ron=8.0, rlist=12.0, order=4, spacing=1.05, precise=False, virial=False),
        # a solvated chain with 1-4 pairs, long cutoff, high spline order and the virial
        dict(name="forces_virial_chain24k", path="forces", kind="chain", tile=2960, tx=2, ty=2, tz=2, drop=41,
             roff=12.0, ron=10.0, rlist=14.0, order=6, spacing=1.0, precise=False, virial=True),
        # the precise form (every pair in 64-bit fixed point), order 8, an elongated box
        dict(name="forces_precise_ortho14k", path="forces", kind="chain", tile=2415, tx=1, ty=2, tz=3, drop=17,
             roff=11.0, ron=9.0, rlist=13.0, order=8, spacing=0.9, precise=True, virial=True),
        # a small solute box under the Langevin thermostat: launch-bound steps
        dict(name="langevin_chain3k", path="md", kind="chain", tile=3030, tx=1, ty=1, tz=1, drop=5,
             roff=10.0, ron=8.0, rlist=12.0, order=4, spacing=1.0, precise=False,
             integrator="langevin", dt=0.002, steps=40),
        # the headline workload's size and settings: chain in water, PME 64^3 order 6, Langevin
        dict(name="langevin_chain24k", path="md", kind="chain", tile=2960, tx=2, ty=2, tz=2, drop=41,
             roff=12.0, ron=10.0, rlist=14.0, order=6, spacing=1.0, precise=False,
             integrator="langevin", dt=0.002, steps=40),
        # constant energy, flexible water, plain leapfrog
        dict(name="leapfrog_water12k", path="md", kind="water", tile=521, tx=2, ty=2, tz=2, drop=8,
             roff=10.0, ron=8.0, rlist=12.0, order=4, spacing=1.05, precise=False,
             integrator="leapfrog", dt=0.0005, steps=40),
        # constant pressure: energy and virial every step, the box moves
        dict(name="piston_chain24k", path="md", kind="chain", tile=2960, tx=2, ty=2, tz=2, drop=41,
             roff=12.0, ron=10.0, rlist=14.0, order=6, spacing=1.0, precise=False,
             integrator="piston", dt=0.002, steps=40),
        # a large protein-sized box in an elongated cell, Nose-Hoover
        dict(name="nose_hoover_chain107k", path="md", kind="chain", tile=2980, tx=3, ty=3, tz=4, drop=59,
             roff=10.0, ron=8.0, rlist=12.0, order=6, spacing=1.0, precise=False,
             integrator="nose_hoover", dt=0.002, steps=40),
        # the largest: a million atoms, PME 216^3 order 4, list radius 11.5
        dict(name="nose_hoover_water998k", path="md", kind="water", tile=333, tx=10, ty=10, tz=10, drop=301,
             roff=10.0, ron=8.0, rlist=11.5, order=4, spacing=1.0, precise=False,
             integrator="nose_hoover", dt=0.002, steps=20),
        # many systems of 3,000 to 24,000 atoms advanced together
        dict(name="batch24", path="batch", kind="chain", systems=24, tile_lo=2990, tile_hi=3060, copies=8,
             drop=7, roff=10.0, ron=8.0, rlist=12.0, order=4, spacing=1.0, precise=False,
             dt=0.002, steps=20),
    ]


def draw(rng):
    """One more case: sizes log-uniform from a few hundred to about 200,000 atoms,
    any box shape of up to 5 cells an edge, every order, form and integrator."""
    path = rng.choice(["forces", "forces", "md", "md", "md", "batch"])
    order = rng.choice([4, 4, 6, 8])
    spacing = round(rng.uniform(0.85, 1.1), 3)
    if path == "batch":
        lo = rng.randrange(2700, 3000)
        return dict(path="batch", kind="chain", systems=rng.randrange(3, 25), tile_lo=lo,
                    tile_hi=lo + rng.randrange(1, 90), copies=rng.choice([1, 2, 4, 8]),
                    drop=rng.randrange(0, 40), roff=10.0, ron=8.0, rlist=12.0, order=order,
                    spacing=spacing, precise=False, dt=0.002, steps=20)
    kind = rng.choice(["water", "chain"])
    # atoms of one cell: its edge is at least twice the list radius
    tile = rng.randrange(205, 700) if kind == "water" else rng.randrange(2300, 3300)
    atoms = 3 * tile if kind == "water" else tile
    copies = max(1.0, math.exp(rng.uniform(math.log(atoms), math.log(2.0e5))) / atoms)
    t = [1, 1, 1]
    while t[0] * t[1] * t[2] < copies and min(t) < 5:
        k = rng.choice([k for k in range(3) if t[k] < 5])
        t[k] += 1
    # the smallest grid a cell may need holds the cutoffs of its edge
    half = 0.5 * (atoms / DENSITY) ** (1.0 / 3.0)
    rlist = round(min(14.0, half - 0.15, rng.uniform(9.0, 14.0)), 2)
    roff = round(rlist - rng.uniform(1.0, 2.0), 2)
    c = dict(path=path, kind=kind, tile=tile, tx=t[0], ty=t[1], tz=t[2], drop=rng.randrange(0, 40),
             roff=roff, ron=round(roff - rng.uniform(1.0, 2.0), 2), rlist=rlist, order=order,
             spacing=spacing, precise=rng.random() < 0.25)
    if path == "forces":
        c["virial"] = rng.random() < 0.5
    else:
        c["integrator"] = rng.choice(["langevin", "nose_hoover", "piston", "leapfrog"])
        if c["integrator"] == "piston":  # the box finds its density: room for the list radius
            c["rlist"] = round(min(rlist, 0.88 * half), 2)
            c["roff"], c["ron"] = round(c["rlist"] - 1.5, 2), round(c["rlist"] - 2.5, 2)
        c["dt"] = 0.0005 if c["integrator"] == "leapfrog" else 0.002
        c["steps"] = rng.choice([20, 40])
    return c


# ---------------------------------------------------------------- systems

def _cell(kind, size):
    """(System, edge) of one relaxed periodic cell: `size` waters, or a chain of
    a tenth of `size` atoms in water; made once per process."""
    key = (kind, size)
    if key not in _cell.made:
        if kind == "water":
            L = (3 * size / DENSITY) ** (1.0 / 3.0)
            s = systems.water_box(size, L, seed=17, name="cell")
        else:
            beads = _beads(size)
            L = (size / DENSITY) ** (1.0 / 3.0)
            s = systems.solvated_chain(n_atoms=size, L=L, n_beads=beads, seed=23, name="cell")
        cut = min(9.0, 0.5 * L - 0.1)
        f = _Field(s, (L, L, L), cut, cut - 1.0, None, 0, _beads(size) if kind == "chain" else 0)
        x = torch.tensor(s.pos, dtype=torch.float64, device=f.device)
        was = torch.are_deterministic_algorithms_enabled(), torch.is_deterministic_algorithms_warn_only_enabled()
        torch.use_deterministic_algorithms(True, warn_only=True)  # the same cell in every process
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            for _ in range(200):  # steepest descent, the largest move 0.03 A
                g = f.bonded(x)[0] + f.pairs14(x)[0] + f.direct(x)[0]
                x = x - (0.03 / float(g.abs().max())) * g
        torch.use_deterministic_algorithms(was[0], warn_only=was[1])
        x = np.round(x.cpu().numpy(), 5)
        waters = api.water_indices(s)
        s.pos = np.round(api.rigid_water_fit(x, waters), 8)
        _cell.made[key] = (s, L)
    return _cell.made[key]


_cell.made = {}


def _beads(size):
    b = max(30, int(round(0.1 * size)))
    return b + (size - b) % 3


def _repeat(kind, size, t, drop):
    """The cell repeated t times with `drop` waters left out (a System whose
    positions are the unshifted ones, the box, beads per chain, chains)."""
    key = (kind, size, tuple(t), drop)
    if key not in _repeat.made:
        s, L = _cell(kind, size)
        beads = _beads(size) if kind == "chain" else 0
        nt = t[0] * t[1] * t[2]
        shifts = np.array([[(i + 0.5) * L - 0.5 * t[0] * L, (j + 0.5) * L - 0.5 * t[1] * L,
                            (k + 0.5) * L - 0.5 * t[2] * L]
                           for i in range(t[0]) for j in range(t[1]) for k in range(t[2])])
        chains = (s.pos[None, :beads] + shifts[:, None]).reshape(-1, 3)
        waters = (s.pos[None, beads:] + shifts[:, None]).reshape(-1, 3, 3)
        keep = np.sort(np.random.default_rng(size + 7 * nt).permutation(len(waters))[drop:])
        waters = waters[keep].reshape(-1, 3)
        nw = len(keep)
        nb = nt * beads
        off = beads * np.arange(nt)[:, None, None]
        wb, wa, wt, wn, wr, wi, ws = systems._water_topology(nw, first_atom=nb)
        k = np.arange(beads)

        def rows(width):
            if beads < width:
                return np.zeros((0, width), np.int64)
            one = np.stack([k[i:beads - width + 1 + i] for i in range(width)], 1)
            return (one[None] + off).reshape(-1, width)

        big = dataclasses.replace(
            s, name="sys", box=tuple(float(n * L) for n in t),
            pos=np.concatenate([chains, waters]),
            charge=np.concatenate([np.tile(s.charge[:beads], nt), np.tile(s.charge[beads:beads + 3], nw)]),
            mass=np.concatenate([np.tile(s.mass[:beads], nt), np.tile(s.mass[beads:beads + 3], nw)]),
            atom_type=s.atom_type[:beads] * nt + wt, atom_name=s.atom_name[:beads] * nt + wn,
            res_name=s.res_name[:beads] * nt + wr, res_id=s.res_id[:beads] * nt + wi,
            seg_id=s.seg_id[:beads] * nt + ws,
            bonds=np.concatenate([rows(2), wb]).astype(np.int64),
            angles=np.concatenate([rows(3), wa]).astype(np.int64),
            dihedrals=rows(4).astype(np.int64))
        with tempfile.TemporaryDirectory() as d:
            systems.write_psf(big, os.path.join(d, "s.psf"))
            systems.write_prm(big, os.path.join(d, "s.prm"))
            psf = api.CharmmPsf(os.path.join(d, "s.psf"))
            prm = api.CharmmParameters(os.path.join(d, "s.prm"))
        _repeat.made[key] = (big, beads, nt, psf, prm)
    return _repeat.made[key]


_repeat.made = {}


def _inputs(big, beads, chains, seed):
    """Coordinates and velocities (A, AKMA) of one seed: the system moved as a whole
    by a random vector, its molecules back in the box and shaken by 0.02 A, and
    velocities of 300 K without a drift."""
    rng = np.random.default_rng(seed)
    box = np.array(big.box)
    nb = beads * chains
    x = big.pos + (rng.random(3) - 0.5) * box
    c = x[:nb].reshape(chains, -1, 3) if beads else x[:0].reshape(0, 1, 3)
    w = x[nb:].reshape(-1, 3, 3)

    def settled(m):
        m = m - box * np.round(m.mean(1, keepdims=True) / box)
        return (m + rng.normal(0.0, 0.02, (len(m), 1, 3))).reshape(-1, 3)

    x = np.concatenate([settled(c), settled(w)])
    v = rng.normal(size=x.shape) * np.sqrt(KBOLTZ * 300.0 / big.mass)[:, None]
    v -= (big.mass[:, None] * v).sum(0) / big.mass.sum()
    return np.ascontiguousarray(x), np.ascontiguousarray(v)


def _grid(case, box):
    """Grid points an axis: the spacing asked for, sizes the transforms take."""
    return tuple(systems.fft_friendly(max(16, int(math.ceil(b / case["spacing"] - 1e-9)))) for b in box)


def _batch_members(case):
    """(cell size, copies) of every system of a batch: both spread over their range."""
    rng = np.random.default_rng(1000 * case["systems"] + case["tile_lo"])
    sizes = np.linspace(case["tile_lo"], case["tile_hi"], 4).astype(int)
    shapes = [t for t in ((1, 1, 1), (1, 1, 2), (1, 2, 2), (2, 2, 2)) if np.prod(t) <= case["copies"]]
    return [(int(rng.choice(sizes)), shapes[int(rng.integers(len(shapes)))]) for _ in range(case["systems"])]


# ---------------------------------------------------------------- prepare and run

def prepare(case, seed):
    if case["path"] == "batch":
        b = api.Batch(case["order"], 8, case["precise"])
        xs, vs = [], []
        for k, (size, t) in enumerate(_batch_members(case)):
            big, beads, chains, psf, prm = _repeat("chain", size, t, case["drop"])
            b.addSystem(psf, prm, big.box, KAPPA, case["rlist"], case["ron"], case["roff"],
                        _grid(case, big.box), seed=seed % 1000003 + k)
            x, v = _inputs(big, beads, chains, seed + 31 * k)
            xs.append(x)
            vs.append(v)
        b.initialize()
        b.setCoordinates(-1, np.concatenate(xs))
        b.setVelocities(-1, np.concatenate(vs))
        b.setLangevin(case["dt"], 1.0, 300.0, seed % 1000003)
        return dict(path="batch", batch=b, steps=case["steps"])
    big, beads, chains, psf, prm = _repeat(case["kind"], case["tile"],
                                           (case["tx"], case["ty"], case["tz"]), case["drop"])
    x, v = _inputs(big, beads, chains, seed)
    fm = api.ForceManager(psf, prm)
    fm.setBoxDimensions(big.box)
    fm.setKappa(KAPPA)
    fm.setCutoff(case["rlist"])
    fm.setCtonnb(case["ron"])
    fm.setCtofnb(case["roff"])
    fm.setFFTGrid(*_grid(case, big.box))
    fm.setPmeSplineOrder(case["order"])
    fm.setPrecisionMode(case["precise"])
    ctx = api.CharmmContext(fm)
    ctx.setCoordinates(x)
    # such a program has evaluated before (it looked at its starting energies): the
    # list and its buffers have their sizes
    ctx.calculateForces(False, True, case.get("virial", False))
    if case["path"] == "forces":
        return dict(path="forces", ctx=ctx, fm=fm, x=x, virial=case["virial"])
    how = case["integrator"]
    if how == "leapfrog":
        ctx.useHolonomicConstraints(False)
    ctx.setVelocities(v)
    if how == "langevin":
        it = api.CudaLangevinThermostatIntegrator(case["dt"])
        it.setThermostatFriction(1.0)
        it.setReferenceTemperature(300.0)
        it.setThermostatRngSeed(seed % 1000003)
    elif how == "nose_hoover":
        it = api.CudaNoseHooverIntegrator(case["dt"])
        it.setReferenceTemperature(300.0)
    elif how == "piston":
        it = api.CudaLangevinPistonIntegrator(case["dt"])
        it.setCrystalType(api.CudaLangevinPistonIntegrator.CUBIC if len(set(big.box)) == 1
                          else api.CudaLangevinPistonIntegrator.ORTHORHOMBIC)
        it.setReferenceTemperature(300.0)
        it.setPressure(np.diag([1.0, 1.0, 1.0]))
        it.setLangevinPistonFriction(20.0)
        it.setLangevinPistonFrictionSeed(seed % 1000003)
    else:
        it = api.CudaLeapFrogIntegrator(case["dt"])
    it.setCharmmContext(ctx)
    return dict(path="md", ctx=ctx, fm=fm, it=it, steps=case["steps"], piston=how == "piston")


def run(state):
    if state["path"] == "batch":
        b = state["batch"]
        b.propagate(state["steps"])
        return dict(coordinates=b.getCoordinates(-1), velocities=b.getVelocities(-1))
    ctx = state["ctx"]
    if state["path"] == "forces":
        ctx.setCoordinates(state["x"])
        ctx.calculateForces(False, True, state["virial"])
        e = ctx.getEnergyComponents()
        out = dict(forces=ctx.getForces(), energies=np.array([e[k] for k in ENERGIES]))
        if state["virial"]:
            out["virial"] = ctx.getVirial()
        return out
    state["it"].propagate(state["steps"])
    out = dict(coordinates=ctx.getCoordinates(), velocities=ctx.getVelocities())
    if state["piston"]:
        out["box"] = state["fm"].getBoxDimensions()
    return out


# ---------------------------------------------------------------- work and tolerance

def _one(n, box, case):
    """(bytes, flops) of one force evaluation: 65 operations per pair inside the
    cutoff, the spline sums, two real transforms; the charge grid, the spectrum and
    the potential each written once and read once."""
    g = float(np.prod(_grid(case, box)))
    rho = n / float(np.prod(box))
    pairs = 0.5 * n * rho * 4.0 / 3.0 * math.pi * case["roff"] ** 3
    p3 = case["order"] ** 3
    return 24.0 * g + 16.0 * n + 24.0 * n, 65.0 * pairs + n * p3 * 10.0 + 5.0 * g * math.log2(g)


def work(case):
    if case["path"] == "batch":
        b = f = 0.0
        for size, t in _batch_members(case):
            n = size * int(np.prod(t)) - 3 * case["drop"]
            L = (size / DENSITY) ** (1.0 / 3.0)
            ob, of = _one(n, [k * L for k in t], case)
            b += case["steps"] * (ob + 144.0 * n) + 48.0 * n
            f += case["steps"] * (of + 100.0 * n)
        return {"bytes": b, "flops": f}
    per = 3 * case["tile"] if case["kind"] == "water" else case["tile"]
    t = (case["tx"], case["ty"], case["tz"])
    L = (per / DENSITY) ** (1.0 / 3.0)
    n = per * int(np.prod(t)) - 3 * case["drop"]
    ob, of = _one(n, [k * L for k in t], case)
    if case["path"] == "forces":
        return {"bytes": ob + 48.0 * n, "flops": of}
    # coordinates, velocities and displacements of 64 bits read and written a step
    return {"bytes": case["steps"] * (ob + 144.0 * n) + 48.0 * n,
            "flops": case["steps"] * (of + 100.0 * n)}


def tolerance(case):
    if case["path"] == "forces":
        # single-precision pair terms and grids, 64-bit sums: about 1.5e-6 from 64 bits
        return {"rel": 6e-6, "max": 4e-4}
    if case.get("integrator") == "leapfrog":
        # the plain and the precise form differ by 1.6e-6 after two passes of 40 steps
        return {"rel": 8e-6, "max": 1e-4}
    # relaxed from a lattice, these runs heat up and part faster: the plain and the
    # precise form differ by 1e-5 after two passes of 40 steps, single atoms by 7e-4
    return {"rel": 5e-5, "max": 5e-3}


# ---------------------------------------------------------------- 64 bits

class _Field:
    """The force field in 64-bit torch arithmetic, every pair of atoms by hand.
    `beads`: atoms of one chain (all chains alike, in front of the waters)."""

    def __init__(self, s, box, roff, ron, grid, order, beads):
        self.device = torch.device("cuda" if torch.cuda.is_available() else "cpu")

        def t(a, kind=torch.float64):
            return torch.tensor(np.asarray(a), dtype=kind, device=self.device)

        n = s.n_atoms
        self.n, self.box, self.roff, self.ron = n, t(box), roff, ron
        self.grid, self.order = grid, order
        self.q = t(s.charge)
        self.mass = t(s.mass)
        types = sorted(set(s.atom_type))
        at = np.array([types.index(a) for a in s.atom_type])
        self.at = t(at, torch.int64)

        def table(of):
            e = np.array([abs(of(k)[0]) for k in types])
            r = np.array([of(k)[1] for k in types])
            eps, rm = np.sqrt(e[:, None] * e[None]), r[:, None] + r[None]
            return t(2.0 * eps * rm ** 6), t(eps * rm ** 12)

        self.c6, self.c12 = table(lambda k: s.lj_params[k])
        self.c6s, self.c12s = table(lambda k: s.lj14_params.get(k, s.lj_params[k]))
        # chains are linear: 1-2, 1-3 and 1-4 partners are the next three beads
        names = s.atom_type
        chain = np.array([not (a in ("OT", "HT")) for a in names])
        nb = int(chain.sum())
        k = np.arange(nb)
        inside = k % max(beads, 1)

        def along(d):
            i = k[inside < beads - d] if beads else k
            return np.stack([i, i + d], 1)

        w = np.arange(nb, n, 3)
        near = np.concatenate([np.stack([w, w + 1], 1), np.stack([w, w + 2], 1), np.stack([w + 1, w + 2], 1)])
        self.near = t(np.concatenate([along(1), along(2), near]), torch.int64)
        self.in14 = t(along(3), torch.int64)
        every = np.concatenate([along(1), along(2), along(3), near])
        every = np.concatenate([every, every[:, ::-1]])
        every = every[np.argsort(every[:, 0], kind="stable")]
        self.excl = t(every, torch.int64)
        self.excl_row = every[:, 0]
        self.bonds, self.angles, self.dihedrals = (t(a, torch.int64) for a in (s.bonds, s.angles, s.dihedrals))

        def looked_up(rows, width, f):
            seen = {}
            out = []
            for r in at[rows] if len(rows) else []:
                key = tuple(int(v) for v in r)
                if key not in seen:
                    seen[key] = f(*(types[v] for v in key))
                out.append(seen[key])
            return t(np.array(out, dtype=np.float64).reshape(len(rows), width))

        self.kb = looked_up(np.asarray(s.bonds), 2, lambda a, b: s.bond_params[tuple(sorted((a, b)))])
        self.ka = looked_up(np.asarray(s.angles), 2, lambda a, b, c: s.angle_params[(min(a, c), b, max(a, c))])
        self.kd = looked_up(np.asarray(s.dihedrals), 3,
                            lambda a, b, c, d: s.dihedral_params[("X",) + tuple(sorted((b, c))) + ("X",)][0])

    def _lj(self, r2, c6, c12):
        """(factor, energy) of the force-switched Lennard-Jones term: the gradient on
        i is factor times (x_i - x_j)."""
        ri2 = 1.0 / r2
        ri6 = ri2 ** 3
        ri3 = torch.sqrt(ri6)
        of3, on3 = self.roff ** 3, self.ron ** 3
        sw = (r2 > self.ron ** 2).to(r2.dtype)
        a6 = 1.0 + sw * (of3 / (of3 - on3) - 1.0)
        a12 = 1.0 + sw * (of3 ** 2 / (of3 ** 2 - on3 ** 2) - 1.0)
        t6, t12 = ri3 - sw / of3, ri6 - sw / of3 ** 2
        f = (6.0 * c6 * a6 * t6 * ri3 - 12.0 * c12 * a12 * t12 * ri6) * ri2
        e = c12 * (a12 * t12 ** 2 - (1.0 - sw) / (on3 ** 2 * of3 ** 2)) - c6 * (a6 * t6 ** 2 - (1.0 - sw) / (on3 * of3))
        return f, e

    def direct(self, x):
        """Gradient, (elec, vdw), virial over all pairs inside the cutoff."""
        g = torch.zeros_like(x)
        sums = torch.zeros(2, dtype=x.dtype, device=x.device)
        vir = torch.zeros(3, 3, dtype=x.dtype, device=x.device)
        step = max(1, min(self.n, 24_000_000 // self.n))
        for a in range(0, self.n, step):
            b = min(self.n, a + step)
            d = [x[a:b, None, k] - x[None, :, k] for k in range(3)]
            d = [v - self.box[k] * torch.round(v / self.box[k]) for k, v in enumerate(d)]
            r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
            near = r2 < self.roff ** 2
            lo, hi = np.searchsorted(self.excl_row, [a, b])
            e = self.excl[lo:hi]
            near[e[:, 0] - a, e[:, 1]] = False
            i = torch.arange(a, b, device=x.device)
            near[i - a, i] = False
            row, col = torch.nonzero(near, as_tuple=True)  # only these are worked out
            d = torch.stack([v[row, col] for v in d], 1)
            r2 = r2[row, col]
            qq = CCELEC * self.q[a:b][row] * self.q[col]
            r = torch.sqrt(r2)
            ec = qq * torch.erfc(KAPPA * r) / r
            fc = -(qq * 2.0 * KAPPA / math.sqrt(math.pi) * torch.exp(-KAPPA ** 2 * r2) + ec) / r2
            ti, tj = self.at[a:b][row], self.at[col]
            fl, el = self._lj(r2, self.c6[ti, tj], self.c12[ti, tj])
            f = (fc + fl)[:, None] * d
            g[a:b].index_add_(0, row, f)
            sums += 0.5 * torch.stack([ec.sum(), el.sum()])
            vir -= 0.5 * d.T @ f
        return g, sums, vir

    def pairs14(self, x):
        """Gradient, (elec, vdw, ewex), virial of the 1-4 pairs and of the 1-2 and
        1-3 pairs' reciprocal-space parts."""
        g = torch.zeros_like(x)
        out = []
        vir = torch.zeros(3, 3, dtype=x.dtype, device=x.device)
        for pairs, scaled in ((self.in14, True), (self.near, False)):
            d = x[pairs[:, 0]] - x[pairs[:, 1]]
            r2 = (d * d).sum(1)
            r = torch.sqrt(r2)
            qq = CCELEC * self.q[pairs[:, 0]] * self.q[pairs[:, 1]]
            e = qq * (torch.erfc(KAPPA * r) if scaled else -torch.erf(KAPPA * r)) / r
            f = -(qq * 2.0 * KAPPA / math.sqrt(math.pi) * torch.exp(-KAPPA ** 2 * r2) + e) / r2
            if scaled:
                ti, tj = self.at[pairs[:, 0]], self.at[pairs[:, 1]]
                fl, el = self._lj(r2, self.c6s[ti, tj], self.c12s[ti, tj])
                f = f + fl
                out.append(el.sum())
            out.append(e.sum())
            v = f[:, None] * d
            g.index_add_(0, pairs[:, 0], v)
            g.index_add_(0, pairs[:, 1], -v)
            vir -= d.T @ v
        return g, torch.stack([out[1], out[0], out[2]]), vir

    def bonded(self, x):
        """Gradient, (bond, angle, dihe), virial by autograd."""
        x = x.detach().requires_grad_(True)
        i, j = self.bonds.T
        b = (self.kb[:, 0] * (torch.linalg.norm(x[i] - x[j], dim=1) - self.kb[:, 1]) ** 2).sum()
        i, j, k = self.angles.T
        u, v = x[i] - x[j], x[k] - x[j]
        c = torch.cross(u, v, dim=1)
        th = torch.atan2(torch.linalg.norm(c, dim=1), (u * v).sum(1))
        a = (self.ka[:, 0] * (th - torch.deg2rad(self.ka[:, 1])) ** 2).sum()
        e = torch.zeros((), dtype=x.dtype, device=x.device)
        if len(self.dihedrals):
            i, j, k, l = self.dihedrals.T
            p, q, r = x[j] - x[i], x[k] - x[j], x[l] - x[k]
            m, n = torch.cross(p, q, dim=1), torch.cross(q, r, dim=1)
            phi = torch.atan2(torch.linalg.norm(q, dim=1) * (p * n).sum(1), (m * n).sum(1))
            e = (self.kd[:, 0] * (1.0 + torch.cos(self.kd[:, 1] * phi - torch.deg2rad(self.kd[:, 2])))).sum()
        g, = torch.autograd.grad(b + a + e, x)
        return g, torch.stack([b, a, e]).detach(), -x.detach().T @ g

    def _spline(self, w):
        """Cardinal B-spline values at w, w + 1, ... w + order - 1, by the recursion
        M_k(u) = (u M_{k-1}(u) + (k - u) M_{k-1}(u - 1)) / (k - 1)."""
        m = [w, 1.0 - w]  # M_2 at w and w + 1
        for k in range(3, self.order + 1):
            prev = [torch.zeros_like(w)] + m + [torch.zeros_like(w)]
            m = [((w + j) * prev[j + 1] + (k - w - j) * prev[j]) / (k - 1) for j in range(k)]
        return torch.stack(m, 1)

    def recip(self, x):
        """Gradient, energy, virial of the smooth particle-mesh sum."""
        p, n3 = self.order, self.grid
        x = x.detach().requires_grad_(True)
        at, wt = [], []
        for k in range(3):
            u = (x[:, k] / self.box[k] + 2.0) * n3[k]
            i = torch.floor(u.detach())
            # point i - j takes M_p(u - i + j)
            wt.append(self._spline(u - i))
            at.append((i.to(torch.int64)[:, None] - torch.arange(p, device=x.device)) % n3[k])
        size = n3[0] * n3[1] * n3[2]
        q = torch.zeros(size, dtype=x.dtype, device=x.device)
        for j in range(p):  # one z point at a time: 1 / p of the memory
            flat = ((at[0][:, :, None] * n3[1] + at[1][:, None, :]) * n3[2] + at[2][:, j, None, None]).reshape(-1)
            val = (self.q * wt[2][:, j])[:, None, None] * wt[0][:, :, None] * wt[1][:, None, :]
            q = q.index_add(0, flat, val.reshape(-1))
        s = torch.fft.rfftn(q.detach().reshape(*n3))
        m = [torch.fft.fftfreq(n3[k], 1.0 / n3[k], dtype=x.dtype, device=x.device) for k in range(3)]
        m[2] = m[2][:n3[2] // 2 + 1].abs()
        m = [v / self.box[k] for k, v in enumerate(m)]
        w = torch.zeros(1, dtype=x.dtype, device=x.device)
        mod = []
        for k in range(3):
            a = self._spline(w)[0]  # M_p(0), M_p(1), ...
            ph = torch.arange(n3[k], device=x.device)[:, None] * torch.arange(p, device=x.device)[None]
            ph = 2.0 * math.pi * (ph % n3[k]).to(x.dtype) / n3[k]
            b = (a * torch.cos(ph)).sum(1) ** 2 + (a * torch.sin(ph)).sum(1) ** 2
            mod.append(1.0 / b)
        mx, my, mz = m[0][:, None, None], m[1][None, :, None], m[2][None, None, :]
        m2 = mx ** 2 + my ** 2 + mz ** 2
        m2[0, 0, 0] = 1.0
        fac = math.pi ** 2 / KAPPA ** 2
        infl = torch.exp(-fac * m2) / (math.pi * self.box.prod() * m2)
        infl = infl * mod[0][:, None, None] * mod[1][None, :, None] * mod[2][None, None, :n3[2] // 2 + 1]
        infl[0, 0, 0] = 0.0
        phi = torch.fft.irfftn(infl * s, s=n3, norm="forward")
        e = 0.5 * CCELEC * (q.detach().reshape(*n3) * phi).sum()
        twice = torch.full_like(m[2], 2.0)
        twice[0] = 1.0
        twice[-1] = 1.0  # every grid size is even
        t1 = 0.5 * CCELEC * infl * s.abs() ** 2 * twice
        vt = 2.0 * (fac + 1.0 / m2)
        dirs = [mx, my, mz]
        vir = torch.stack([torch.stack([(t1 * (vt * dirs[a] * dirs[b] - (1.0 if a == b else 0.0))).sum()
                                        for b in range(3)]) for a in range(3)])
        g, = torch.autograd.grad((q * phi.reshape(-1)).sum(), x)
        return CCELEC * g, e, -vir

    def all(self, x):
        gd, (el, vd), wd = self.direct(x)
        gp, (e14, v14, ex), wp = self.pairs14(x)
        gb, (b, a, dh), wb = self.bonded(x)
        gr, ek, wr = self.recip(x)
        z = torch.zeros_like(ek)
        se = -KAPPA * CCELEC / math.sqrt(math.pi) * (self.q ** 2).sum()
        return (gd + gp + gb + gr, torch.stack([b, a, z, dh, z, ek, se, ex, el + e14, vd + v14]),
                wd + wp + wb + wr)


def exact(case, seed):
    if case["path"] == "batch" or (case["path"] == "md" and case["integrator"] != "leapfrog"):
        return None  # constraint and noise algorithms with states of their own
    big, beads, chains, _, _ = _repeat(case["kind"], case["tile"], (case["tx"], case["ty"], case["tz"]),
                                       case["drop"])
    n = big.n_atoms
    if n > 60000 or (case["path"] == "md" and n * float(n) * case["steps"] > 1.2e10):
        return None  # over about 20 seconds
    x, v = _inputs(big, beads, chains, seed)
    f = _Field(big, big.box, case["roff"], case["ron"], _grid(case, big.box), case["order"], beads)
    x = torch.tensor(x, dtype=torch.float64, device=f.device)
    if case["path"] == "forces":
        g, e, w = f.all(x)
        out = dict(forces=g, energies=e)
        if case["virial"]:
            out["virial"] = w
        return {k: val.cpu().numpy() for k, val in out.items()}
    # leapfrog: v -= dt g / m, x += dt v; at the start of every 20 steps molecules
    # whose centre has left the box come back into it
    v = torch.tensor(v, dtype=torch.float64, device=f.device)
    dt = case["dt"] / TIMFAC
    nb = beads * chains
    for k in range(case["steps"]):
        if k % 20 == 0:
            for part in ([x[:nb].reshape(chains, -1, 3)] if beads else []) + [x[nb:].reshape(-1, 3, 3)]:
                c = part.mean(1, keepdim=True)
                part -= f.box * ((c > 0.5 * f.box).to(x.dtype) - (c < -0.5 * f.box).to(x.dtype))
        g = f.direct(x)[0] + f.pairs14(x)[0] + f.bonded(x)[0] + f.recip(x)[0]
        v = v - dt * g / f.mass[:, None]
        x = x + dt * v
    return dict(coordinates=x.cpu().numpy(), velocities=v.cpu().numpy())
