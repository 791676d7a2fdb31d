"""The calls whose speed this repository measures, with inputs of the shapes that simulations give them.

A case is a plain dict; its "kind" says which part of the framework it calls:

  moves     Ewald energy differences of single moves, each accepted: the innermost call of a host-driven simulation
  trials    the trial energies of CBMC insertions into a large mixture (first beads, then orientations)
  grids     the interpolation grids of one framework (two Lennard-Jones probes and the unit-charge Ewald grid)
  quintic   one triquintic grid
  gridtest  the grid test that follows a build
  full      the full structure-factor recompute of a system
  batch     one move in each of many systems that share a box
  gcmc      many independent GCMC chains of rigid CO2
  mixture   one large CO2 / N2 system on the whole GPU
  alkane    batched flexible-chain CBMC over systems of uneven size
  proposal  training and tabulating the learned first-bead proposal

Sizes are those of the benchmark's workloads (bench.py, raspa3_b200/synthetic.py, mixture.py, alkane.py) and of smaller
systems of the same make.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from raspa3_b200 import native
from raspa3_b200.alkane import alkane_batch_systems, alkane_forcefield
from raspa3_b200.forcefield import (COULOMBIC_CONVERSION_FACTOR, ENERGY_TO_KELVIN, grid_points_for_spacing, make_atoms,
                                    positions_of)
from raspa3_b200.gcmc import beta_of, co2_component, fugacity_of, n2_component
from raspa3_b200.mixture import MIXTURE_CELL, molecules_as_atoms, total_energy
from raspa3_b200.synthetic import (CO2_NAMES, CO2_OFFSETS, SYNTHETIC_CELL, random_molecules, random_rotation, replicate,
                                   rigid_molecule, synthetic_forcefield, synthetic_framework)

RC = 12.0


def listed():
    return [
        # a small charged box (2 x 2 x 3 unit cells, 30 CO2): the call a host-driven simulation makes for every
        # charged move; latency and launches are all of it
        {"name": "moves_small_box", "kind": "moves", "kmax": 8, "sphere": True, "reps": "2x2x3", "molecules": 30,
         "moves": 8},
        # one CBMC insertion after another into a mixture of 12,000 sites, all energies in FP64
        {"name": "trials_large_mixture", "kind": "trials", "co2": 2000, "n2": 2000, "reps": "4x4x4", "insertions": 4,
         "trials": 10, "fp32c": False},
        # the headline build: three grids of 133 x 133 x 89 points in FP32C
        {"name": "grids_fp32c", "kind": "grids", "spacing": 0.15, "fp32c": True},
        # the same three grids in the reference's precision, at the coarser ragged 80 x 80 x 54 points
        {"name": "grids_fp64", "kind": "grids", "spacing": 0.25, "fp32c": False},
        # a triquintic Lennard-Jones grid (27 values per point, FP64)
        {"name": "quintic_lj", "kind": "quintic", "spacing": 0.2, "ewald": False},
        # the reference's default number of test points after a build, energies and charge term
        {"name": "gridtest_100k", "kind": "gridtest", "spacing": 0.25, "points": 100000},
        # the recompute at initialisation and for drift checks: 12,000 sites x 8,124 k-vectors
        {"name": "full_large_mixture", "kind": "full", "kmax": 12, "sphere": False, "reps": "4x4x4", "molecules": 4000},
        # a screening run: one translation in each of 1,184 systems
        {"name": "batch_1184", "kind": "batch", "kmax": 12, "sphere": False, "reps": "4x4x4", "systems": 1184},
        # GCMC of CO2 with eight chains per SM, at a loading of about eight molecules
        {"name": "gcmc_1184", "kind": "gcmc", "chains": 1184, "moves": 200, "kmax": 8},
        # the large mixture as one system on all SMs
        {"name": "mixture_4000", "kind": "mixture", "co2": 2000, "n2": 2000, "reps": "4x4x4", "kmax": 12,
         "moves": 1000},
        # 64 uneven systems, chains of 4 to 8 beads
        {"name": "alkane_64", "kind": "alkane", "systems": 64, "moves": 200},
        # the learned proposal from grid samples to the tabulated density
        {"name": "proposal", "kind": "proposal", "samples": 1 << 18, "steps": 100, "batch": 4096, "cells": 48},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["moves", "trials", "grids", "quintic", "gridtest", "full", "batch", "gcmc", "mixture", "alkane",
                       "proposal"])
    reps = lambda m: "x".join(str(rng.randint(1, m)) for _ in range(3))  # noqa: E731
    if kind == "moves":
        return {"kind": kind, "kmax": rng.randint(4, 12), "sphere": rng.random() < 0.5, "reps": reps(3),
                "molecules": _log(rng, 8, 400), "moves": rng.randint(2, 12)}
    if kind == "trials":
        r = rng.randint(1, 3)
        most = 30 * r ** 3
        return {"kind": kind, "co2": _log(rng, 4, most), "n2": _log(rng, 4, most), "reps": f"{r}x{r}x{r + 1}",
                "insertions": rng.randint(1, 4), "trials": rng.randint(4, 16), "fp32c": rng.random() < 0.3}
    if kind == "grids":
        fp32c = rng.random() < 0.5
        return {"kind": kind, "spacing": round(rng.uniform(0.16 if fp32c else 0.26, 0.8), 3), "fp32c": fp32c}
    if kind == "quintic":
        return {"kind": kind, "spacing": round(rng.uniform(0.32, 0.8), 3), "ewald": rng.random() < 0.5}
    if kind == "gridtest":
        return {"kind": kind, "spacing": round(rng.uniform(0.3, 0.8), 3), "points": _log(rng, 500, 100000)}
    if kind == "full":
        return {"kind": kind, "kmax": rng.randint(4, 12), "sphere": rng.random() < 0.5, "reps": reps(4),
                "molecules": _log(rng, 20, 4000)}
    if kind == "batch":
        return {"kind": kind, "kmax": rng.randint(4, 12), "sphere": rng.random() < 0.5, "reps": reps(4),
                "systems": _log(rng, 16, 1184)}
    if kind == "gcmc":
        return {"kind": kind, "chains": _log(rng, 100, 1184), "moves": rng.randint(50, 200), "kmax": rng.randint(5, 8)}
    if kind == "mixture":
        r = rng.randint(2, 3)
        most = 25 * r ** 3
        return {"kind": kind, "co2": _log(rng, 20, most), "n2": _log(rng, 20, most), "reps": f"{r}x{r}x{r}",
                "kmax": rng.randint(6, 10), "moves": rng.randint(200, 1000)}
    if kind == "alkane":
        return {"kind": kind, "systems": _log(rng, 4, 64), "moves": rng.randint(50, 200)}
    return {"kind": kind, "samples": _log(rng, 1 << 14, 1 << 18), "steps": rng.randint(20, 100),
            "batch": rng.choice([1024, 1536, 2048, 4096]), "cells": rng.randint(16, 48)}


# ---- inputs ----

_CTX = None


def _context():
    """One context for the process, as a program keeps one per host thread."""
    global _CTX
    if _CTX is None:
        _CTX = native.Context(0)
    return _CTX


def _reps(case):
    return tuple(int(v) for v in case["reps"].split("x"))


def _empty(n, dtype=torch.float64):
    return torch.empty(n, dtype=dtype, device="cuda")


def _unit(case, seed):
    """The force field and framework unit cell of a grid case."""
    ff = synthetic_forcefield(charges=True)
    cell, atoms = synthetic_framework(ff, seed=1000 + seed)
    return ff, cell, atoms


def _ewald_box(case):
    ff = synthetic_forcefield(charges=True, alpha=0.265, kmax=case["kmax"], sphere=case["sphere"])
    lengths = SYNTHETIC_CELL if case["kind"] == "moves" else MIXTURE_CELL
    return ff, np.diag(np.asarray(lengths) * np.asarray(_reps(case), dtype=np.float64))


def _translations(ff, mols, rng, count):
    """`count` pairs (new atoms, old atoms) of random CO2 translations."""
    moved = []
    for _ in range(count):
        m = int(rng.integers(len(mols) // 3))
        old = mols[3 * m:3 * m + 3].copy()
        new = old.copy()
        for axis, step in zip("xyz", 0.5 * rng.normal(size=3)):
            new[axis] += step
        moved.append((new, old))
    return moved


def _moves_inputs(case, seed):
    rng = np.random.default_rng(seed)
    ff, cell = _ewald_box(case)
    mols = random_molecules(ff, cell, case["molecules"], seed=int(rng.integers(1 << 30)))
    # distinct molecules, so that undoing the moves in any order restores the configuration
    picks = rng.permutation(case["molecules"])[:case["moves"]]
    moved = []
    for m in picks:
        moved += _translations(ff, mols[3 * m:3 * m + 3], rng, 1)
    return ff, cell, mols, moved


def _full_inputs(case, seed):
    rng = np.random.default_rng(seed)
    ff, cell = _ewald_box(case)
    n = case["molecules"]
    com = rng.random((n, 1, 3)) @ cell
    axis = rng.normal(size=(n, 1, 3))
    axis /= np.linalg.norm(axis, axis=2, keepdims=True)
    pos = com + np.asarray([1.16, 0.0, -1.16])[None, :, None] * axis
    types = np.tile([ff.index(v) for v in CO2_NAMES], n)
    charges = np.array([ff.pseudo_atoms[t].charge for t in types])
    return ff, cell, make_atoms(pos.reshape(-1, 3), types, charges, molecule_ids=np.repeat(np.arange(n), 3))


def _batch_inputs(case, seed):
    rng = np.random.default_rng(seed)
    ff, cell = _ewald_box(case)
    mols = random_molecules(ff, cell, 200, seed=int(rng.integers(1 << 30)))
    moved = _translations(ff, mols, rng, case["systems"])
    ahead = np.concatenate([np.concatenate([new, old]) for new, old in moved])
    back = np.concatenate([np.concatenate([old, new]) for new, old in moved])
    return ff, cell, mols, ahead, back


def _linear(rng, cell, comp):
    """Whole linear molecules (CO2 where comp is 0, N2 where it is 1) at random points: [molecules, 3 atoms, xyz]."""
    n = len(comp)
    axis = rng.normal(size=(n, 1, 3))
    axis /= np.linalg.norm(axis, axis=2, keepdims=True)
    half = np.where(comp == 0, 1.16, 0.55)[:, None, None]
    return rng.random((n, 1, 3)) @ cell + np.asarray([1.0, 0.0, -1.0])[None, :, None] * half * axis


def _place(rng, ucell, ufw, scell, counts, min_fw=2.6, min_mol=2.8):
    """A random mixture without overlaps: no atom within min_fw of the framework or min_mol of another molecule's."""
    left = list(counts)
    tries = 16 * sum(counts) + 200
    comp = rng.permutation(np.repeat([0, 1], [tries * counts[0] // sum(counts) + 1,
                                              tries * counts[1] // sum(counts) + 1]))
    xyz = _linear(rng, scell, comp)
    x = torch.from_numpy(xyz).cuda()
    fw = torch.from_numpy(positions_of(ufw)).cuda()
    small, box = (torch.from_numpy(np.diag(c).copy()).cuda() for c in (ucell, scell))

    def near(a, b, lengths, reach):
        d = a[:, :, None, None, :] - b[None, None]
        d -= lengths * (d / lengths).round()
        return ((d * d).sum(-1) < reach * reach).any(1).any(-1)

    free = torch.cat([~near(x[i:i + 1024], fw[:, None, :], small, min_fw).any(1) for i in range(0, len(x), 1024)])
    x, keep = x[free], free.cpu().numpy()
    xyz, comp = xyz[keep], comp[keep]
    clash = torch.cat([near(x[i:i + 64], x, box, min_mol) for i in range(0, len(x), 64)]).cpu().numpy()
    blocked = np.zeros(len(xyz), dtype=bool)
    taken = []
    for i in range(len(xyz)):
        if not blocked[i] and left[comp[i]] > 0:
            left[comp[i]] -= 1
            taken.append(i)
            blocked |= clash[i]
    if any(left):
        raise RuntimeError("could not place the molecules")
    return xyz[taken], comp[taken].astype(np.int32)


def _mixture_inputs(case, seed):
    rng = np.random.default_rng(seed)
    ff = synthetic_forcefield(charges=True, alpha=0.265, kmax=case.get("kmax", 6), sphere=False)
    ucell, ufw = synthetic_framework(ff, MIXTURE_CELL, n_t=96, seed=1000 + seed)
    scell, sfw = replicate(ucell, ufw, _reps(case))
    comps = [co2_component(), n2_component()]
    if case["kind"] == "trials":
        # the partner sites only: whole molecules at random points, as the pair sums see them
        comp = rng.permutation(np.repeat([0, 1], [case["co2"], case["n2"]]))
        xyz = _linear(rng, scell, comp)
    else:
        xyz, comp = _place(rng, ucell, ufw, scell, (case["co2"], case["n2"]))
    return ff, ucell, ufw, scell, sfw, comps, xyz, comp, rng


def _trial_sets(case, ff, scell, n_mol, rng):
    sets = []
    tc = ff.index("C_co2")
    for _ in range(case["insertions"]):
        first = make_atoms(rng.random((case["trials"], 3)) @ scell, tc, ff.pseudo_atoms[tc].charge,
                           molecule_ids=np.full(case["trials"], n_mol))
        centre = positions_of(first)[int(rng.integers(case["trials"]))]
        orient = np.concatenate([rigid_molecule(ff, CO2_NAMES, CO2_OFFSETS, centre, random_rotation(rng), n_mol)
                                 for _ in range(case["trials"])])
        sets.append((first, orient))
    return sets


def _grids(ctx, ff, cell, atoms, dims, probes, ewald, precision):
    """Device grids of the named probes and, if asked, the unit-charge Ewald grid: [(slot, buffer)]."""
    types = [0] * len(probes) + ([1] if ewald else [])
    probe = [ff.index(n) for n in probes] + ([0] if ewald else [])
    bufs = [_empty(8 * dims[0] * dims[1] * dims[2]) for _ in types]
    torch.cuda.synchronize()
    ctx.grid_build_set(ff, cell, atoms, RC, dims, precision, types, probe, [b.data_ptr() for b in bufs])
    return list(zip([ff.n_types if t else p for t, p in zip(types, probe)], bufs))


def _attach(system, cell, dims, grids):
    for slot, buf in grids:
        system.set_grid(slot, cell, dims, buf.data_ptr(), on_device=True)


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    s = {"case": case, "ctx": ctx}
    if kind == "moves":
        ff, cell, mols, moved = _moves_inputs(case, seed)
        ew = native.Ewald(ctx, ff, cell)
        ew.full(mols, [3] * case["molecules"])
        s.update(ewald=ew, moved=moved)
    elif kind == "trials":
        ff, ucell, ufw, scell, sfw, comps, xyz, comp, rng = _mixture_inputs(case, seed)
        dims = grid_points_for_spacing(ucell, 0.3)
        system = native.System(ctx, ff, scell, sfw)
        grids = _grids(ctx, ff, ucell, ufw, dims, ("C_co2", "O_co2"), True, native.PRECISION_FP64)
        _attach(system, ucell, dims, grids)
        system.set_molecules(molecules_as_atoms(ff, comps, xyz, comp))
        if case["fp32c"]:
            system.set_precision(native.PRECISION_FP32C)
        s.update(system=system, grids=grids, sets=_trial_sets(case, ff, scell, len(comp), rng))
    elif kind == "grids":
        ff, cell, atoms = _unit(case, seed)
        dims = grid_points_for_spacing(cell, case["spacing"])
        s.update(ff=ff, cell=cell, atoms=atoms, dims=dims,
                 out=[_empty(8 * dims[0] * dims[1] * dims[2]) for _ in range(3)])
    elif kind == "quintic":
        ff, cell, atoms = _unit(case, seed)
        dims = grid_points_for_spacing(cell, case["spacing"])
        s.update(ff=ff, cell=cell, atoms=atoms, dims=dims, out=_empty(27 * dims[0] * dims[1] * dims[2]))
    elif kind == "gridtest":
        ff, cell, atoms = _unit(case, seed)
        dims = grid_points_for_spacing(cell, case["spacing"])
        scell, _ = replicate(cell, atoms, (2, 2, 3))
        points = np.random.default_rng(seed).random((case["points"], 3))
        s.update(ff=ff, cell=cell, atoms=atoms, dims=dims, scell=scell, points=points,
                 grids=_grids(ctx, ff, cell, atoms, dims, ("C_co2",), True, native.PRECISION_FP64))
    elif kind == "full":
        ff, cell, atoms = _full_inputs(case, seed)
        s.update(ewald=native.Ewald(ctx, ff, cell), atoms=atoms,
                 sizes=np.full(case["molecules"], 3, dtype=np.int32))
    elif kind == "batch":
        ff, cell, mols, ahead, back = _batch_inputs(case, seed)
        ew = native.Ewald(ctx, ff, cell)
        ew.full(mols, [3] * 200)
        batch = native.EwaldBatch(ew, case["systems"])
        for i in range(case["systems"]):
            batch.set(i)
        s.update(ewald=ew, batch=batch, ahead=ahead, back=back, three=np.full(case["systems"], 3, dtype=np.int32),
                 accept=np.ones(case["systems"], dtype=np.uint8))
    elif kind == "gcmc":
        # framework charges off, as in the comparison of proposals: with them the wells between randomly placed sites
        # fill without end and no loading is typical
        ff = synthetic_forcefield(charges=True, alpha=0.265, kmax=case["kmax"])
        for pa in ff.pseudo_atoms[:2]:
            pa.charge = 0.0
        cell, atoms = synthetic_framework(ff, seed=1000 + seed)
        scell, sfw = replicate(cell, atoms, (2, 2, 3))
        dims = grid_points_for_spacing(cell, 0.15)
        grids = _grids(ctx, ff, cell, atoms, dims, ("C_co2", "O_co2"), True, native.PRECISION_FP32C)
        system = native.System(ctx, ff, scell, sfw)
        _attach(system, cell, dims, grids)
        ew = native.Ewald(ctx, ff, scell)
        ew.set_framework(sfw)
        g = native.Gcmc(system, ew, co2_component(), beta_of(300.0), fugacity_of(1e6), n_chains=case["chains"],
                        seed=1 + seed)
        g.run(1500, record=False)
        s.update(system=system, ewald=ew, grids=grids, gcmc=g)
    elif kind == "mixture":
        ff, ucell, ufw, scell, sfw, comps, xyz, comp, rng = _mixture_inputs(case, seed)
        dims = grid_points_for_spacing(ucell, 0.2)
        system = native.System(ctx, ff, scell, sfw)
        grids = _grids(ctx, ff, ucell, ufw, dims, ("C_co2", "O_co2", "N_n2", "N_com"), True, native.PRECISION_FP32C)
        _attach(system, ucell, dims, grids)
        ew = native.Ewald(ctx, ff, scell)
        ew.set_framework(sfw)
        energy = total_energy(system, ew, ff, comps, xyz, comp)
        mx = native.Mixture(system, ew, comps, beta_of(300.0), [fugacity_of(1e5)] * 2, xyz, comp,
                            max_molecules=len(comp) + len(comp) // 2 + 200, seed=1 + seed)
        mx.set_state(energy, ew.structure_factors(0))
        mx.run(200, record=False)
        s.update(system=system, ewald=ew, grids=grids, mixture=mx)
    elif kind == "alkane":
        ff = alkane_forcefield()
        systems = alkane_batch_systems(ff, n_systems=case["systems"], seed=1000 + seed, max_molecules=128)
        w_ig = {}
        for q in systems:
            nb = q.chain.n_beads
            if nb not in w_ig:
                w_ig[nb] = native.alkane_grow_vacuum(ctx, ff, q.chain, q.beta, 20000, seed=17)
            q.w_ig = w_ig[nb]
        a = native.Alkane(ctx, ff, systems, seed=1 + seed)
        # the plan the autotuner chooses for this batch, given outright so that every run takes the same one
        a.set_plan(1, 1, 512, 0, 500)
        a.run(1000, record=False)
        s.update(alkane=a)
    else:
        ff, cell, atoms = _unit(case, seed)
        scell, sfw = replicate(cell, atoms, (2, 2, 3))
        dims = grid_points_for_spacing(cell, 0.25)
        system = native.System(ctx, ff, scell, sfw)
        grids = _grids(ctx, ff, cell, atoms, dims, ("C_co2",), False, native.PRECISION_FP64)
        _attach(system, cell, dims, grids)
        n, nc = case["samples"], case["cells"] ** 3
        centres, weights, queries = _proposal_inputs(case, seed)
        mlp = native.Mlp(ctx, seed=1)
        mlp.set_params(weights)
        s.update(system=system, ff=ff, cell=cell, grids=grids, mlp=mlp, s=_empty((n, 3), torch.float32),
                 t=_empty(n, torch.float32), centres=torch.from_numpy(centres).cuda(), f=_empty(nc, torch.float32),
                 queries=queries, seed=1 + seed)
    ctx.synchronize()
    return s


def _proposal_inputs(case, seed):
    rng = np.random.default_rng(seed)
    g = (np.arange(case["cells"], dtype=np.float64) + 0.5) / case["cells"]
    k, j, i = np.meshgrid(g, g, g, indexing="ij")
    centres = np.stack([i, j, k], -1).reshape(-1, 3).astype(np.float32)
    u = lambda shape, fan: ((2.0 * rng.random(shape) - 1.0) * math.sqrt(6.0 / fan)).reshape(-1)  # noqa: E731
    weights = np.concatenate([u((64, 96), 96), np.zeros(64), u((64, 64), 64), np.zeros(64), u(64, 64), np.zeros(1)])
    return centres, weights.astype(np.float32), rng.random((1000, 3))


def _arrays(d):
    return {k: np.asarray(v) for k, v in d.items()}


def _energy_arrays(rows):
    return {"framework_vdw": np.array([r.framework_vdw for r in rows]),
            "framework_charge": np.array([r.framework_charge for r in rows]),
            "molecule_vdw": np.array([r.molecule_vdw for r in rows]),
            "molecule_charge": np.array([r.molecule_charge for r in rows]),
            "overlap": np.array([r.overlap for r in rows], dtype=np.int32)}


def _statistics(results):
    keys = results[0].keys()
    return {k: np.array([r[k] for r in results]) for k in keys}


def run(s):
    case = s["case"]
    kind = case["kind"]
    ctx = s["ctx"]
    if kind == "moves":
        # every move is taken and then undone, so that the state is the same before each pass
        ew = s["ewald"]
        out = []
        for new, old in s["moved"]:
            out.append(ew.delta(new, old)["ewald_fourier"])
            ew.accept()
        sk = ew.structure_factors(0)
        for new, old in reversed(s["moved"]):
            out.append(ew.delta(old, new)["ewald_fourier"])
            ew.accept()
        return {"energies": np.array(out), "structure_factors": sk}
    if kind == "trials":
        system = s["system"]
        out = []
        for first, orient in s["sets"]:
            out.append(_energy_arrays(system.external_energies(first, 1)))
            out.append(_energy_arrays(system.external_energies(orient, 3, skip=1)))
        return out
    if kind == "grids":
        ff = s["ff"]
        precision = native.PRECISION_FP32C if case["fp32c"] else native.PRECISION_FP64
        ctx.grid_build_set(ff, s["cell"], s["atoms"], RC, s["dims"], precision, [0, 0, 1],
                           [ff.index("C_co2"), ff.index("O_co2"), 0], [o.data_ptr() for o in s["out"]])
        return s["out"]
    if kind == "quintic":
        ctx.grid_build_triquintic(1 if case["ewald"] else 0, s["ff"], s["cell"], s["atoms"],
                                  0 if case["ewald"] else s["ff"].index("C_co2"), RC, s["dims"],
                                  out_device=s["out"].data_ptr(), host=False)
        return s["out"]
    if kind == "gridtest":
        ff = s["ff"]
        return _arrays(ctx.grid_validate(ff, s["cell"], s["atoms"], s["scell"], ff.index("C_co2"), s["dims"],
                                         s["grids"][0][1].data_ptr(), s["grids"][1][1].data_ptr(), 0.70, 1.0 / 300.0,
                                         points=s["points"]))
    if kind == "full":
        return {"energy": _arrays(s["ewald"].full(s["atoms"], s["sizes"])),
                "structure_factors": s["ewald"].structure_factors(0)}
    if kind == "batch":
        batch, three = s["batch"], s["three"]
        ahead = batch.delta(s["ahead"], 6, three, three)
        batch.accept(s["accept"])
        back = batch.delta(s["back"], 6, three, three)
        batch.accept(s["accept"])
        return [ahead, back]
    if kind == "gcmc":
        s["gcmc"].run(case["moves"], record=True)
        return _statistics(s["gcmc"].results())
    if kind == "mixture":
        s["mixture"].run(case["moves"], record=True)
        xyz, comp = s["mixture"].positions()
        room = s["mixture"].max_molecules
        positions, components = np.zeros((room,) + xyz.shape[1:]), np.full(room, -1, dtype=np.int32)
        positions[:len(comp)], components[:len(comp)] = xyz, comp
        return {"results": _arrays(s["mixture"].results()), "positions": positions, "components": components}
    if kind == "alkane":
        s["alkane"].run(case["moves"], record=True)
        return _statistics(s["alkane"].results())
    mlp, ff, n = s["mlp"], s["ff"], case["samples"]
    tc = ff.index("C_co2")
    native.sample_targets(s["system"], tc, 0.0, beta_of(300.0), -15.0, s["cell"], n, s["seed"], s["s"].data_ptr(),
                          s["t"].data_ptr())
    loss, gradient = mlp.loss_and_gradient(s["s"].data_ptr(), s["t"].data_ptr(), min(n, case["batch"]))
    mlp.train(s["s"].data_ptr(), s["t"].data_ptr(), n, case["steps"], batch=case["batch"], lr=2e-3, seed=s["seed"])
    mlp.evaluate(s["centres"].data_ptr(), case["cells"] ** 3, s["f"].data_ptr())
    proposal = native.Proposal(mlp, cells_per_axis=case["cells"], eps_uniform=0.05)
    q = proposal.density(s["queries"])
    proposal.close()
    return {"samples": s["s"], "targets": s["t"], "loss": torch.tensor(loss), "gradient": gradient,
            "parameters": mlp.params(), "log_density": s["f"], "density": q}


# ---- what a pass cannot do without ----


def _kcount(case):
    m, reach = case["kmax"], case["kmax"] ** 2
    n = 0
    for kx in range(0, m + 1):
        for ky in range(-m, m + 1):
            for kz in range(-m, m + 1):
                k2 = kx * kx + ky * ky + kz * kz
                n += k2 != 0 and (not case.get("sphere", True) or k2 <= reach)
    return n


def work(case):
    kind = case["kind"]
    density = 288 / float(np.prod(SYNTHETIC_CELL))
    ball = 4.0 / 3.0 * math.pi * RC ** 3
    if kind == "moves":
        # per difference: read S(k), write the trial S(k), read the prefactor and the k-vector; 6 atoms x 8 FLOPs per k
        nk, n = _kcount(case), 2 * case["moves"]
        return {"bytes": n * 44 * nk, "flops": n * nk * 6 * 8}
    if kind == "trials":
        sites = 3 * (case["co2"] + case["n2"])
        sets = case["insertions"] * 2
        cells = np.prod(_reps(case)) * float(np.prod(MIXTURE_CELL))
        pairs = case["insertions"] * 3 * case["trials"] * sites * min(1.0, ball / cells)
        tests = case["insertions"] * 3 * case["trials"] * sites
        return {"bytes": sets * sites * 64 + tests // max(1, sites) * 2 * 512, "flops": tests * 14 + pairs * 60}
    if kind in ("grids", "quintic"):
        dims = grid_points_for_spacing(np.diag(SYNTHETIC_CELL), case["spacing"])
        points = dims[0] * dims[1] * dims[2]
        if kind == "quintic":
            return {"bytes": points * 27 * 8, "flops": points * density * ball * (130 if case["ewald"] else 2 / 3 * 95)}
        return {"bytes": points * 3 * 64, "flops": points * density * ball * (2 / 3 * 2 * 55 + 65)}
    if kind == "gridtest":
        n = case["points"]
        return {"bytes": n * (24 + 2 * 512), "flops": n * density * ball * (2 / 3 * 25 + 45)}
    if kind == "full":
        nk, n = _kcount(case), 3 * case["molecules"]
        return {"bytes": n * 64 + nk * 16 * 2, "flops": n * nk * 4.0}
    if kind == "batch":
        nk = _kcount(case)
        return {"bytes": 2 * case["systems"] * (nk * 32 + 6 * 64), "flops": 2.0 * case["systems"] * nk * (6 * 8 + 10)}
    if kind == "gcmc":
        # per move: the Fourier difference of about 4.5 atoms and, for a third of the moves, 30 trial atoms
        nk = _kcount(dict(case, sphere=True))
        moves = case["chains"] * case["moves"]
        return {"bytes": moves * (nk * 24 + 20 * 512), "flops": moves * (nk * 4.5 * 8 + 14 * 250 * 2)}
    if kind == "mixture":
        nk = _kcount(dict(case, sphere=False))
        sites = 3 * (case["co2"] + case["n2"])
        return {"bytes": case["moves"] * (nk * 24 + sites * 16), "flops": case["moves"] * (nk * 30 * 8 + sites * 15 * 14)}
    if kind == "alkane":
        moves = case["systems"] * case["moves"]
        return {"bytes": moves * 950 * 16, "flops": moves * 950 * 35 * 16.0}
    per = 2.0 * (96 * 64 + 64 * 64 + 64)
    nc = case["cells"] ** 3
    return {"bytes": case["samples"] * (16 + 512) + case["steps"] * (case["batch"] * 16 + 10433 * 16) + nc * 32,
            "flops": (case["steps"] + 1) * case["batch"] * 3 * per + 2 * nc * per}


# ---- the same outputs in 64 bits from plain torch and numpy ----


def _kvectors(ff, cell):
    """(k integer triples, prefactors temp(k)) of an orthorhombic box, in the reference's order."""
    m = [int(v) for v in ff.kmax]
    kx, ky, kz = np.meshgrid(np.arange(0, m[0] + 1), np.arange(-m[1], m[1] + 1), np.arange(-m[2], m[2] + 1),
                             indexing="ij")
    k = np.stack([kx, ky, kz], -1).reshape(-1, 3)
    n2 = (k * k).sum(1)
    k = k[(n2 > 0) & (n2 <= min(ff.recip_int_cutoff_sq, 1 << 40))]
    lengths = np.diag(cell)
    g2 = ((2.0 * np.pi * k / lengths) ** 2).sum(1)
    pre = COULOMBIC_CONVERSION_FACTOR * 2.0 * np.pi / np.prod(lengths)
    temp = np.where(k[:, 0] == 0, 1.0, 2.0) * pre * np.exp(-0.25 * g2 / ff.ewald_alpha ** 2) / g2
    return k, temp


def _structure_factor(k, cell, atoms, chunk=2000):
    """sum_a q_a exp(2 pi i k.s_a), as a complex tensor on the GPU."""
    kt = torch.from_numpy(k.astype(np.float64)).cuda()
    s = torch.from_numpy(positions_of(atoms) / np.diag(cell)).cuda()
    q = torch.from_numpy(np.ascontiguousarray(atoms["charge"] * atoms["scaling_coulomb"])).cuda()
    total = torch.zeros(len(k), dtype=torch.complex128, device="cuda")
    for b in range(0, len(atoms), chunk):
        turns = s[b:b + chunk] @ kt.T
        turns = 2.0 * math.pi * (turns - turns.round())
        total += torch.complex(q[b:b + chunk] @ turns.cos(), q[b:b + chunk] @ turns.sin())
    return total


def _interleaved(z):
    return torch.view_as_real(z).reshape(-1).cpu().numpy()


def _net_charge(ff, temp, charge):
    """The net-charge term of a system of that charge, and its single-ion energy."""
    u = -(float(np.sum(temp)) - COULOMBIC_CONVERSION_FACTOR * ff.ewald_alpha / math.sqrt(math.pi))
    return u * charge * charge


def _exact_moves(case, seed):
    ff, cell, mols, moved = _moves_inputs(case, seed)
    k, temp = _kvectors(ff, cell)
    t = torch.from_numpy(temp).cuda()
    sk = _structure_factor(k, cell, mols)
    out = []
    for new, old in moved:
        d = _structure_factor(k, cell, new) - _structure_factor(k, cell, old)
        out.append(float((t * (2.0 * (sk.conj() * d).real + d.abs() ** 2)).sum()))
        sk = sk + d
    return {"energies": np.array(out + [-v for v in reversed(out)]), "structure_factors": _interleaved(sk)}


def _exact_full(case, seed):
    ff, cell, atoms = _full_inputs(case, seed)
    k, temp = _kvectors(ff, cell)
    sk = _structure_factor(k, cell, atoms)
    C, alpha = COULOMBIC_CONVERSION_FACTOR, ff.ewald_alpha
    q = atoms["charge"]
    fourier = float((torch.from_numpy(temp).cuda() * sk.abs() ** 2).sum()) + _net_charge(ff, temp, float(q.sum()))
    pos = positions_of(atoms).reshape(-1, 3, 3)
    q3 = q.reshape(-1, 3)
    excl = 0.0
    for i, j in ((0, 1), (0, 2), (1, 2)):
        r = np.linalg.norm(pos[:, i] - pos[:, j], axis=1)
        e = torch.erf(torch.from_numpy(alpha * r)).numpy()
        excl -= float(np.sum(C * q3[:, i] * q3[:, j] * e / r))
    self_energy = -C * alpha / math.sqrt(math.pi) * float(np.sum(q * q))
    return {"energy": _arrays({"ewald_fourier": fourier, "ewald_self": self_energy, "ewald_exclusion": excl,
                               "dudlambda_ewald": np.zeros(4)}),
            "structure_factors": _interleaved(sk)}


def _exact_batch(case, seed):
    ff, cell, mols, ahead, _ = _batch_inputs(case, seed)
    k, temp = _kvectors(ff, cell)
    t = torch.from_numpy(temp).cuda()
    sk = _structure_factor(k, cell, mols)
    kt = torch.from_numpy(k.astype(np.float64)).cuda()
    s = torch.from_numpy(positions_of(ahead) / np.diag(cell)).cuda().reshape(-1, 6, 3)
    q = ahead["charge"].reshape(-1, 6) * np.array([1.0] * 3 + [-1.0] * 3)
    q = torch.from_numpy(q).cuda()
    out = []
    for b in range(0, len(s), 64):
        turns = s[b:b + 64] @ kt.T
        turns = 2.0 * math.pi * (turns - turns.round())
        w = q[b:b + 64, :, None]
        d = torch.complex((w * turns.cos()).sum(1), (w * turns.sin()).sum(1))
        out.append((t * (2.0 * (sk.conj() * d).real + d.abs() ** 2)).sum(1))
    e = torch.cat(out).cpu().numpy()
    return [e, -e]


def _images(cell, atoms, keep, reach):
    """Positions and source indices of the periodic images of the atoms within reach of the cell."""
    lengths = np.diag(cell)
    pos, src = [], []
    n = [int(math.ceil(reach / v)) + 1 for v in lengths]
    base = positions_of(atoms)[keep]
    index = np.nonzero(keep)[0]
    for i in range(-n[0], n[0] + 1):
        for j in range(-n[1], n[1] + 1):
            for l in range(-n[2], n[2] + 1):
                p = base + np.array([i, j, l]) * lengths
                ok = np.all((p > -reach) & (p < lengths + reach), axis=1)
                pos.append(p[ok])
                src.append(index[ok])
    return np.concatenate(pos), np.concatenate(src)


class _Radial:
    """U(r) of a probe in a framework and its radial factors F_k = (1/r d/dr)^k U."""

    def __init__(self, ff, cell, atoms, probe):
        self.rc2 = ff.cutoff_framework_vdw ** 2
        types = atoms["type"].astype(int)
        if probe is None:
            keep = atoms["charge"] != 0.0
        else:
            keep = (ff.lj[types, probe] != 0) & (ff.epsilon[types, probe] != 0.0)
        pos, src = _images(cell, atoms, keep, RC + 1e-6)
        self.pos = torch.from_numpy(pos).cuda()
        self.alpha = ff.ewald_alpha if probe is None else None
        t = types[src]
        if probe is None:
            self.par = (torch.from_numpy(COULOMBIC_CONVERSION_FACTOR * atoms["charge"][src]).cuda(),)
        else:
            self.par = tuple(torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in
                             (4.0 * ff.epsilon[t, probe], ff.sigma[t, probe] ** 2, ff.shift[t, probe]))

    def factors(self, rr, n):
        """F_0..F_{n-1} for squared distances rr[points, images], zero outside the cutoff."""
        inside = (rr < self.rc2).to(rr.dtype)
        if self.alpha is None:
            a, s2, shift = self.par
            x = s2 / rr
            t = x * x * x
            out, power = [], inside * a
            c12 = c6 = 1.0
            for k in range(n):
                f = power * (c12 * t * t - c6 * t)
                out.append(f - inside * shift if k == 0 else f)
                power = power / rr
                c12 *= -(12.0 + 2.0 * k)
                c6 *= -(6.0 + 2.0 * k)
            return out
        cq, = self.par
        al = self.alpha
        r = rr.sqrt()
        b = torch.erfc(al * r) / r
        ex = torch.exp(-al * al * rr) / (al * math.sqrt(math.pi))
        out = []
        for k in range(n):
            out.append((-1.0) ** k * cq * b * inside)
            b = ((2 * k + 1) * b + (2.0 * al * al) ** (k + 1) * ex) / rr
        return out


def _grid_points(cell, dims, index):
    step = np.diag(cell) / (np.asarray(dims) - 1.0)
    i, j, k = index % dims[0], (index // dims[0]) % dims[1], index // (dims[0] * dims[1])
    return torch.from_numpy(np.stack([i, j, k], 1) * step).cuda()


def _axis_terms(order, x):
    """Derivative of order 0..2 along one axis: [(shift of k, factor)]."""
    if order == 0:
        return [(0, None)]
    if order == 1:
        return [(1, x)]
    return [(1, None), (2, x * x)]


_TRICUBIC = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1)]
_TRIQUINTIC = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (2, 0, 0), (1, 1, 0), (1, 0, 1), (0, 2, 0), (0, 1, 1),
               (0, 0, 2), (2, 1, 0), (2, 0, 1), (1, 2, 0), (1, 1, 1), (0, 2, 1), (1, 0, 2), (0, 1, 2), (2, 2, 0),
               (2, 0, 2), (0, 2, 2), (2, 1, 1), (1, 2, 1), (1, 1, 2), (2, 2, 1), (2, 1, 2), (1, 2, 2), (2, 2, 2)]


def _exact_grid(ff, cell, atoms, probe, dims, orders, index=None):
    """Grid channels at all grid points (or those of `index`): [points, channels]."""
    radial = _Radial(ff, cell, atoms, probe)
    if index is None:
        index = np.arange(dims[0] * dims[1] * dims[2])
    points = _grid_points(cell, dims, index)
    lengths = np.diag(cell)
    n = 1 + max(sum(o) for o in orders)
    scale = torch.tensor([math.prod((lengths[a] / (dims[a] - 1.0)) ** o[a] for a in range(3)) for o in orders],
                         dtype=torch.float64, device="cuda")
    out = torch.empty((len(index), len(orders)), dtype=torch.float64, device="cuda")
    per = 4096
    for b in range(0, len(index), per):
        p = points[b:b + per]
        # the images near this run of points, so that far ones are not evaluated at all
        lo, hi = p.amin(0) - RC, p.amax(0) + RC
        near = ((radial.pos > lo) & (radial.pos < hi)).all(1)
        part = _Radial.__new__(_Radial)
        part.rc2, part.alpha = radial.rc2, radial.alpha
        part.par = tuple(v[near] for v in radial.par)
        d = p[:, None, :] - radial.pos[near][None, :, :]
        f = part.factors((d * d).sum(2).clamp_min(0.1), n)
        x = [d[:, :, a].contiguous() for a in range(3)]
        for c, o in enumerate(orders):
            total = 0.0
            for k0, x0 in _axis_terms(o[0], x[0]):
                for k1, x1 in _axis_terms(o[1], x[1]):
                    for k2, x2 in _axis_terms(o[2], x[2]):
                        term = f[k0 + k1 + k2]
                        for y in (x0, x1, x2):
                            if y is not None:
                                term = term * y
                        total = total + term.sum(1)
            out[b:b + per, c] = total
    out *= scale
    # the overlap clamp
    oc = ff.overlap_criteria
    clash = out[:, 0] > oc
    out[clash, 1:4] = out[clash, 1:4].clamp(-oc, oc)
    out[clash, 4:] = 0.0
    out[clash, 0] = 2.0 * oc
    return out


def _exact_interpolant(cell, dims, corners, pos):
    """Tricubic value and Cartesian gradient at positions, from corners(index) -> [n, 8] channels."""
    lengths = torch.from_numpy(np.diag(cell).copy()).cuda()
    nc = torch.tensor([d - 1 for d in dims], dtype=torch.float64, device="cuda")
    s = pos / lengths
    s = s - s.floor()
    i0 = torch.minimum((s * nc).floor(), nc - 1)
    t = s * nc - i0
    i0 = i0.long()
    h = [[2 * t ** 3 - 3 * t ** 2 + 1, t ** 3 - 2 * t ** 2 + t], [3 * t ** 2 - 2 * t ** 3, t ** 3 - t ** 2]]
    g = [[6 * t ** 2 - 6 * t, 3 * t ** 2 - 4 * t + 1], [6 * t - 6 * t ** 2, 3 * t ** 2 - 2 * t]]
    index = []
    for c in range(8):
        i = i0 + torch.tensor([c & 1, (c >> 1) & 1, c >> 2], device="cuda")
        index.append(i[:, 0] + dims[0] * (i[:, 1] + dims[1] * i[:, 2]))
    values = corners(torch.cat(index)).reshape(8, len(pos), 8)
    e = torch.zeros(len(pos), dtype=torch.float64, device="cuda")
    grad = torch.zeros((len(pos), 3), dtype=torch.float64, device="cuda")
    for c in range(8):
        bits = (c & 1, (c >> 1) & 1, c >> 2)
        for l, o in enumerate(_TRICUBIC):
            v = values[c, :, l]
            b = [h[bits[a]][o[a]][:, a] for a in range(3)]
            db = [g[bits[a]][o[a]][:, a] for a in range(3)]
            e += v * b[0] * b[1] * b[2]
            grad[:, 0] += v * db[0] * b[1] * b[2]
            grad[:, 1] += v * b[0] * db[1] * b[2]
            grad[:, 2] += v * b[0] * b[1] * db[2]
    return e, grad * nc / lengths


def _corner_lookup(ff, cell, atoms, probe, dims):
    def corners(index):
        unique, inverse = torch.unique(index, return_inverse=True)
        return _exact_grid(ff, cell, atoms, probe, dims, _TRICUBIC, unique.cpu().numpy())[inverse]
    return corners


def _exact_gridtest(case, seed):
    ff, cell, atoms = _unit(case, seed)
    dims = grid_points_for_spacing(cell, case["spacing"])
    scell, _ = replicate(cell, atoms, (2, 2, 3))
    points = np.random.default_rng(seed).random((case["points"], 3))
    pos = torch.from_numpy(points @ scell).cuda()
    lengths = torch.from_numpy(np.diag(cell).copy()).cuda()
    inside = (pos / lengths - (pos / lengths).floor()) * lengths
    probe = ff.index("C_co2")
    sums = []
    count = []
    for which, scale in ((probe, ENERGY_TO_KELVIN), (None, 0.70 * ENERGY_TO_KELVIN)):
        radial = _Radial(ff, cell, atoms, which)
        ef, gf = [], []
        for b in range(0, len(inside), 8192):
            d = inside[b:b + 8192, None, :] - radial.pos[None, :, :]
            f = radial.factors((d * d).sum(2).clamp_min(0.1), 2)
            ef.append(f[0].sum(1))
            gf.append((f[1][:, :, None] * d).sum(1))
        ef, gf = torch.cat(ef) * scale, torch.cat(gf) * scale
        dense = _exact_grid(ff, cell, atoms, which, dims, _TRICUBIC)
        ei, gi = _exact_interpolant(cell, dims, lambda index: dense[index], pos)
        ei, gi = ei * scale, gi * scale
        if which is not None:
            w = torch.exp(-ef / 300.0)
            take = torch.ones_like(w)
            accessible = (ef < ff.overlap_criteria).to(w.dtype)
        else:
            take = accessible
        count.append(int(take.sum()))
        v = w * take
        part = [v.sum(), (v * ei).sum(), (v * ef).sum(), (v * (ef - ei) ** 2).sum(), (v * ef * ef).sum()]
        part += [(v[:, None] * m).sum(0) for m in (gi, gf, (gf - gi) ** 2, gf ** 2)]
        sums.append(torch.cat([p.reshape(-1) for p in part]).cpu().numpy())
    out = {"n_points": count[0], "n_points_charge": count[1], "sums": np.concatenate(sums)}
    for prefix, v in (("", sums[0]), ("charge_", sums[1])):
        out[prefix + "energy_table"], out[prefix + "energy_full"] = v[1] / v[0], v[2] / v[0]
        out[prefix + "energy_relative_error"] = math.sqrt(v[3] / v[4])
        out[prefix + "gradient_table"], out[prefix + "gradient_full"] = v[5:8] / v[0], v[8:11] / v[0]
        out[prefix + "gradient_relative_error"] = np.sqrt(v[11:14] / v[14:17])
    return _arrays(out)


def _exact_trials(case, seed):
    ff, ucell, ufw, scell, _, comps, xyz, comp, rng = _mixture_inputs(case, seed)
    dims = grid_points_for_spacing(ucell, 0.3)
    partners = molecules_as_atoms(ff, comps, xyz, comp)
    sets = _trial_sets(case, ff, scell, len(comp), rng)
    box = torch.from_numpy(np.diag(scell).copy()).cuda()
    ppos = torch.from_numpy(positions_of(partners)).cuda()
    ptype = partners["type"].astype(int)
    pq = torch.from_numpy(np.ascontiguousarray(partners["charge"])).cuda()
    grids = {}
    for name in ("C_co2", "O_co2", None):
        probe = None if name is None else ff.index(name)
        grids[probe] = _corner_lookup(ff, ucell, ufw, probe, dims)
    out = []
    for first, orient in sets:
        for atoms, size in ((first, 1), (orient[np.arange(len(orient)) % 3 != 1], 2)):
            pos = torch.from_numpy(positions_of(atoms)).cuda()
            t = int(atoms["type"][0])
            q = float(atoms["charge"][0])
            fv, _ = _exact_interpolant(ucell, dims, grids[t], pos)
            fc, _ = _exact_interpolant(ucell, dims, grids[None], pos)
            d = pos[:, None, :] - ppos[None, :, :]
            d = d - box * (d / box).round()
            rr = (d * d).sum(2)
            eps, sig2, shift = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in
                                (4.0 * ff.epsilon[ptype, t], ff.sigma[ptype, t] ** 2, ff.shift[ptype, t]))
            lj = torch.from_numpy((ff.lj[ptype, t] != 0).astype(np.float64)).cuda()
            x3 = (sig2 / rr) ** 3
            pair = torch.where(rr < RC * RC, lj * (eps * (x3 * x3 - x3) - shift), torch.zeros_like(rr))
            r = rr.sqrt()
            coul = torch.where(rr < RC * RC, COULOMBIC_CONVERSION_FACTOR * q * pq * torch.erfc(ff.ewald_alpha * r) / r,
                               torch.zeros_like(rr))
            sets_of = lambda v: v.reshape(-1, size).sum(1).cpu().numpy()  # noqa: E731
            out.append({"framework_vdw": sets_of(fv), "framework_charge": sets_of(q * fc),
                        "molecule_vdw": sets_of(pair.sum(1)), "molecule_charge": sets_of(coul.sum(1)),
                        "overlap": None})
    return out


def _exact_proposal(case, seed):
    """The samples, the first loss and its gradient; training itself follows the rounding of its own steps."""
    ff, cell, atoms = _unit(case, seed)
    n, count = case["samples"], min(case["samples"], case["batch"])
    state = (1 + seed + 0x9E3779B97F4A7C15 * np.arange(1, 3 * n + 1, dtype=np.uint64)).astype(np.uint64)
    z = (state ^ (state >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    z = z ^ (z >> np.uint64(31))
    u = ((z >> np.uint64(11)).astype(np.float64) * 2.0 ** -53).reshape(n, 3)
    dims = grid_points_for_spacing(cell, 0.25)
    dense = _exact_grid(ff, cell, atoms, ff.index("C_co2"), dims, _TRICUBIC)
    e, _ = _exact_interpolant(cell, dims, lambda index: dense[index], torch.from_numpy(u @ cell).cuda())
    targets = (-beta_of(300.0) * e).clamp_min(-15.0)
    _, weights, _ = _proposal_inputs(case, seed)
    w = torch.from_numpy(weights.astype(np.float64)).cuda().requires_grad_()
    s = torch.from_numpy(u[:count].astype(np.float32).astype(np.float64)).cuda()
    angle = 2.0 * math.pi * s[:, :, None] * torch.arange(1, 17, dtype=torch.float64, device="cuda")
    phi = torch.stack([angle.sin(), angle.cos()], 3).reshape(count, 96)
    h1 = torch.nn.functional.silu(phi @ w[:6144].reshape(64, 96).T + w[6144:6208])
    h2 = torch.nn.functional.silu(h1 @ w[6208:10304].reshape(64, 64).T + w[10304:10368])
    f = h2 @ w[10368:10432] + w[10432]
    loss = ((f - targets[:count].float().double()) ** 2).mean()
    loss.backward()
    return {"samples": torch.from_numpy(u).cuda(), "targets": targets, "loss": loss.detach(), "gradient": w.grad,
            "parameters": None, "log_density": None, "density": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "grids":
        ff, cell, atoms = _unit(case, seed)
        dims = grid_points_for_spacing(cell, case["spacing"])
        return [_exact_grid(ff, cell, atoms, p, dims, _TRICUBIC).reshape(-1)
                for p in (ff.index("C_co2"), ff.index("O_co2"), None)]
    if kind == "quintic":
        ff, cell, atoms = _unit(case, seed)
        dims = grid_points_for_spacing(cell, case["spacing"])
        probe = None if case["ewald"] else ff.index("C_co2")
        return _exact_grid(ff, cell, atoms, probe, dims, _TRIQUINTIC).reshape(-1)
    call = {"moves": _exact_moves, "trials": _exact_trials, "gridtest": _exact_gridtest, "full": _exact_full,
            "batch": _exact_batch, "proposal": _exact_proposal}.get(kind)
    # a Monte Carlo run has no other value than its own sequence of moves
    return call(case, seed) if call else None
