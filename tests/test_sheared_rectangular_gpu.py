"""Cells given as rectangular (rg_box.triclinic = 0) whose vectors are not along the axes: points, images and fractional
coordinates are by the full vectors, as in the triclinic branch; derivatives and minimum images by the diagonal."""

import math

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.forcefield import box_struct, make_atoms, positions_of
from raspa3_b200.synthetic import random_molecules, synthetic_forcefield

pytestmark = pytest.mark.gpu
CELL = np.array([[17.0, 0.0, 0.0], [5.0, 16.0, 0.0], [-8.0, 6.0, 15.0]])


@pytest.fixture(scope="module")
def ctx():
    c = native.Context(0)
    yield c
    c.close()


@pytest.fixture()
def rectangular(monkeypatch):
    monkeypatch.setattr(native, "box_struct", lambda cell: box_struct(cell, triclinic=False))


def framework(ff, n=40):
    rng = np.random.default_rng(9)
    types = np.where(np.arange(n) % 3 == 0, ff.index("T"), ff.index("O")).astype(np.uint16)
    return make_atoms(rng.random((n, 3)) @ CELL, types, np.where(types == ff.index("T"), 2.05, -1.025))


def lennard_jones(ff, atoms, probe, dims, rc):
    """Energy sums and the number of pairs at the grid points, over all images within rc (FP64, numpy)."""
    g = [np.arange(n) / (n - 1) for n in dims]
    k, j, i = np.meshgrid(g[2], g[1], g[0], indexing="ij")
    points = np.stack([i, j, k], -1).reshape(-1, 3) @ CELL
    shifts = np.stack(np.meshgrid(*[np.arange(-3, 4)] * 3, indexing="ij"), -1).reshape(-1, 3) @ CELL
    energy, pairs = np.zeros(len(points)), 0
    for a, r in zip(atoms, positions_of(atoms)):
        eps = ff.epsilon[probe, a["type"]]
        if eps == 0.0:
            continue
        d = points[:, None] - (r + shifts)[None]
        rr = np.maximum((d * d).sum(-1), 0.1)
        inside = rr < rc * rc
        t = (ff.sigma[probe, a["type"]] ** 2 / rr) ** 3
        energy += np.where(inside, 4.0 * eps * t * (t - 1.0) - ff.shift[probe, a["type"]], 0.0).sum(1)
        pairs += int(inside.sum())
    return energy, pairs


# the grid's own pair of bricks, ragged ones, and a spacing of several Angstrom; tricubic and triquintic
@pytest.mark.parametrize("scheme", [8, 27])
@pytest.mark.parametrize("dims", [(9, 5, 5), (17, 9, 13), (4, 3, 3)])
def test_lennard_jones_grid(ctx, rectangular, scheme, dims):
    """Every pair within the cutoff is there: equal counts, and energies to 1e-9 (some 300 terms of a few ulp, the largest
    up to 1e4 times the sum)."""
    ff = synthetic_forcefield(charges=True)
    atoms = framework(ff)
    probe = ff.index("C_co2")
    build = ctx.grid_build_triquintic if scheme == 27 else ctx.grid_build
    got, stats = build(0, ff, CELL, atoms, probe, 12.0, dims, count_pairs=True)
    energy, pairs = lennard_jones(ff, atoms, probe, dims, ff.cutoff_framework_vdw)
    assert stats["pair_count"] == pairs
    e = got.reshape(-1, scheme)[:, 0]
    open_ = energy <= ff.overlap_criteria
    assert open_.sum() > len(energy) // 8
    scale = np.maximum(np.abs(energy), math.sqrt(np.mean(energy[open_] ** 2)))
    assert np.max((np.abs(e - energy) / scale)[open_]) < 1e-9


# the atoms' own terms of 255 and 258 atoms: on the host, and on the device for a cell along the axes
@pytest.mark.parametrize("molecules", [85, 86])
def test_ewald_exclusion(ctx, oracle, rectangular, monkeypatch, molecules):
    """Self and exclusion energies against the oracle's: 1e-9, as for the other recomputes."""
    obox = oracle.obox
    monkeypatch.setattr(oracle, "obox", lambda cell, triclinic=None: obox(cell, False))
    ff = synthetic_forcefield(charges=True, kmax=4)
    mols = random_molecules(ff, CELL, molecules, seed=5)
    shift = np.random.default_rng(2).integers(-1, 2, size=(len(mols), 3)) @ CELL  # split over the cell's faces
    for a, axis in enumerate("xyz"):
        mols[axis] += shift[:, a]
    ew = native.Ewald(ctx, ff, CELL)
    got = ew.full(mols, [3] * molecules)
    ref, _ = oracle.ewald_fourier_energy(ff, CELL, mols, [3] * molecules)
    for k in ("ewald_self", "ewald_exclusion"):
        assert abs(got[k] - ref[k]) <= 1e-9 * max(1.0, abs(ref[k])), (k, got[k], ref[k])
    ew.close()
