"""The Ewald kernels at the edges of their dispatch, against the FP64 oracle.

Tolerance 1e-9 of the largest of 1 and the value: a structure factor is a sum of at most 2,112 weighted phasors whose
arguments 2 pi k.s (|k.s| <= 104) are rounded at 2^-53 of themselves, so each phasor is off by at most 8e-14 and the sum
by 2e-10; the energies sum squares of those over the k-vectors with weights that fall off as exp(-k^2)."""

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.forcefield import COULOMBIC_CONVERSION_FACTOR, make_atoms
from raspa3_b200.synthetic import (CO2_NAMES, CO2_OFFSETS, random_molecules, random_rotation, rigid_molecule,
                                   synthetic_forcefield)

pytestmark = pytest.mark.gpu

TERMS = ("ewald_fourier", "ewald_self", "ewald_exclusion")
BOX = np.diag([31.0, 29.5, 33.2])
SKEW = np.array([[30.0, 0.0, 0.0], [6.0, 29.0, 0.0], [-4.0, 7.0, 31.0]])


@pytest.fixture(scope="module")
def ctx():
    c = native.Context(0)
    yield c
    c.close()


def forcefield(kmax, sphere=True):
    ff = synthetic_forcefield(charges=True, alpha=0.265, kmax=max(kmax), sphere=False)
    ff.kmax = tuple(kmax)
    if sphere:
        ff.use_sphere_kvectors()
    return ff


def close(a, b, what):
    assert abs(a - b) <= 1e-9 * max(1.0, abs(b)), (what, a, b)


# kmax_z 4, 5, 6 and 12 take 5, 6, 7 and 2 x 7 values of |kz| per thread; 2, 3, 85 and 86 molecules are 6, 9, 255 and 258
# atoms: one chunk and two, the own terms on the host and on the device
@pytest.mark.parametrize("kmax,sphere,cell,molecules,rest", [
    ((1, 1, 1), False, BOX, 1, 0), ((4, 4, 4), True, BOX, 2, 0), ((5, 5, 5), True, SKEW, 3, 2),
    ((6, 3, 6), False, BOX, 85, 0), ((3, 7, 2), False, SKEW, 86, 1), ((12, 12, 12), True, BOX, 86, 0),
    ((2, 2, 13), False, SKEW, 704, 0), ((8, 8, 8), True, BOX, 0, 0)])
def test_full_recompute_and_framework(ctx, oracle, kmax, sphere, cell, molecules, rest):
    """`rest` molecules stand outside the molecule sizes: they have no exclusion terms."""
    ff = forcefield(kmax, sphere)
    ew = native.Ewald(ctx, ff, cell)
    fw = random_molecules(ff, cell, 43, seed=8)
    ew.set_framework(fw)
    s_rigid = oracle.ewald_rigid(ff, cell, fw)
    np.testing.assert_allclose(ew.structure_factors(2), s_rigid, rtol=0, atol=1e-9)
    atoms = random_molecules(ff, cell, molecules, seed=molecules)
    scaled = rigid_molecule(ff, CO2_NAMES, CO2_OFFSETS, np.array([3.0, 4.0, 5.0]), random_rotation(np.random.default_rng(1)),
                            molecules, lam=0.7)
    atoms = np.concatenate([atoms, scaled]) if molecules > 3 else atoms
    sizes = [3] * (len(atoms) // 3 - rest)
    e = ew.full(atoms, sizes)
    ref, stored = oracle.ewald_fourier_energy(ff, cell, atoms, sizes, s_rigid=s_rigid)
    for k in TERMS:
        close(e[k], ref[k], k)
    s = ew.structure_factors(0)
    np.testing.assert_allclose(s[0::2], stored[0::10], rtol=0, atol=1e-9)
    np.testing.assert_allclose(s[1::2], stored[1::10], rtol=0, atol=1e-9)
    ew.close()


# 297 to 3,796 k-vectors are 2 to 15 blocks, each of which gives its own sums to the host; 17,328 are 68, whose sums the last
# one adds (from 65 on); up to 16 atoms travel in the launch's parameters and are one tile of the phase tables
@pytest.mark.parametrize("kmax,sphere,cell", [((5, 5, 5), True, BOX), ((8, 8, 8), True, SKEW), ((8, 8, 8), False, BOX),
                                              ((12, 12, 12), True, SKEW), ((1, 100, 1), False, BOX),
                                              ((20, 20, 20), True, BOX)])
@pytest.mark.parametrize("new,old,groups", [(0, 1, 0), (1, 1, 0), (3, 2, 0), (40, 41, 0), (1, 1, 1), (3, 3, 4)])
def test_difference(ctx, oracle, kmax, sphere, cell, new, old, groups):
    """`new` and `old` molecules; with groups the first is fractional."""
    ff = forcefield(kmax, sphere)
    ew = native.Ewald(ctx, ff, cell, n_groups=groups)
    rng = np.random.default_rng(new + old)

    def molecules(n, seed):
        mols = random_molecules(ff, cell, n, seed=seed)
        if groups and n:
            mols[:3] = rigid_molecule(ff, CO2_NAMES, CO2_OFFSETS, rng.random(3) @ cell, random_rotation(rng), 0, lam=0.6,
                                      group=groups, fractional=True)
        return mols

    b = molecules(old, 4)
    atoms = np.concatenate([b, random_molecules(ff, cell, 10, seed=3, first_id=old)])
    ew.full(atoms, [3] * (len(atoms) // 3))
    _, stored = oracle.ewald_fourier_energy(ff, cell, atoms, [3] * (len(atoms) // 3))
    a = molecules(new, 5)
    e = ew.delta(a, b)
    ref, trial = oracle.ewald_delta(ff, cell, stored, a, b)
    for k in TERMS:
        close(e[k], ref[k], k)
    for x, y in zip(e["dudlambda_ewald"], ref["dudlambda_ewald"]):
        close(x, y, "dudlambda")
    t = ew.structure_factors(1).reshape(-1, 1 + groups, 2)
    np.testing.assert_allclose(t, trial.reshape(-1, 5, 2)[:, :1 + groups], rtol=0, atol=1e-9)
    ew.close()


@pytest.mark.parametrize("kmax,sphere,systems", [((1, 1, 1), False, 1), ((3, 3, 13), False, 2), ((6, 6, 3), True, 5)])
def test_batch(ctx, oracle, kmax, sphere, systems):
    """One system and few; groups of |kz| that the runs do not fill; atom counts of every parity. The batch gives the
    Fourier sum alone: the oracle's correction for a change of the net charge is taken off."""
    ff = forcefield(kmax, sphere)
    ew = native.Ewald(ctx, ff, BOX)
    batch = native.EwaldBatch(ew, systems)
    stored, atoms, n_new, n_old = [], make_atoms(np.zeros((7 * systems, 3)), np.zeros(7 * systems, np.uint16),
                                                 np.zeros(7 * systems)), [], []
    for s in range(systems):
        mols = random_molecules(ff, BOX, 4, seed=s)
        ew.full(mols, [3] * 4)
        batch.set(s)
        assert np.array_equal(batch.get(s, 0), ew.structure_factors(0))
        stored.append(oracle.ewald_fourier_energy(ff, BOX, mols, [3] * 4)[1])
        new, old = random_molecules(ff, BOX, 2, seed=50 + s)[:s % 5], mols[:3 - s % 2]
        atoms[7 * s:7 * s + len(new)] = new
        atoms[7 * s + len(new):7 * s + len(new) + len(old)] = old
        n_new.append(len(new))
        n_old.append(len(old))
    for sweep in range(2):  # the second on the other of the two buffers of the systems accepted by the first
        d = batch.delta(atoms, 7, n_new, n_old)
        trials = []
        for s in range(systems):
            new = atoms[7 * s:7 * s + n_new[s]]
            ref, trial = oracle.ewald_delta(ff, BOX, stored[s], new, atoms[7 * s + n_new[s]:7 * s + n_new[s] + n_old[s]])
            moved = atoms[7 * s:7 * s + n_new[s] + n_old[s]]
            charge = float(np.sum(moved["charge"][:n_new[s]]) - np.sum(moved["charge"][n_new[s]:]))
            u_ion = -(ew.single_ion_sum - COULOMBIC_CONVERSION_FACTOR * ff.ewald_alpha / np.sqrt(np.pi))
            close(d[s], ref["ewald_fourier"] - u_ion * charge ** 2, s)
            t = batch.get(s, 1).reshape(-1, 2)
            np.testing.assert_allclose(t, trial.reshape(-1, 5, 2)[:, 0], rtol=0, atol=1e-9)
            trials.append(trial)
        accept = np.arange(systems) % 2 == 0
        batch.accept(accept)
        for s in range(systems):
            stored[s] = trials[s] if accept[s] else stored[s]
            np.testing.assert_allclose(batch.get(s, 0).reshape(-1, 2), stored[s].reshape(-1, 5, 2)[:, 0], rtol=0, atol=1e-9)
    batch.close()
    ew.close()
