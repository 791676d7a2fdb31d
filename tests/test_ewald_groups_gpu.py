"""The recompute's own terms (self, exclusion, net charge) on both sides of their rule, with dU/dlambda groups and without
k-vectors, against the FP64 oracle.

Tolerance 1e-9 of the largest of 1 and the value, as for the other recomputes (test_ewald_edges_gpu.py); a group's derivative
is a sum of the same terms times weights of 1, so its scale is the largest energy."""

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.forcefield import make_atoms
from raspa3_b200.synthetic import CO2_NAMES, CO2_OFFSETS, random_rotation, rigid_molecule, synthetic_forcefield

pytestmark = pytest.mark.gpu
CELL = np.diag([41.0, 49.5, 43.2])


@pytest.fixture(scope="module")
def ctx():
    c = native.Context(0)
    yield c
    c.close()


def molecules(ff, n, per, groups, rng):
    """n chains of `per` charged atoms; the first ones, CO2, are fractional, one of each group."""
    com = rng.random((n, 1, 3)) @ CELL
    pos = (com + rng.normal(size=(n, per, 3))).reshape(-1, 3)
    atoms = make_atoms(pos, ff.index("O_co2"), 0.3 * rng.normal(size=len(pos)), molecule_ids=np.repeat(np.arange(n), per))
    first = [rigid_molecule(ff, CO2_NAMES, CO2_OFFSETS, rng.random(3) @ CELL, random_rotation(rng), n + g, lam=0.6,
                            group=g + 1, fractional=True) for g in range(groups)]
    return np.concatenate(first + [atoms]), [3] * groups + [per] * n


# 255 and 258 atoms; 1,299 and 1,302 pairs of three-atom molecules (with one group's); 1,215 and 1,305 pairs of larger ones;
# no pairs
@pytest.mark.parametrize("n,per", [(84, 3), (85, 3), (432, 3), (433, 3), (27, 10), (29, 10), (300, 1)])
@pytest.mark.parametrize("kmax,groups", [(5, 1), (5, 4), (0, 1), (0, 0)])
def test_own_terms(ctx, oracle, n, per, kmax, groups):
    ff = synthetic_forcefield(charges=True, alpha=0.265, kmax=kmax)
    atoms, sizes = molecules(ff, n, per, groups, np.random.default_rng(n + per))
    ew = native.Ewald(ctx, ff, CELL, n_groups=groups)
    got = ew.full(atoms, sizes)
    ref, _ = oracle.ewald_fourier_energy(ff, CELL, atoms, sizes)
    scale = max(1.0, *[abs(ref[k]) for k in ("ewald_fourier", "ewald_self", "ewald_exclusion")])
    for k in ("ewald_fourier", "ewald_self", "ewald_exclusion"):
        assert abs(got[k] - ref[k]) <= 1e-9 * max(1.0, abs(ref[k])), (k, got[k], ref[k])
    for g in range(groups):
        assert abs(got["dudlambda_ewald"][g] - ref["dudlambda_ewald"][g]) <= 1e-9 * scale, g
    ew.close()
