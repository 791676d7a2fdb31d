"""The mixture kernel at its edges: deletions that take the last molecule of the list, and a k-range that only just fits."""

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.gcmc import beta_of, co2_component, fugacity_of, n2_component
from raspa3_b200.mixture import molecules_as_atoms
from raspa3_b200.synthetic import synthetic_forcefield
from test_gcmc_gpu import empty_framework

pytestmark = pytest.mark.gpu
CELL = np.diag([26.0, 27.5, 25.0])


@pytest.fixture(scope="module")
def ctx():
    c = native.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("blocks,swap_only", [(1, True), (5, True), (3, False)])
def test_deletion_of_the_last_molecule(ctx, blocks, swap_only):
    """At a loading of one or two, most deletions take the last molecule, which no other is moved into the place of. The
    counts follow the accepted swaps, and the structure factors that the moves changed are those of the molecules that are
    there: 1e-9, 6,000 updates of FP64 sums of 18 unit phasors (each off by a few 1e-15)."""
    ff = synthetic_forcefield(charges=True, alpha=0.265, kmax=5)
    system = native.System(ctx, ff, CELL, empty_framework())
    ew = native.Ewald(ctx, ff, CELL)
    ew.set_framework(empty_framework())
    comps = [co2_component(), n2_component()]
    mx = native.Mixture(system, ew, comps, beta_of(300.0), [fugacity_of(1.5e5)] * 2, np.zeros((0, 3, 3)),
                        np.zeros(0, dtype=np.int32), max_molecules=6, seed=blocks, n_blocks=blocks,
                        probabilities=(0.0, 0.0, 1.0, 0.0) if swap_only else (1.0, 1.0, 1.0, 1.0))
    mx.set_state(0.0, ew.structure_factors(2))
    deletions = 0
    for _ in range(20):
        mx.run(300, record=True)
        r = mx.results()
        assert r["status"] == 0
        xyz, comp = mx.positions()
        assert len(comp) == sum(r["n_molecules"]) == r["accepted"][2] - r["accepted"][3]
        assert [int(np.sum(comp == c)) for c in range(2)] == list(r["n_molecules"][:2])
        deletions = r["accepted"][3]
        if len(comp):
            ew.full(molecules_as_atoms(ff, comps, xyz, comp), [3] * len(comp))
        ref = ew.structure_factors(0 if len(comp) else 2)
        assert np.max(np.abs(mx.structure_factors() - ref)) <= 1e-9 * max(1.0, np.max(np.abs(ref)))
    assert deletions > 50
    mx.close()
    ew.close()
    system.close()


# one CTA with 6,347 and 5,669 k-vectors and the tables of 3 and 6 orientations: 211 KB of shared memory beside the kernel's
# own, of 227 in all
@pytest.mark.parametrize("kmax,orientations", [((11, 11, 11), 3), ((9, 10, 13), 6)])
def test_largest_k_range_of_one_cta(ctx, kmax, orientations):
    """Created and run; the structure factors are those of the molecules that are there (1e-9, as above)."""
    ff = synthetic_forcefield(charges=True, alpha=0.265, kmax=max(kmax), sphere=False)
    ff.kmax = kmax
    system = native.System(ctx, ff, CELL, empty_framework())
    ew = native.Ewald(ctx, ff, CELL)
    ew.set_framework(empty_framework())
    comps = [co2_component(), n2_component()]
    mx = native.Mixture(system, ew, comps, beta_of(300.0), [fugacity_of(1e6)] * 2, np.zeros((0, 3, 3)),
                        np.zeros(0, dtype=np.int32), max_molecules=60, seed=4, n_blocks=1, n_orient=orientations)
    mx.set_state(0.0, ew.structure_factors(2))
    mx.run(2000, record=True)
    r = mx.results()
    xyz, comp = mx.positions()
    assert r["status"] == 0 and len(comp) > 4
    ew.full(molecules_as_atoms(ff, comps, xyz, comp), [3] * len(comp))
    ref = ew.structure_factors(0)
    assert np.max(np.abs(mx.structure_factors() - ref)) <= 1e-9 * max(1.0, np.max(np.abs(ref)))
    mx.close()
    ew.close()
    system.close()
