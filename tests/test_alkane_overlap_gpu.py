"""Deletion of a chain whose Rosenbluth weight vanishes: Pacc = N / (beta f V) W_IG / W is infinite, so the first deletion
that is tried is accepted, however far below zero the exponent lies."""

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.alkane import AlkaneChain, AlkaneSystem, alkane_forcefield
from raspa3_b200.forcefield import make_atoms
from raspa3_b200.gcmc import beta_of

pytestmark = pytest.mark.gpu


def test_vanishing_weight():
    """One trial per step, and a bead 0.2 to 0.9 A from a framework atom: exponents of -1e4 to -1e18, which FP32 rounds
    by up to 1e10. The overlap criterion is above all of them, and the fugacity lets no insertion through."""
    ff = alkane_forcefield()
    ff.overlap_criteria = 1e30
    cell = np.diag([30.0, 30.0, 30.0])
    fw = make_atoms(np.array([[5.0, 5.0, 5.0]]), ff.index("O"), 0.0)
    distances = np.linspace(0.2, 0.9, 48)
    systems = [AlkaneSystem(cell=cell, framework=fw, chain=AlkaneChain(2, n_first=1, n_directions=1), beta=beta_of(300.0),
                            fugacity=1e-200, max_molecules=4, p_translation=0.0, p_swap=1.0) for _ in distances]
    ctx = native.Context(0)
    a = native.Alkane(ctx, ff, systems, seed=3)
    for i, r in enumerate(distances):
        a.set_positions(i, np.array([[5.0 + r, 5.0, 5.0], [5.0 + r + 1.54, 5.0, 5.0]]))
    a.run(30, record=True)  # at least one of 30 swaps is a deletion (but for one run in 1e9)
    results = a.results()
    assert all(r["attempted"][3] > 0 for r in results)
    assert [r["accepted"][3] for r in results] == [1] * len(results)
    assert all(r["n_molecules"] == 0 for r in results)
    ctx.close()
