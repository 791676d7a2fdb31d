"""The GCMC kernel's variants: structure factors in shared memory and, for sets too large for it, in global memory;
molecules of one atom and of three; with and without charges. Every chain's running energy equals the oracle's
recomputation of its last configuration: 1e-6, as for the drift of the reference's Monte Carlo runs."""

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.gcmc import beta_of, co2_component, fugacity_of, methane_component
from raspa3_b200.synthetic import synthetic_forcefield
from test_gcmc_gpu import empty_framework, recompute

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = native.Context(0)
    yield c
    c.close()


# kmax 6 and 9 of the full half-box and 14 of the sphere have 1,182, 3,609 and 6,062 k-vectors: 38, 115 and 194 KB of
# structure factors and changes; 50 KB is the most that stays in shared memory
@pytest.mark.parametrize("kmax,sphere,component,chains", [(1, False, co2_component, 3), (6, False, co2_component, 5),
                                                          (9, False, co2_component, 5), (14, True, co2_component, 3),
                                                          (None, True, methane_component, 7)])
def test_running_energy(ctx, oracle, kmax, sphere, component, chains):
    charges = kmax is not None
    ff = synthetic_forcefield(charges=charges, alpha=0.265, kmax=kmax or 8, sphere=sphere)
    cell = np.diag([26.0, 27.5, 25.0])
    comp = component()
    system = native.System(ctx, ff, cell, empty_framework())
    ew = native.Ewald(ctx, ff, cell) if charges else None
    if ew:
        ew.set_framework(empty_framework())
    g = native.Gcmc(system, ew, comp, beta_of(300.0), fugacity_of(6e6), n_chains=chains, seed=5)
    g.run(1500, record=True)
    res = g.results()
    assert max(r["n_molecules"] for r in res) > 2
    for c in range(chains):
        e = recompute(oracle, ff, cell, comp, g.positions(c))
        assert abs(e - res[c]["energy"]) <= 1e-6 * max(1.0, abs(e)), (c, e, res[c]["energy"])
