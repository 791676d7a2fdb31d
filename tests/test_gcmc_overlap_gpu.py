"""Pairs whose (r^2 / sigma^2)^3 is too small for a reciprocal are overlaps like any other."""

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.gcmc import beta_of, co2_component, fugacity_of, methane_component
from raspa3_b200.synthetic import synthetic_forcefield
from test_gcmc_gpu import empty_framework

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("component", [methane_component, co2_component])
def test_vanishing_ratio_is_an_overlap(component):
    """With a huge sigma every pair within the cutoff overlaps, whatever the value: at 1e20 the ratio's cube is 1e-114 and
    the energy a large number, at 1e60 the cube is 0. The chains are then the same, number by number, and trials
    beyond the cutoff of all molecules are still accepted."""
    cell = np.diag([60.0, 60.0, 60.0])
    results = []
    for sigma in (1e20, 1e60):
        ff = synthetic_forcefield(charges=False)
        ff.sigma = np.full_like(ff.sigma, sigma)
        ff.shift = np.zeros_like(ff.shift)
        ctx = native.Context(0)
        system = native.System(ctx, ff, cell, empty_framework())
        g = native.Gcmc(system, None, component(), beta_of(300.0), fugacity_of(1e6), n_chains=8, seed=3)
        g.run(3000, record=True)
        results.append(g.results())
        ctx.close()
    assert all(r["n_molecules"] > 4 for r in results[0])
    assert results[0] == results[1]
