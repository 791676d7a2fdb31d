"""Device memory of the GCMC's structure factors: where they fit in shared memory, the change of a move is there only."""

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.gcmc import beta_of, co2_component, fugacity_of
from raspa3_b200.synthetic import synthetic_forcefield
from test_gcmc_gpu import empty_framework

pytestmark = pytest.mark.gpu


# 1,152 and 3,609 k-vectors: in shared memory, and in global memory with their change
@pytest.mark.parametrize("kmax,sphere,arrays", [(8, True, 1), (9, False, 2)])
def test_structure_factor_memory(kmax, sphere, arrays):
    torch = pytest.importorskip("torch")
    chains = 20000
    ff = synthetic_forcefield(charges=True, alpha=0.265, kmax=kmax, sphere=sphere)
    cell = np.diag([26.0, 27.5, 25.0])
    ctx = native.Context(0)
    system = native.System(ctx, ff, cell, empty_framework())
    ew = native.Ewald(ctx, ff, cell)
    ew.set_framework(empty_framework())
    one = 16 * ew.n_kvectors * chains
    other = chains * (8 * 3 * 32 + 300)  # positions, counts, energies and statistics
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    g = native.Gcmc(system, ew, co2_component(), beta_of(300.0), fugacity_of(1e6), n_chains=chains, seed=1,
                    max_molecules=8)
    used = before - torch.cuda.mem_get_info()[0]
    assert arrays * one <= used <= arrays * one + other + (64 << 20)
    g.run(5, record=True)
    assert len(g.results()) == chains
    ctx.close()
