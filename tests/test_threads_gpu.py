"""Two host threads, each with a context of its own, launch the same kernels with different amounts of shared memory: the
limit of a kernel's shared memory is the device's, so one thread must not lower it between another's setting and launch
(the launch would be refused). Every result is that of the same calls made by one thread."""

import threading

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.gcmc import beta_of, co2_component, fugacity_of
from raspa3_b200.synthetic import random_molecules, synthetic_forcefield
from test_gcmc_gpu import empty_framework

pytestmark = pytest.mark.gpu
CELL = np.diag([26.0, 27.5, 25.0])


def gcmc_runs(kmax, rounds):
    ctx = native.Context(0)
    ff = synthetic_forcefield(charges=True, alpha=0.265, kmax=kmax)
    system = native.System(ctx, ff, CELL, empty_framework())
    ew = native.Ewald(ctx, ff, CELL)
    ew.set_framework(empty_framework())
    g = native.Gcmc(system, ew, co2_component(), beta_of(300.0), fugacity_of(2e6), n_chains=2, seed=kmax)
    for _ in range(rounds):
        g.run(2, record=True)
    out = [r["energy"] for r in g.results()]
    ctx.close()
    return out


def recomputes(kmax, groups, rounds):
    ctx = native.Context(0)
    ff = synthetic_forcefield(charges=True, alpha=0.265, kmax=kmax)
    mols = random_molecules(ff, CELL, 12, seed=kmax)
    ew = native.Ewald(ctx, ff, CELL, n_groups=groups)
    out = [ew.full(mols, [3] * 12)["ewald_fourier"] for _ in range(rounds)]
    ctx.close()
    return out


def batches(kmax, rounds):
    ctx = native.Context(0)
    ff = synthetic_forcefield(charges=True, alpha=0.265, kmax=kmax)
    mols = random_molecules(ff, CELL, 12, seed=kmax)
    ew = native.Ewald(ctx, ff, CELL)
    ew.full(mols, [3] * 12)
    batch = native.EwaldBatch(ew, 2)
    for s in range(2):
        batch.set(s)
    new = mols[:6].copy()
    new["x"] += 0.2
    atoms = np.concatenate([new, mols[:6], new, mols[:6]])
    six = np.full(2, 6, dtype=np.int32)
    out = [batch.delta(atoms, 12, six, six) for _ in range(rounds)]
    ctx.close()
    return np.concatenate(out)


# shared memory of 13 and 44 KB for the GCMC; tables of more and fewer k-vectors and atoms for the Ewald sums
@pytest.mark.parametrize("call,first,second", [(gcmc_runs, (4, 1500), (8, 1500)),
                                               (recomputes, (4, 0, 1500), (20, 0, 1500)),
                                               (recomputes, (4, 1, 1500), (40, 1, 800)),
                                               (batches, (4, 1500), (40, 400))])
def test_two_threads(call, first, second):
    alone = [call(*first), call(*second)]
    together, errors = [None, None], []

    def work(i, args):
        try:
            together[i] = call(*args)
        except Exception as e:  # noqa: BLE001 - reported by the assertion below
            errors.append(str(e))

    threads = [threading.Thread(target=work, args=(i, a)) for i, a in enumerate((first, second))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, b in zip(alone, together):
        assert np.array_equal(a, b)
