"""Every point of the FP64 grids at the edges of their bricks, against the FP64 oracle: points below the overlap criterion by
value, clamped ones as the reference clamps them (interpolation_energy_grid.cpp:3847-3874, 3937-3955).

Tolerance 1e-9 of the larger of the value and the channel's RMS over the points below 1e4 K (over all that are not
clamped where there is none), as in test_grid_edges_gpu.py; first derivatives of clamped points to 1e-9 of the criterion
that they are clamped to."""

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.forcefield import KELVIN_TO_ENERGY, positions_of
from raspa3_b200.synthetic import synthetic_forcefield, synthetic_framework

pytestmark = pytest.mark.gpu
TOL = 1e-9


@pytest.fixture(scope="module")
def ctx():
    c = native.Context(0)
    yield c
    c.close()


def open_framework(ff, seed):
    """The synthetic framework moved so that the cell's origin, the only point of a 2 x 2 x 2 grid, is in its widest void."""
    cell, atoms = synthetic_framework(ff, seed=seed)
    lengths = np.diag(cell)
    g = np.stack(np.meshgrid(*[np.arange(12) / 12] * 3, indexing="ij"), -1).reshape(-1, 3) * lengths
    d = g[:, None] - positions_of(atoms)[None]
    d -= lengths * np.round(d / lengths)
    origin = g[np.argmax((d * d).sum(-1).min(1))]
    for a, axis in enumerate("xyz"):
        atoms[axis] = np.mod(atoms[axis] - origin[a], lengths[a])
    return cell, atoms


def check(got, ref, channels, criterion):
    g, r = got.reshape(-1, channels), ref.reshape(-1, channels)
    clamped = r[:, 0] == 2.0 * criterion
    assert np.array_equal(g[:, 0] == 2.0 * criterion, clamped)
    assert np.all(np.abs(g[clamped, 1:4] - r[clamped, 1:4]) <= TOL * criterion)
    assert np.all(g[clamped, 4:] == 0.0) and np.all(r[clamped, 4:] == 0.0)
    assert not clamped.all()
    low = np.abs(r[:, 0]) < 1e4 * KELVIN_TO_ENERGY
    scale = np.maximum(np.abs(r), np.sqrt(np.mean(r[low if low.any() else ~clamped] ** 2, axis=0)))
    assert np.all((np.abs(g - r) <= TOL * scale)[~clamped])
    return int(low.sum()), int(clamped.sum())


# one brick short of, equal to and one point beyond the 8 x 8 x 4 brick and its 4 x 4 x 2 warps; the smallest grid
@pytest.mark.parametrize("dims", [(2, 2, 2), (8, 8, 4), (9, 7, 5), (17, 3, 10), (25, 24, 17)])
@pytest.mark.parametrize("grid_type", [0, 1, 2, 3])
@pytest.mark.parametrize("cutoff", [12.0, 6.5])
def test_tricubic(ctx, oracle, dims, grid_type, cutoff):
    ff = synthetic_forcefield(charges=True)
    cell, atoms = open_framework(ff, 11)
    probe = ff.index("C_co2")
    got, _ = ctx.grid_build(grid_type, ff, cell, atoms, probe, cutoff, dims, native.PRECISION_FP64)
    low, clamped = check(got, oracle.make_grid(grid_type, ff, cell, atoms, probe, cutoff, dims), 8, ff.overlap_criteria)
    if grid_type in (0, 2) and dims == (25, 24, 17):
        assert low > 500 and clamped > 500


# the triquintic kernel's brick is 8 x 4 x 4; alpha rc beyond 6 takes the library's erfc
@pytest.mark.parametrize("dims", [(2, 2, 2), (8, 4, 4), (9, 5, 3), (25, 24, 17)])
@pytest.mark.parametrize("grid_type,alpha", [(0, 0.265), (1, 0.265), (1, 0.6)])
@pytest.mark.parametrize("cutoff", [12.0, 6.5])
def test_triquintic(ctx, oracle, dims, grid_type, alpha, cutoff):
    ff = synthetic_forcefield(charges=True, alpha=alpha)
    cell, atoms = open_framework(ff, 14)
    probe = ff.index("C_co2")
    got, _ = ctx.grid_build_triquintic(grid_type, ff, cell, atoms, probe, cutoff, dims)
    ref = oracle.make_grid_triquintic(grid_type, ff, cell, atoms, probe, cutoff, dims)
    low, clamped = check(got, ref, 27, ff.overlap_criteria)
    if grid_type == 0 and dims == (25, 24, 17):
        assert low > 500 and clamped > 500
