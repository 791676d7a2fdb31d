"""FP64 grid kernels at the edges of their bricks and of their dispatch rule, against the FP64 oracle.

Tolerance: a channel is a sum of N terms whose largest are M times the sum, evaluated with a few ulp per term, so its
error is about (N + 8) M 2^-52 relative: N = 400 pairs and M up to 1e4 (the cancelling Ewald terms) give 1e-9."""

import math

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.forcefield import KELVIN_TO_ENERGY
from raspa3_b200.synthetic import synthetic_forcefield, synthetic_framework

pytestmark = pytest.mark.gpu

TOL = 1e-9


@pytest.fixture(scope="module")
def ctx():
    c = native.Context(0)
    yield c
    c.close()


def worst(got, ref, channels):
    """max |got - ref| / max(|ref|, RMS of the channel) over the points below 1e4 K; the clamped points exactly."""
    g, r = got.reshape(-1, channels), ref.reshape(-1, channels)
    ok = np.abs(r[:, 0]) < 1e4 * KELVIN_TO_ENERGY
    if not ok.any():
        return 0.0
    rms = np.sqrt(np.mean(r[ok] ** 2, axis=0)) + 1e-300
    return float((np.abs(g[ok] - r[ok]) / np.maximum(np.abs(r[ok]), rms)).max())


# one brick short of, equal to and one point beyond the 8 x 8 x 4 brick and its 4 x 4 x 2 warps; the smallest grid
@pytest.mark.parametrize("dims", [(2, 2, 2), (8, 8, 4), (9, 7, 5), (17, 3, 10)])
@pytest.mark.parametrize("grid_type", [0, 1, 2, 3])
def test_tricubic_fp64_bricks(ctx, oracle, dims, grid_type):
    ff = synthetic_forcefield(charges=True)
    cell, atoms = synthetic_framework(ff, seed=11)
    probe = ff.index("C_co2")
    for cutoff in (12.0, 6.5):  # the reference's supercell, and one that clips pairs
        got, stats = ctx.grid_build(grid_type, ff, cell, atoms, probe, cutoff, dims, native.PRECISION_FP64,
                                    count_pairs=True)
        ref = oracle.make_grid(grid_type, ff, cell, atoms, probe, cutoff, dims)
        assert worst(got, ref, 8) < TOL
        assert stats["pair_count"] == oracle.grid_pair_count(grid_type, ff, cell, atoms, probe, cutoff, dims)


# alpha rc on both sides of 6, where the Ewald terms leave the polynomial for the library's erfc
@pytest.mark.parametrize("alpha", [0.1, 0.4999, 0.5001, 0.9])
def test_ewald_fp64_alpha(ctx, oracle, alpha):
    ff = synthetic_forcefield(charges=True, alpha=alpha)
    cell, atoms = synthetic_framework(ff, seed=12)
    dims = (9, 8, 6)
    got, _ = ctx.grid_build(1, ff, cell, atoms, 0, 12.0, dims, native.PRECISION_FP64)
    assert worst(got, oracle.make_grid(1, ff, cell, atoms, 0, 12.0, dims), 8) < TOL


def test_fp64_pair_of_probes_equals_single_builds(ctx):
    torch = pytest.importorskip("torch")
    ff = synthetic_forcefield(charges=True)
    cell, atoms = synthetic_framework(ff, seed=13)
    dims = (19, 18, 13)
    probes = [ff.index("C_co2"), ff.index("O_co2"), ff.index("CH4")]
    out = [torch.empty(8 * math.prod(dims), dtype=torch.float64, device="cuda") for _ in probes]
    ctx.grid_build_set(ff, cell, atoms, 12.0, dims, native.PRECISION_FP64, [0, 0, 0], probes,
                       [o.data_ptr() for o in out])
    ctx.synchronize()
    for probe, o in zip(probes, out):
        single, _ = ctx.grid_build(0, ff, cell, atoms, probe, 12.0, dims, native.PRECISION_FP64)
        assert worst(o.cpu().numpy(), single, 8) < 1e-13  # the same pair terms in the same order


# the triquintic kernel's brick is 8 x 4 x 4; alpha rc beyond 6 takes the library's erfc
@pytest.mark.parametrize("dims", [(2, 2, 2), (8, 4, 4), (9, 5, 3)])
@pytest.mark.parametrize("grid_type,alpha", [(0, 0.265), (1, 0.265), (1, 0.6)])
@pytest.mark.parametrize("reference_rectangular", [False, True])
def test_triquintic_fp64_bricks(ctx, oracle, dims, grid_type, alpha, reference_rectangular):
    ff = synthetic_forcefield(charges=True, alpha=alpha)
    cell, atoms = synthetic_framework(ff, seed=14)
    probe = ff.index("C_co2")
    for cutoff in (12.0, 6.5):
        got, stats = ctx.grid_build_triquintic(grid_type, ff, cell, atoms, probe, cutoff, dims,
                                               reference_rectangular=reference_rectangular, count_pairs=True)
        ref = oracle.make_grid_triquintic(grid_type, ff, cell, atoms, probe, cutoff, dims,
                                          reference_rectangular=reference_rectangular)
        assert worst(got, ref, 27) < TOL
        assert stats["pair_count"] == oracle.grid_pair_count(grid_type, ff, cell, atoms, probe, cutoff, dims)


def _grid_test(ctx, ff, cell, atoms, dims, bufs, points, scheme):
    probe = ff.index("C_co2")
    call = ctx.grid_validate_triquintic if scheme == 27 else ctx.grid_validate
    return call(ff, cell, atoms, cell, probe, dims, bufs[0].data_ptr(), bufs[1].data_ptr(), 0.70, 1.0 / 300.0,
                points=points)


# one point, the edges of warps (32), blocks (128) and bins, and enough points that the image lists are not split
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 700, 4100])
@pytest.mark.parametrize("scheme,alpha", [(8, 0.265), (8, 0.6), (27, 0.265)])
def test_grid_test_point_counts(ctx, oracle, n, scheme, alpha):
    """Sums of w x within 1e-9 of sqrt(sum w x^2 sum w), the accuracy of the pair sums above. The interpolated side of
    the triquintic scheme is left out: the oracle sums the reference's monomial form, whose own rounding at cells next
    to clamped points is larger."""
    torch = pytest.importorskip("torch")
    ff = synthetic_forcefield(charges=True, alpha=alpha)
    cell, atoms = synthetic_framework(ff, seed=15)
    dims = (21, 20, 14)
    host = []
    for gt, probe in ((0, ff.index("C_co2")), (1, 0)):
        if scheme == 27:
            host.append(ctx.grid_build_triquintic(gt, ff, cell, atoms, probe, 12.0, dims)[0])
        else:
            host.append(ctx.grid_build(gt, ff, cell, atoms, probe, 12.0, dims, native.PRECISION_FP64)[0])
    bufs = [torch.from_numpy(h).cuda() for h in host]
    points = np.random.default_rng(n).random((n, 3))
    got = _grid_test(ctx, ff, cell, atoms, dims, bufs, points, scheme)
    check = oracle.grid_validate_triquintic if scheme == 27 else oracle.grid_validate
    ref = check(ff, cell, atoms, cell, ff.index("C_co2"), dims, host[0], host[1], 0.70, 1.0 / 300.0, points)
    assert got["n_points"] == ref[34] == n
    assert got["n_points_charge"] == ref[35]
    s = np.array(got["sums"])
    for base in (0, 17):
        o = np.asarray(ref[base:base + 17])
        scale = np.abs(o).copy()
        scale[[1, 2]] = np.sqrt(o[4] * o[0])
        scale[3] = o[4]
        for a in range(3):
            scale[[5 + a, 8 + a]] = np.sqrt(o[14 + a] * o[0])
            scale[11 + a] = o[14 + a]
        use = [0, 2, 4, 8, 9, 10, 14, 15, 16] if scheme == 27 else list(range(17))
        d = np.abs(s[base:base + 17] - o)
        assert np.all(d[use] <= 1e-9 * scale[use] + 1e-280), (base, s[base:base + 17], o)


def test_grid_test_in_rounds(ctx):
    """More points than one round holds: the sums are those of the two parts (rounding of 2^21 added terms)."""
    torch = pytest.importorskip("torch")
    ff = synthetic_forcefield(charges=True)
    cell, atoms = synthetic_framework(ff, seed=16)
    dims = (21, 20, 14)
    bufs = []
    for gt, probe in ((0, ff.index("C_co2")), (1, 0)):
        bufs.append(torch.from_numpy(ctx.grid_build(gt, ff, cell, atoms, probe, 12.0, dims,
                                                    native.PRECISION_FP64)[0]).cuda())
    n = (1 << 21) + 1000
    points = np.random.default_rng(3).random((n, 3))
    whole = _grid_test(ctx, ff, cell, atoms, dims, bufs, points, 8)
    parts = [_grid_test(ctx, ff, cell, atoms, dims, bufs, p, 8) for p in (points[:777777], points[777777:])]
    assert whole["n_points"] == n
    assert whole["n_points_charge"] == sum(p["n_points_charge"] for p in parts)
    a, b = np.array(whole["sums"]), np.array(parts[0]["sums"]) + np.array(parts[1]["sums"])
    scale = np.maximum(np.abs(a), np.repeat([np.sqrt(a[0] * a[4]), np.sqrt(a[17] * a[21])], 17))
    assert np.all(np.abs(a - b) <= 1e-11 * scale)
