"""A context's calls stay in order across rg_ctx_set_stream: energy calls return when their results are there, with their
kernel's other stores possibly still under way, and a batch's S(k) is copied on the stream without a wait.

The same calls on one stream give the values to compare with, bit for bit: no sum depends on the stream."""

import ctypes

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.gcmc import beta_of, co2_component, fugacity_of
from raspa3_b200.synthetic import random_molecules, synthetic_forcefield
from test_gcmc_gpu import empty_framework

pytestmark = pytest.mark.gpu
CELL = np.diag([26.0, 27.5, 25.0])


@pytest.fixture()
def ctx():
    c = native.Context(0)
    yield c
    c.close()


@pytest.fixture()
def torch():
    return pytest.importorskip("torch")


def forcefield(kmax):
    return synthetic_forcefield(charges=True, alpha=0.265, kmax=kmax, sphere=False)


def moved(mols, k, step):
    new = mols[3 * k:3 * k + 3].copy()
    new["x"] += step
    return new, mols[3 * k:3 * k + 3]


def batch_energies(torch, switch):
    """64 systems set behind a run of some 100 ms, then a difference on another stream."""
    ctx = native.Context(0)
    ff = forcefield(8)
    system = native.System(ctx, ff, CELL, empty_framework())
    ew = native.Ewald(ctx, ff, CELL)
    mols = random_molecules(ff, CELL, 20, seed=1)
    ew.full(mols, [3] * 20)
    batch = native.EwaldBatch(ew, 64)
    g = native.Gcmc(system, ew, co2_component(), beta_of(300.0), fugacity_of(1e6), n_chains=64, seed=5)
    streams = [torch.cuda.Stream() for _ in range(2)]
    ctx.synchronize()
    ctx.set_stream(streams[0].cuda_stream)
    g.run(8000, record=False)
    for s in range(64):
        batch.set(s)
    if switch:
        ctx.set_stream(streams[1].cuda_stream)
    pairs = [moved(mols, s % 20, 0.1 + 0.01 * s) for s in range(64)]
    atoms = np.concatenate([np.concatenate(p) for p in pairs])
    three = np.full(64, 3, dtype=np.int32)
    out = batch.delta(atoms, 6, three, three)
    trial = np.concatenate([batch.get(s, 1) for s in (0, 63)])
    ctx.set_stream(None)
    ctx.close()
    return out, trial


def test_batch_set_behind_a_run(torch):
    for a, b in zip(batch_energies(torch, False), batch_energies(torch, True)):
        assert np.array_equal(a, b)


# kmax 8: 11 blocks post their own sums; kmax 16: 73 blocks, whose last one adds them and resets the counter
@pytest.mark.parametrize("kmax,groups", [(8, 0), (16, 0), (8, 2)])
def test_energies_on_alternating_streams(torch, kmax, groups):
    ff = forcefield(kmax)
    mols = random_molecules(ff, CELL, 90, seed=2)
    runs = []
    for switch in (False, True):
        ctx = native.Context(0)
        system = native.System(ctx, ff, CELL, empty_framework())
        system.set_molecules(mols)
        ew = native.Ewald(ctx, ff, CELL, n_groups=groups)
        streams = [torch.cuda.Stream() for _ in range(3)]
        out, calls = [], 0

        def turn():
            nonlocal calls
            calls += 1
            if switch:
                ctx.set_stream(streams[calls % 3].cuda_stream if calls % 4 else None)

        state = mols.copy()
        for sweep in range(12):
            out.append(ew.full(state, [3] * 90)["ewald_fourier"])
            turn()
            for k in range(8):
                new, old = moved(state, (7 * sweep + k) % 90, 0.2)
                out.append(ew.delta(new, old)["ewald_fourier"])
                turn()
                ew.accept()
                at = 3 * ((7 * sweep + k) % 90)
                state[at:at + 3] = new
                out += [t.molecule_vdw for t in system.external_energies(new, 3, skip=(7 * sweep + k) % 90)]
                turn()
        out.append(ew.structure_factors(0))
        ctx.set_stream(None)
        ctx.close()
        runs.append(np.concatenate([np.atleast_1d(x) for x in out]))
    assert np.array_equal(runs[0], runs[1])


def test_switch_during_a_capture(ctx, torch):
    """A switch to a stream that is being captured neither breaks the capture nor takes part in it."""
    ff = forcefield(8)
    ew = native.Ewald(ctx, ff, CELL)
    mols = random_molecules(ff, CELL, 20, seed=3)
    ew.full(mols, [3] * 20)
    new, old = moved(mols, 4, 0.3)
    first = ew.delta(new, old)["ewald_fourier"]
    x = torch.zeros(4, device="cuda")
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        ctx.set_stream(stream.cuda_stream)
        x += 1.0
        ctx.set_stream(None)
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [1.0] * 4
    assert ew.delta(new, old)["ewald_fourier"] == first


def test_batch_set_is_refused_during_a_capture(ctx, torch):
    runtime = ctypes.CDLL("libcudart.so.12")  # as loaded by torch
    ff = forcefield(4)
    ew = native.Ewald(ctx, ff, CELL)
    batch = native.EwaldBatch(ew, 1)
    stream = torch.cuda.Stream()
    graph = ctypes.c_void_p()
    ctx.set_stream(stream.cuda_stream)
    assert runtime.cudaStreamBeginCapture(ctypes.c_void_p(stream.cuda_stream), 2) == 0
    with pytest.raises(native.RaspaGpuError):
        batch.set(0)
    assert runtime.cudaStreamEndCapture(ctypes.c_void_p(stream.cuda_stream), ctypes.byref(graph)) != 0
    runtime.cudaGetLastError()
    ctx.set_stream(None)
    batch.set(0)
    assert np.array_equal(batch.get(0), ew.structure_factors(0))
