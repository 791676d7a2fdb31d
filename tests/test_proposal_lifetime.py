"""A proposal stays alive, and its table untouched, while a run may read it."""

import gc
import weakref

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.gcmc import beta_of, fugacity_of, methane_component
from raspa3_b200.synthetic import synthetic_forcefield
from test_gcmc_gpu import empty_framework

CELL = np.diag([30.0, 30.0, 30.0])


class _Library:
    """Stands in for the library: every call succeeds, or fails."""

    def __init__(self, status):
        self.status = status

    def __getattr__(self, name):
        return lambda *args: b"refused" if name == "rg_ctx_last_error" else self.status


class _Handle:
    handle = 1


def _unopened(cls):
    """An object of the binding without a device behind it."""
    x = object.__new__(cls)
    x.ctx, x.handle = _Handle(), 1
    x._proposals = {}
    x.close = lambda: None
    return x


@pytest.mark.parametrize("cls,first", [(native.Gcmc, ()), (native.Mixture, (0,))])
def test_proposal_in_use_is_referenced(monkeypatch, cls, first):
    monkeypatch.setattr(native, "lib", lambda: _Library(0))
    user, proposal, other = _unopened(cls), _Handle(), _Handle()
    ref = weakref.ref(proposal)
    user.set_proposal(*first, proposal, CELL)
    del proposal
    gc.collect()
    assert ref() is not None
    monkeypatch.setattr(native, "lib", lambda: _Library(1))
    with pytest.raises(native.RaspaGpuError):  # the one in use stays
        user.set_proposal(*first, other, CELL)
    gc.collect()
    assert ref() is not None
    monkeypatch.setattr(native, "lib", lambda: _Library(0))
    user.set_proposal(*first, None)
    gc.collect()
    assert ref() is None


def _chains(torch, reuse):
    """A run with one proposal, queued on a stream; then, on another, that proposal is destroyed and (reuse) its memory
    taken for the next, which has another network's density."""
    ctx = native.Context(0)
    ff = synthetic_forcefield(charges=False)
    system = native.System(ctx, ff, CELL, empty_framework())
    g = native.Gcmc(system, None, methane_component(), beta_of(300.0), fugacity_of(2e6), n_chains=64, seed=9)
    theta = np.random.default_rng(1).normal(size=(2, native.lib().rg_mlp_num_params())).astype(np.float32)
    nets = [native.Mlp(ctx, seed=1) for _ in range(2)]
    for m, t in zip(nets, theta):
        m.set_params(0.3 * t)
    first = native.Proposal(nets[0], cells_per_axis=40, eps_uniform=0.05)
    streams = [torch.cuda.Stream() for _ in range(2)]
    g.set_proposal(first, CELL)
    ctx.synchronize()
    ctx.set_stream(streams[0].cuda_stream)
    g.run(8000, record=True)
    if reuse:
        ctx.set_stream(streams[1].cuda_stream)
        g.set_proposal(None)
        first.close()
        second = native.Proposal(nets[1], cells_per_axis=40, eps_uniform=0.05)
        second.close()
        ctx.set_stream(streams[0].cuda_stream)
    out = g.results()
    ctx.set_stream(None)
    ctx.close()
    return out


@pytest.mark.gpu
def test_destroyed_behind_a_run():
    torch = pytest.importorskip("torch")
    assert _chains(torch, False) == _chains(torch, True)


# small after large and large after small, across the sizes that are kept (up to 64 MB, 161^3 cells) and handed on
@pytest.mark.gpu
def test_tables_of_changing_sizes():
    ctx = native.Context(0)
    m = native.Mlp(ctx, seed=5)
    sizes = (2, 200, 3, 128, 60, 128, 1, 162, 8)
    s = np.random.default_rng(2).random((50, 3))
    fresh = {}
    for cells in set(sizes):
        one = native.Context(0)
        n = native.Mlp(one, seed=5)
        fresh[cells] = native.Proposal(n, cells_per_axis=cells).density(s)
        one.close()
    for cells in sizes:
        p = native.Proposal(m, cells_per_axis=cells)
        assert np.array_equal(p.density(s), fresh[cells])
        p.close()
    ctx.close()
