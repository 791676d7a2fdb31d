"""A proposal stays alive, and its table untouched, while a run may read it."""

import gc
import weakref

import numpy as np
import pytest

from raspa3_b200 import native

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
