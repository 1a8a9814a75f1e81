"""CPU: batches and their members let go of the library's objects in any order, over a fake library."""
import ctypes as C
import gc

import pytest

from gromos_nb import _lib, nonbonded
from gromos_nb.nonbonded import Batch, Forcefield


class FakeLib:
    """Contexts and batches by number; a context that is in a batch cannot be destroyed."""

    def __init__(self):
        self.ctx, self.batch, self.next = set(), {}, 1

    def gr_batch_create(self, device, out):
        out._obj.value = self.next
        self.batch[self.next] = set()
        self.next += 1
        return _lib.GR_OK

    def gr_batch_add(self, b, c):
        self.batch[b.value].add(c.value)
        return _lib.GR_OK

    def gr_batch_remove(self, b, c):
        self.batch[b.value].remove(c.value)
        return _lib.GR_OK

    def gr_batch_destroy(self, b):
        del self.batch[b.value]
        return _lib.GR_OK

    def gr_ctx_destroy(self, c):
        if any(c.value in m for m in self.batch.values()):
            return _lib.GR_ERR_STATE
        self.ctx.remove(c.value)
        return _lib.GR_OK

    def gr_last_error(self):
        return b"refused"

    def member(self):
        ff = Forcefield.__new__(Forcefield)
        ff._L, ff._h = self, C.c_void_p(1 + len(self.ctx))
        self.ctx.add(ff._h.value)
        return ff


@pytest.fixture
def lib(monkeypatch):
    fake = FakeLib()
    monkeypatch.setattr(nonbonded._lib, "lib", lambda: fake)
    gc.collect()
    gc.disable()  # the cycles below go when the test says so
    yield fake
    gc.enable()


def batch_of(lib, n, members_first=True):
    b = None if members_first else Batch()
    ffs = [lib.member() for _ in range(n)]
    b = Batch() if b is None else b
    for ff in ffs:
        b.add(ff)
    return b, ffs


class Owner:
    """A program's object that refers to itself."""

    def __init__(self, *what):
        self.what, self.me = what, self


@pytest.mark.parametrize("members_first", [True, False])  # the collector finalizes the older first
def test_a_cycle_that_holds_batch_and_members(lib, members_first):
    b, ffs = batch_of(lib, 3, members_first)
    Owner(b, *ffs)
    del b, ffs
    assert len(lib.ctx) == 3
    gc.collect()
    assert not lib.ctx and not lib.batch


def test_dropped_by_reference_counts(lib):
    b, ffs = batch_of(lib, 3)
    del b                      # no cycle: the batch goes, its members stay
    assert not lib.batch and len(lib.ctx) == 3
    del ffs
    assert not lib.ctx
    b, ffs = batch_of(lib, 3)
    del ffs                    # the batch holds its members
    assert len(lib.ctx) == 3
    del b
    assert not lib.ctx and not lib.batch


def test_closed_members_leave_the_batch(lib):
    b, ffs = batch_of(lib, 3)
    ffs[1].close()
    assert len(b) == 2 and len(lib.ctx) == 2
    b.remove(ffs[0])
    ffs[0].close()
    b.close()
    ffs[2].close()
    assert not lib.ctx and not lib.batch
