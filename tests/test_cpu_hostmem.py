"""CPU: the pool of page-locked result arrays, over a fake of the library's allocation calls."""
import ctypes as C
import sys
import threading

import numpy as np
import pytest

from gromos_nb import hostmem


CTX = object()  # a context's handle


class FakeLib:
    def __init__(self):
        self.live = {}
        self.calls = 0

    def gr_ctx_host_alloc(self, ctx, n, out):
        assert ctx is CTX         # never without the context whose device is meant
        self.calls += 1
        buf = C.create_string_buffer(int(n))
        p = C.addressof(buf)
        self.live[p] = (buf, int(n))
        C.cast(out, C.POINTER(C.c_void_p))[0] = p
        return 0

    def gr_host_free(self, p):
        del self.live[p]
        return 0

    def bytes(self):
        return sum(n for _, n in self.live.values())


@pytest.fixture
def lib(monkeypatch):
    fake = FakeLib()
    monkeypatch.setattr(hostmem._lib, "lib", lambda: fake)
    hostmem._free.clear()
    hostmem._blocks.clear()
    hostmem._dropped.clear()
    hostmem._returned.clear()
    hostmem._held = 0
    yield fake
    hostmem._free.clear()
    hostmem._blocks.clear()
    hostmem._dropped.clear()
    hostmem._returned.clear()
    hostmem._held = 0


def test_memory_is_reused_after_every_view_is_gone(lib):
    a = hostmem.empty((5000, 3), CTX)
    a[:] = 7.0
    at, view = a.ctypes.data, a[10:]
    del a
    b = hostmem.empty((5000, 3), CTX)
    assert b.ctypes.data != at and (view == 7.0).all()   # the view still owns the block
    del view
    c = hostmem.empty((5000, 3), CTX)
    assert c.ctypes.data == at and c.flags.c_contiguous and c.flags.writeable and c.dtype == np.float64
    assert len(lib.live) == 1                             # one arena for the three


def test_limit_and_release(lib, monkeypatch):
    monkeypatch.setattr(hostmem, "LIMIT", 20 << 20)
    keep = [hostmem.empty((1 << 20,), CTX) for _ in range(4)]  # 8 MB each: the first two fit
    assert lib.bytes() <= 20 << 20 and hostmem._held == lib.bytes()
    for k, x in enumerate(keep):
        x[:] = k                                          # the others are ordinary arrays
    assert [x[0] for x in keep] == [0, 1, 2, 3]
    del keep, x
    y = hostmem.empty((1000, 3), CTX)                          # another size: idle arenas make room
    assert lib.bytes() <= 20 << 20
    hostmem.release()
    assert len(lib.live) == 1                             # the arena of y stays
    del y
    hostmem.release()
    assert not lib.live and hostmem._held == 0


def test_small_arrays_are_ordinary(lib):
    hostmem.empty((10, 3), CTX)[:] = 1.0
    assert not lib.live


def test_threads_never_share_a_block(lib):
    bad = []

    def work(tag):
        for _ in range(300):
            a, b = hostmem.empty((2000, 3), CTX), hostmem.empty((2000, 3), CTX)
            a[:], b[:] = tag, -tag
            if (a != tag).any() or (b != -tag).any():
                bad.append(tag)

    ts = [threading.Thread(target=work, args=(k + 1,)) for k in range(6)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad


def test_a_forcefields_arrays_are_allocated_on_its_device(lib):
    from gromos_nb.nonbonded import Forcefield

    for name in ("gr_md_download", "gr_result_download", "gr_forces_eval"):
        setattr(lib, name, lambda *a: 0)
    ff = Forcefield.__new__(Forcefield)
    ff._L, ff._h, ff.n_atoms, ff.G = lib, CTX, 3000, 1
    kept = [ff.md_state(), ff.result()["forces"], ff.apply()["forces"]]
    assert len(lib.live) == 1 and kept
    ff._h = None


def test_idle_memory_is_given_back(lib, monkeypatch):
    now = [0.0]
    monkeypatch.setattr(hostmem.time, "monotonic", lambda: now[0])
    monkeypatch.setattr(hostmem, "_looked", 0.0)
    hostmem.opened(1)
    hostmem.opened(2)
    a, b = hostmem.empty((5000, 3), CTX), hostmem.empty((1 << 20,), CTX)
    del a
    now[0] = hostmem.IDLE_S - 1.0
    c = hostmem.empty((1000, 3), CTX)
    assert len(lib.live) == 3                  # kept for the next array of its size
    now[0] += 2.0
    hostmem.empty((1000, 3), CTX)
    assert len(lib.live) == 2                  # idle for too long: only b's and c's arenas
    del b
    hostmem.closed(1)
    assert len(lib.live) == 2
    hostmem.closed(2)                          # the last context: what no array uses
    assert len(lib.live) == 1 and hostmem._held == lib.bytes()
    c[:] = 1.0
    del c                                      # and the rest with its array
    assert not lib.live and hostmem._held == 0


def test_arrays_may_outlive_the_module(lib, monkeypatch):
    """At the interpreter's exit a module's names are cleared while arrays still live: no message."""
    said = []
    monkeypatch.setattr(sys, "unraisablehook", lambda u: said.append(u.exc_value))
    a = hostmem.empty((5000, 3), CTX)
    names = [n for n in vars(hostmem) if not n.startswith("__")]
    with monkeypatch.context() as m:
        for n in names:
            m.setattr(hostmem, n, None)
        del a
    assert not said


def test_kept_results_are_not_page_locked(lib):
    """Memory is page-locked for arrays that come and go, not for a list of results that grows."""
    hostmem.opened(1)
    kept = [(hostmem.empty((90000, 3), CTX), hostmem.empty((90000, 3), CTX)) for _ in range(40)]
    assert lib.calls == 1 and kept
    del kept
    for _ in range(40):
        hostmem.empty((90000, 3), CTX), hostmem.empty((90000, 3), CTX)
    assert lib.calls <= 2
    hostmem.closed(1)


def test_uneven_sizes_share_their_memory(lib):
    """The results of 256 uneven systems, dropped after every pass: page-locked a few times, then reused."""
    hostmem.opened(1)
    sizes = [3 * n for n in range(500, 8180, 30)]
    calls = []
    for _ in range(8):
        results = [hostmem.empty((n, 3), CTX) for n in sizes for _ in range(2)]
        assert all(a.flags.c_contiguous and a.shape == (n, 3) for a, n in zip(results[::2], sizes))
        del results
        calls.append(lib.calls)
    assert calls[-1] == calls[3] and calls[-1] < 128
    assert lib.bytes() <= 2.5 * sum(2 * 24 * n for n in sizes)
    hostmem.closed(1)


def test_block_sizes():
    for n in (8192, 8193, 24000, 36000, 131072, 131073, 2160000, 123456789):
        assert n <= hostmem._class(n) <= max(1.25 * n, n + 4095) and hostmem._class(n) % 4096 == 0
        assert hostmem._class(hostmem._class(n)) == hostmem._class(n)
