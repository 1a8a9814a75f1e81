"""Result arrays in recycled page-locked memory.

A download into ordinary memory is staged by the driver, and a result array
of a few MB is fresh memory from the operating system on every call, so each of
its pages is faulted in on the way: reading 90,000 positions and velocities
took 1.4 ms, of which the transfer is 0.1.  :func:`empty` returns arrays whose
memory is page-locked and goes back to a pool when the array (and every view
of it) is gone.  Live and pooled blocks together stay within
:data:`LIMIT` bytes; beyond that, and for small arrays, it returns ordinary
arrays.

Page-locking takes longer than a pageable download saves (3 to 10 ms for 8 MB),
so it has to pay: blocks come in size classes of at most a quarter more than
asked for, which arrays of uneven systems share, and beyond a class's first two
blocks only as many are made as arrays of the class have been dropped.  A
program that keeps its results gets ordinary arrays.

Memory that no array uses is given back when it has been idle for
:data:`IDLE_S` seconds (looked at on the next call here and when a context is
closed), all of it when the process has no open context left, and whenever
:func:`release` is called.  Safe with several threads: a block has one owner at
a time.
"""
from __future__ import annotations

import ctypes as C
import threading
import time
from collections import deque
from typing import Dict, List

import numpy as np

from . import _lib

LIMIT = 512 << 20          # bytes of page-locked memory held at most, in use or pooled
SMALLEST = 8 << 10        # smaller arrays gain nothing

IDLE_S = 10.0              # seconds that memory without an array is kept for the next one
ARENA = 8 << 20            # blocks of one size are cut from arenas of at most about this many bytes

_lock = threading.Lock()
_free: Dict[int, List[tuple]] = {}  # block size -> (address, arena)
_blocks: Dict[int, int] = {}        # block size -> blocks in all its arenas
_dropped: Dict[int, int] = {}       # block size -> ordinary arrays of it that are gone, less the blocks made since
_held = 0                           # bytes of all arenas
_open: set = set()                  # handles of the contexts that may want arrays
_looked = 0.0                       # when idle arenas were last looked for
_returned: deque = deque()          # (block size, (address, arena) or None, when) of arrays that are gone


class _Arena:
    """One page-locked allocation of `size` bytes cut into blocks of one size."""

    def __init__(self, address: int, size: int, blocks: int):
        self.address, self.size, self.blocks, self.idle = address, size, blocks, 0
        self.since = 0.0   # when its last array went


class _Block:
    """One page-locked block, or the ordinary memory in its place: the base of the array over it."""

    def __init__(self, place, size: int, shape):
        self._place, self._size = place, size
        if place is None:
            self._memory = np.empty(shape)
            self.__array_interface__ = self._memory.__array_interface__
        else:
            self.__array_interface__ = {"data": (place[0], False), "shape": tuple(shape), "typestr": "<f8",
                                        "version": 3}

    def __del__(self, returned=_returned, clock=time):
        returned.append((self._size, self._place, clock.monotonic()))  # no lock: this may run inside any allocation
        try:
            if not _open:
                _give_back(0.0)
        except Exception:      # the interpreter exits: this module's names may be gone
            pass


def _drain() -> None:
    while _returned:
        size, place, when = _returned.popleft()
        if place is None:
            _dropped[size] = _dropped.get(size, 0) + 1
            continue
        _free.setdefault(size, []).append(place)
        place[1].idle += 1
        place[1].since = when


def _pop(size: int):
    place = _free[size].pop()
    place[1].idle -= 1
    return place


def _class(n: int) -> int:
    """The block size for n bytes: whole pages, four sizes to a power of two."""
    pages = -(-n // 4096)
    step = 1 << max(0, pages.bit_length() - 3)
    return -(-pages // step) * step * 4096


def _take(size: int, ctx):
    """A block of `size` bytes, or None where an ordinary array does as well or the limit is reached.
    A new arena is allocated on the device of the context handle `ctx`."""
    global _held
    if time.monotonic() - _looked > 0.1 * IDLE_S:
        _give_back(IDLE_S)
    with _lock:
        _drain()
        if _free.get(size):
            return _pop(size)
        made, dropped = _blocks.get(size, 0), _dropped.get(size, 0)
        if made and not dropped:
            return None
        n = max(1, min(ARENA // size, 64, max(2, made, dropped)))  # few calls: each takes about a millisecond
        full = _held + n * size > LIMIT
    if full:
        _give_back(1.0)    # arenas that the current results do not need make room
    with _lock:
        if _held + n * size > LIMIT:
            return None
        _held += n * size
        _blocks[size] = _blocks.get(size, 0) + n
        _dropped[size] = max(0, _dropped.get(size, 0) - n)
    p = C.c_void_p()
    if _lib.lib().gr_ctx_host_alloc(ctx, n * size, C.byref(p)) != _lib.GR_OK:
        with _lock:
            _held -= n * size
            _blocks[size] -= n
        return None
    arena = _Arena(int(p.value), n * size, n)
    with _lock:
        arena.idle += n
        _free.setdefault(size, []).extend((arena.address + k * size, arena) for k in range(n))
        return _pop(size)


def empty(shape, ctx) -> np.ndarray:
    """An uninitialised C-contiguous float64 array for a download from the context `ctx` to fill."""
    n = 8 * int(np.prod(shape))
    if n < SMALLEST:
        return np.empty(shape)
    size = _class(n)
    return np.asarray(_Block(_take(size, ctx), size, shape))


def _idle(age: float) -> list:
    """Takes the arenas that no array has used for `age` seconds out of the pool (the caller holds the lock)."""
    global _held, _looked
    _drain()
    _looked = now = time.monotonic()
    idle = {p[1] for places in _free.values() for p in places
            if p[1].idle == p[1].blocks and now - p[1].since >= age}
    if idle:
        for size in list(_free):
            _free[size] = [p for p in _free[size] if p[1] not in idle]
        for a in idle:
            _held -= a.size
            _blocks[a.size // a.blocks] -= a.blocks
    return list(idle)


def _give_back(age: float) -> None:
    """Frees the arenas idle for `age` seconds, unless the pool is in use at this moment (this runs in
    finalizers too, which may come in the middle of any of these functions)."""
    if not _lock.acquire(blocking=False):
        return
    try:
        idle = _idle(age)
    finally:
        _lock.release()
    for a in idle:
        _lib.lib().gr_host_free(a.address)


def release() -> None:
    """Give back the arenas that no array uses."""
    with _lock:
        idle = _idle(0.0)
    for a in idle:
        _lib.lib().gr_host_free(a.address)


def opened(ctx) -> None:
    """The context `ctx` was opened."""
    _open.add(ctx)


def closed(ctx) -> None:
    """The context `ctx` was closed; with the last one go all idle arenas."""
    _open.discard(ctx)
    _give_back(IDLE_S if _open else 0.0)
