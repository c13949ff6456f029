"""Page-locked host arrays for results, reused.

A result in ordinary memory is filled by the driver through a small bounce buffer while the kernel clears fresh pages under it:
5 GB/s, 1.5 ms for the logits of 64 rows of 32,768 values, in which the GPU waits.  The device writes page-locked memory at the
bus's rate (0.17 ms), but locking pages costs about as much as one such fill, so blocks are kept: an array owns its block until
the last reference to it (or to a view of it) is gone, then the block serves another array.
"""
from __future__ import annotations

import ctypes
import threading
from typing import List, Tuple

import numpy as np

from .. import capi

GRAIN = 1 << 16           # sizes are rounded up to this, so that a step with a row more finds a block too


class _Block:
    """What an array refers to as its base: a block on loan."""

    def __init__(self, pool: "HostPool", address: int, size: int, shape: Tuple[int, ...]):
        self._pool, self._address, self._size = pool, address, size
        self.__array_interface__ = {"data": (address, False), "shape": shape, "typestr": "<f4", "version": 3}

    def __del__(self):
        try:
            self._pool._give_back(self._address, self._size)
        except Exception:
            pass


class HostPool:
    """Blocks of page-locked memory behind float32 arrays, `limit` bytes at most, lent out or free; beyond it arrays are ordinary ones.
     Any thread may ask for arrays and drop them.  `context`: the engine's,
    whose device a thread works on that asks for an array (one that never chose would set up the first device)."""

    def __init__(self, limit: int, alloc=None, free=None, context=None):
        self._limit, self._held, self._closed = limit, 0, False
        self._free: List[Tuple[int, int]] = []       # (size, address)
        self._lock = threading.RLock()                # re-entrant: a collection inside it may drop an array
        self._alloc, self._release = alloc or (lambda size: _host_alloc(context, size)), free or _host_free

    @property
    def held(self) -> int:
        """Bytes of page-locked memory, lent out or free."""
        return self._held

    def array(self, shape: Tuple[int, ...]) -> np.ndarray:
        """An uninitialised float32 array."""
        need = 4 * int(np.prod(shape, dtype=np.int64))
        block = self._take(-(-need // GRAIN) * GRAIN) if need else None
        if block is None:
            return np.empty(shape, dtype=np.float32)
        return np.asarray(_Block(self, block[1], block[0], tuple(int(n) for n in shape)))

    def _take(self, size: int):
        with self._lock:
            if self._closed:
                return None
            fits = [b for b in self._free if size <= b[0] <= 2 * size]
            if fits:
                block = min(fits)
                self._free.remove(block)
                return block
            unused = sorted(self._free)
            if self._held - sum(s for s, _ in unused) + size > self._limit:    # not even without them: they stay
                return None
            while unused and self._held + size > self._limit:    # blocks of sizes no longer asked for make room
                s, address = unused.pop()
                self._free.remove((s, address))
                self._release(address)
                self._held -= s
            address = self._alloc(size)
            if not address:
                return None
            self._held += size
            return size, address

    def _give_back(self, address: int, size: int) -> None:
        with self._lock:
            if not self._closed:
                self._free.append((size, address))
                return
            self._held -= size
        self._release(address)

    def close(self) -> None:
        """Free what is not lent out; the rest follows as its arrays go."""
        with self._lock:
            self._closed = True
            blocks, self._free = self._free, []
            self._held -= sum(size for size, _ in blocks)
        for _, address in blocks:
            self._release(address)


def _host_alloc(context, size: int) -> int:
    p, lib = ctypes.c_void_p(), capi.load()
    rc = lib.imp_context_host_alloc(context, size, ctypes.byref(p)) if context else lib.imp_host_alloc(size, ctypes.byref(p))
    return (p.value or 0) if rc == 0 else 0


def _host_free(address: int) -> None:
    capi.load().imp_host_free(address)
