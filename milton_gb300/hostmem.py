"""Result arrays in page-locked host memory, from a bounded pool.

The device writes such an array itself (mgpu_host_alloc), so a film read needs no staging copy and
touches no fresh pages (256 x 256 means: 157 -> 40 us a read).  A block goes back to the pool when the
last numpy view of it is gone; the pool holds at most LIMIT bytes, in use and free together, beyond
which results are ordinary numpy arrays.  Safe with several threads.
"""
from __future__ import annotations

import ctypes as C
import math
import threading
import weakref

import numpy as np

from . import _native as N

LIMIT = 256 << 20
MIN = 1 << 17    # smaller results are ordinary arrays: their copy costs less than the bookkeeping
_GRAIN = 1 << 16

_lock = threading.RLock()  # reentrant: a collection inside the lock may return a block
_free: dict[int, list[int]] = {}
_total = 0


def _release(size: int, addr: int) -> None:
    with _lock:
        _free.setdefault(size, []).append(addr)


def _take(size: int) -> int | None:
    """A block of size bytes, or None: the pool is at its limit or page-locked memory is short."""
    global _total
    lib = N.load()
    with _lock:
        blocks = _free.get(size)
        if blocks:
            return blocks.pop()
        if _total + size > LIMIT:
            for s, bs in list(_free.items()):
                while bs:
                    lib.mgpu_host_free(bs.pop())
                    _total -= s
        if _total + size > LIMIT:
            return None
        p = C.c_void_p()
        if lib.mgpu_host_alloc(size, C.byref(p)) != N.MGPU_OK or not p.value:
            return None
        _total += size
        return p.value


def empty(shape, dtype) -> np.ndarray:
    """An uninitialised array for a result that the library fills."""
    count = math.prod(shape)
    n = count * np.dtype(dtype).itemsize
    size = -(-n // _GRAIN) * _GRAIN
    addr = _take(size) if n >= MIN else None
    if addr is None:
        return np.empty(shape, dtype)
    owner = (C.c_byte * size).from_address(addr)
    weakref.finalize(owner, _release, size, addr).atexit = False
    return np.frombuffer(owner, dtype, count=count).reshape(shape)
