"""Result arrays in ordinary host memory whose pages exist already, from a bounded pool.

A fresh array's pages have to be made first (1024 x 1024 means: 0.8 ms of a read that takes 0.3 into
pages that exist), so the memory of a result goes back to the pool when the last numpy view of it is gone, as
malloc would take it, but stays mapped.  It is pageable: a copy to a device has read it when the call that
starts it returns, whatever its stream does, and forked processes have their own.  (Page-locked blocks,
which the device could write itself, gave neither: an asynchronous copy from a temporary result was still
reading when the next result was written there.)  The pool holds at most LIMIT bytes, in use and free
together, beyond which results are ordinary numpy arrays.  Safe with several threads.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import threading
import weakref

import numpy as np

LIMIT = 256 << 20
MIN = 1 << 17    # smaller results are ordinary arrays: malloc keeps their pages
_GRAIN = 1 << 16

_lock = threading.RLock()  # reentrant: a collection inside the lock may return a block
_free: dict[int, list[np.ndarray]] = {}
_total = 0


def _after_fork() -> None:
    global _lock
    _lock = threading.RLock()  # another thread may have held it


os.register_at_fork(after_in_child=_after_fork)


def _release(size: int, block: np.ndarray) -> None:
    with _lock:
        _free.setdefault(size, []).append(block)


def _take(size: int) -> np.ndarray | None:
    """A block of size bytes, or None: the pool is at its limit."""
    global _total
    with _lock:
        blocks = _free.get(size)
        if blocks:
            return blocks.pop()
        if _total + size > LIMIT:
            for s, bs in list(_free.items()):
                while bs:
                    bs.pop()
                    _total -= s
        if _total + size > LIMIT:
            return None
        block = np.empty(size, np.uint8)
        _total += size
        return block


def empty(shape, dtype) -> np.ndarray:
    """An uninitialised array for a result that the library fills."""
    count = math.prod(shape)
    n = count * np.dtype(dtype).itemsize
    size = -(-n // _GRAIN) * _GRAIN
    block = _take(size) if n >= MIN else None
    if block is None:
        return np.empty(shape, dtype)
    owner = (C.c_byte * size).from_address(block.ctypes.data)
    weakref.finalize(owner, _release, size, block).atexit = False
    return np.frombuffer(owner, dtype, count=count).reshape(shape)
