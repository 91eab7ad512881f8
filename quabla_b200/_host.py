"""Page-locked landing buffers for what a plan reads back.

A device-to-host copy into fresh pageable memory pays for the driver's bounce buffer (1.3 MB of gradients: 0.57 ms); into
a page-locked block it runs at link speed (0.03 ms).  A reader copies what it hands out from such an array into ordinary
memory and drops it: page-locked memory is shared with forked children, and one array kept by a caller would keep the block.
When the last array made from a block is gone the block goes back to the pool.  The pool is shared by all plans and
threads and bounded: beyond `LIMIT` bytes in use the caller gets ordinary memory, and at most `IDLE_LIMIT` bytes stay
page-locked without an owner.
"""

from __future__ import annotations

import ctypes as C
import os
import threading

import numpy as np

from . import _lib

LIMIT = 128 << 20
IDLE_LIMIT = 32 << 20
_SMALLEST = 4096

_lock = threading.RLock()  # a collection inside a locked section may run _Block.__del__ on the same thread
_idle: dict[int, list[int]] = {}   # block size -> addresses
_total = 0                         # page-locked bytes, handed out or idle
_idle_bytes = 0
_forked = False                    # in a child: the blocks are the parent's, the CUDA runtime is not usable


def _after_fork() -> None:
    global _lock, _forked
    _lock = threading.RLock()  # another thread of the parent may have held it
    _forked = True
    _idle.clear()


os.register_at_fork(after_in_child=_after_fork)


class _Block:
    """Owner of one page-locked block; NumPy arrays made from it keep it alive."""

    __slots__ = ("address", "size", "__array_interface__")

    def __init__(self, address: int, size: int, count: int, dtype: np.dtype) -> None:
        self.address = address
        self.size = size
        self.__array_interface__ = {"data": (address, False), "shape": (count,), "typestr": dtype.str, "version": 3}

    def __del__(self) -> None:
        if _lock is not None and not _forked:  # else: the interpreter is going down, or the block is the parent's
            _give_back(self.address, self.size)


def _give_back(address: int, size: int) -> None:
    global _total, _idle_bytes
    with _lock:
        if _idle_bytes + size <= IDLE_LIMIT:
            _idle.setdefault(size, []).append(address)
            _idle_bytes += size
            return
        _total -= size
    _lib.load().qb200_host_free(address)


def empty(count: int, dtype: np.dtype) -> np.ndarray:
    """An uninitialised one-dimensional array, page-locked when the pool has room."""
    global _total, _idle_bytes
    if _forked:
        return np.empty((count,), dtype=dtype)
    size = _SMALLEST
    while size < count * dtype.itemsize:
        size *= 2
    with _lock:
        found = _idle.get(size)
        if found:
            address = found.pop()
            _idle_bytes -= size
        elif _total + size <= LIMIT:
            address = None
            _total += size
        else:
            return np.empty((count,), dtype=dtype)
    if address is None:
        out = C.c_void_p()
        if _lib.load().qb200_host_alloc(size, C.byref(out)) != _lib.OK:
            with _lock:
                _total -= size
            return np.empty((count,), dtype=dtype)
        address = out.value
    return np.asarray(_Block(address, size, count, dtype))
