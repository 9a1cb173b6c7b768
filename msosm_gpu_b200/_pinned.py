"""Page-locked staging for results, and the result arrays themselves.

A copy from the device straight into pageable memory is staged by the driver:
512 KB take 54 us (149 us into fresh zeroed pages), into page-locked memory and
from there by the host 42 us; above about 1 MB the driver's own staging is the
faster one (2 MB: 136 against 174 us).  ``fetch`` returns results in ordinary
memory, read through a page-locked block where that pays.  The blocks never
leave this module: a caller's array over one (21 us for the 512 KB) could be
rewritten by a later result while the caller's own asynchronous copy out of it
was still under way, and a forked process would share it with its parent.

``empty`` hands out arrays over page-locked blocks; when an array and every view
of it are gone its block goes back to a pool (at most POOL_BYTES per CUDA context,
handed out or waiting; beyond that, and for small or large sizes, the array is an
ordinary one).  Safe to use from several threads.
"""
from __future__ import annotations

import ctypes
import threading

import numpy as np

GRAIN = 64 << 10       # block sizes are multiples of this
MIN_BYTES = 32 << 10   # below, the driver's staging costs no more
MAX_BYTES = (1 << 20) + GRAIN
POOL_BYTES = 16 << 20

_lock = threading.RLock()  # re-entrant: an array may be collected while the pool is in use
_free: "dict[int, list]" = {}  # block size -> addresses
_total = 0                     # bytes of all blocks
_context = 0                   # the CUDA context (msosm_context_id) these belong to
_others: "dict[int, tuple]" = {}  # _free and _total of other contexts


def _take(size: int):
    """Address of a block of `size` bytes, or None."""
    global _total
    from ._abi import lib
    with _lock:
        if _free.get(size):
            return _free[size].pop()
        while _total + size > POOL_BYTES:
            # (a snapshot: an array collected meanwhile may add a size)
            other = next((s for s, b in list(_free.items()) if b), None)
            if other is None:
                return None
            lib().msosm_host_free(ctypes.c_void_p(_free[other].pop()), 1)
            _total -= other
        p = ctypes.c_void_p()
        if lib().msosm_host_alloc(size, 1, ctypes.byref(p)) != 0 or not p.value:
            return None
        _total += size
        return p.value


def _follow_context() -> None:
    """Switch to the current context's blocks.  Those of a context that is gone
    (a program that resets the device takes its page-locked memory with it) are
    never handed out again: ids do not come back.  Under the lock."""
    global _context, _free, _total
    from ._abi import check, lib
    now = ctypes.c_ulonglong()
    check(lib().msosm_context_id(ctypes.byref(now)))
    if now.value != _context:
        _others[_context] = (_free, _total)
        _context = now.value
        _free, _total = _others.pop(_context, ({}, 0))


class _Block:
    """Owner of a block for as long as an array refers to it."""

    def __init__(self, address: int, size: int, shape, dtype):
        self._address, self._size, self._context = address, size, _context
        self.__array_interface__ = {"data": (address, False), "shape": tuple(shape), "typestr": np.dtype(dtype).str,
                                    "version": 3}

    def __del__(self):
        try:
            with _lock:
                mine = _free if self._context == _context else _others[self._context][0]
                mine.setdefault(self._size, []).append(self._address)
        except Exception:  # interpreter shutdown
            pass


def empty(shape, dtype) -> np.ndarray:
    """An uninitialised array, page-locked where that pays."""
    shape = (int(shape),) if np.isscalar(shape) else tuple(int(s) for s in shape)
    nbytes = int(np.prod(shape)) * np.dtype(dtype).itemsize
    if MIN_BYTES <= nbytes <= MAX_BYTES:
        size = -(-nbytes // GRAIN) * GRAIN
        address = _take(size)
        if address is not None:
            return np.asarray(_Block(address, size, shape, dtype))
    return np.empty(shape, dtype)


def fetch(shape, dtype, read) -> np.ndarray:
    """A new array of ordinary memory that read(address) has filled; read
    returns when its copy is done."""
    with _lock:
        _follow_context()
        a = empty(shape, dtype)
    read(a.ctypes.data)
    return a.copy() if isinstance(a.base, _Block) else a
