"""The pool of page-locked blocks behind result arrays: block sizes, and arrays collected in the
middle of its work."""
import ctypes
import gc

import numpy as np
import pytest

from msosm_gpu_b200 import _abi, _pinned


class FakeLib:
    def __init__(self):
        self.blocks = {}

    def msosm_host_alloc(self, size, pinned, out):
        b = ctypes.create_string_buffer(size)
        self.blocks[ctypes.addressof(b)] = b
        out._obj.value = ctypes.addressof(b)
        return 0

    def msosm_host_free(self, p, pinned):
        del self.blocks[p.value]
        return 0


@pytest.fixture
def fake(monkeypatch):
    f = FakeLib()
    monkeypatch.setattr(_abi, "lib", lambda: f)
    monkeypatch.setattr(_pinned, "_free", {})
    monkeypatch.setattr(_pinned, "_total", 0)
    yield f
    gc.collect()


def test_block_sizes_follow_the_request(fake):
    a = _pinned.empty((1 << 17) + 1, np.uint32)  # a series with its trailing element: not twice the memory
    assert _pinned._total <= a.nbytes + _pinned.GRAIN


def test_array_collected_while_room_is_made(fake, monkeypatch):
    """Making room walks the waiting blocks; an array of a new size collected
    just then comes back to the pool in the middle of the walk."""
    monkeypatch.setattr(_pinned, "POOL_BYTES", 1 << 20)
    held = [_pinned.empty(3 * _pinned.GRAIN, np.uint8)]

    class Collected(list):
        def __bool__(self):
            held.clear()
            gc.collect()
            return len(self) > 0
    keep = _pinned.empty(1 << 18, np.uint8)
    _pinned._free.setdefault(_pinned.GRAIN, Collected())
    _pinned._free[2 * _pinned.GRAIN] = Collected()
    big = _pinned.empty(10 << 16, np.uint8)
    assert big.size == 10 << 16 and keep.size == 1 << 18 and not held
