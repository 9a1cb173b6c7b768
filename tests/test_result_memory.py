"""The pool of page-locked blocks behind result arrays: block sizes."""
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
