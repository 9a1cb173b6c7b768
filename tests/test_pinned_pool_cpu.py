"""The pool of result arrays (_pinned): blocks come back when the last view is
gone, are reused, never exceed the bound, and small, large or refused requests
fall back to ordinary arrays.  The page-locked allocator is replaced by an
ordinary one."""
import ctypes
import gc
import threading

import numpy as np
import pytest

from msosm_gpu_b200 import _abi, _pinned


class FakeLib:
    def __init__(self):
        self.blocks, self.refuse = {}, False

    def msosm_host_alloc(self, size, pinned, out):
        assert pinned == 1
        if self.refuse:
            return 2
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
    monkeypatch.setattr(_pinned, "POOL_BYTES", 1 << 20)
    yield f
    gc.collect()


def test_block_returns_after_the_last_view(fake):
    a = _pinned.empty((100, 200), np.float32)
    assert a.shape == (100, 200) and a.dtype == np.float32 and a.flags.writeable and a.flags.c_contiguous
    a[:] = 3.0
    view = a[5:, ::2]
    addr = a.ctypes.data
    assert list(fake.blocks) == [addr]
    del a
    gc.collect()
    assert not any(_pinned._free.values()) and view[0, 0] == 3.0
    del view
    gc.collect()
    b = _pinned.empty(20000, np.float32)  # the same size class: the same block
    assert b.ctypes.data == addr and len(fake.blocks) == 1


def test_bound_and_fallbacks(fake):
    keep = [_pinned.empty(1 << 18, np.uint8) for _ in range(6)]
    assert len(fake.blocks) == 4  # 1 MB of blocks, the rest ordinary
    for i, k in enumerate(keep):
        k[:] = i
    assert [int(k[-1]) for k in keep] == list(range(6))
    del keep, k
    gc.collect()
    big = _pinned.empty(1 << 20, np.uint8)  # waiting blocks of another size make room
    assert list(fake.blocks) == [big.ctypes.data] and _pinned._total == 1 << 20
    assert _pinned.empty(10, np.complex64).size == 10 and len(fake.blocks) == 1
    assert _pinned.empty(_pinned.MAX_BYTES + 1, np.uint8).size == _pinned.MAX_BYTES + 1 and len(fake.blocks) == 1
    fake.refuse = True
    assert _pinned.empty(1 << 17, np.uint8).size == 1 << 17


def test_threads(fake):
    def work(seed):
        for i in range(200):
            a = _pinned.empty((1 << 15) + (seed % 3) * 40000, np.uint8)
            a[:] = seed
            assert a[0] == seed and a[-1] == seed
            del a
    ts = [threading.Thread(target=work, args=(s,)) for s in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    gc.collect()
    assert _pinned._total <= 1 << 20
    assert sum(s * len(b) for s, b in _pinned._free.items()) == _pinned._total
