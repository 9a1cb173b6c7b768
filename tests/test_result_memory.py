"""Results are ordinary arrays of their own: page-locked blocks are only passed
through, so nothing a caller holds, copies asynchronously or shares with a
forked process is ever rewritten by a later result."""
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

    context = 7

    def msosm_context_id(self, out):
        out._obj.value = self.context
        return 0


@pytest.fixture
def fake(monkeypatch):
    f = FakeLib()
    monkeypatch.setattr(_abi, "lib", lambda: f)
    monkeypatch.setattr(_pinned, "_free", {})
    monkeypatch.setattr(_pinned, "_total", 0)
    monkeypatch.setattr(_pinned, "_context", f.context)
    monkeypatch.setattr(_pinned, "_others", {})
    yield f
    gc.collect()


@pytest.mark.parametrize("n", [10, 1 << 13, (1 << 16) + 1, 1 << 18, 1 << 19])
def test_results_own_their_memory(fake, n):
    seen = []

    def read(value):
        def f(p):
            seen.append(p)
            ctypes.memset(p, value, 4 * n)
        return f
    a = _pinned.fetch(n, np.float32, read(1))
    b = _pinned.fetch((n, 1), np.float32, read(2))
    assert a.shape == (n,) and b.shape == (n, 1)
    assert a.flags.owndata and b.flags.owndata and a.ctypes.data not in fake.blocks
    assert np.all(a.view(np.uint8) == 1) and np.all(b.view(np.uint8) == 2)
    staged = _pinned.MIN_BYTES <= 4 * n <= _pinned.MAX_BYTES
    assert (seen[0] in fake.blocks) == staged and (seen[0] == seen[1]) >= staged  # one block, used again


def test_error_gives_the_block_back(fake):
    def read(p):
        raise RuntimeError("no result")
    with pytest.raises(RuntimeError):
        _pinned.fetch(1 << 16, np.float32, read)
    gc.collect()
    assert sum(len(b) for b in _pinned._free.values()) == 1


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


@pytest.mark.gpu
def test_results_of_the_public_calls():
    import torch
    from msosm_gpu_b200 import Dedisperser
    from msosm_gpu_b200.dm_proposal import DMProposalNet
    rng = np.random.default_rng(4)
    d = Dedisperser(16e6, np.linspace(0.0, 9.0, 32).astype(np.float32), 1242e6, 1024, 8)
    d.fold_init(1500.25 / 16e6, 16e6, time_bin=1000, discard_Nd=1)
    net = DMProposalNet(8, 64, 40, max_batch=4)
    x = rng.standard_normal((4, 8, 64)).astype(np.float32)
    one = np.ones(4, np.float32)

    def results():
        d.filter_block((rng.standard_normal(d.block_samples) + 0j).astype(np.complex64))
        return [d.get_output(), d.get_output(dtype=np.uint16), d.get_profiles(),
                net.gradient(x * rng.standard_normal(), one, one, want_grad=True)[1]]
    first = results()
    copies = [r.copy() for r in first]
    assert all(r.nbytes >= _pinned.MIN_BYTES for r in first)
    for r in first:
        assert not torch.from_numpy(r.view(np.int16)).is_pinned()
    second = results()
    for a, b, c in zip(first, second, copies):
        assert np.array_equal(a, c) and not np.array_equal(a, b)
