"""A program that resets the device (as the reference's reset_device does) and
goes on with new handles: nothing kept for the process outlives its context --
the kernels' shared-memory attributes, the page-locked status words and the
staging blocks of results.  The pool's part on the CPU with a stand-in for the
library; on the GPU in a process of its own, through the driver's primary
context reset."""
import ctypes
import gc
import subprocess
import sys

import numpy as np
import pytest

from msosm_gpu_b200 import _abi, _pinned

SCRIPT = """
import numpy as np
from cuda.bindings import driver
from msosm_gpu_b200 import Dedisperser, Fold_GPU
from msosm_gpu_b200.dm_proposal import DMProposalNet


def results():
    out = []
    rng = np.random.default_rng(1)
    for fft, precision in ((1024, "fp32"), (4096, "fp32"), (16384, "fp32"), (4096, "fp16"), (8192, "bf16"), (1 << 16, "fp32")):
        d = Dedisperser(16e6, np.linspace(0.0, 3.0, 9).astype(np.float32), 1242e6, fft, 4, precision=precision)
        d.fold_init(2000.25 / 16e6, 16e6, time_bin=1000, discard_Nd=1)
        for _ in range(2):
            d.filter_block((rng.standard_normal(d.block_samples) + 0j).astype(np.complex64))
        out += [d.get_output(), d.get_profiles()]
        d.close()
    net = DMProposalNet(8, 64, 40, max_batch=4)
    x = rng.standard_normal((4, 8, 64)).astype(np.float32)
    one = np.ones(4, np.float32)
    out.append(net.gradient(x, one, one, want_grad=True)[1])
    net.close()
    return out


before = results()
for _ in range(2):
    status = driver.cuDevicePrimaryCtxReset(driver.cuDeviceGet(0)[1])[0]
    assert int(status) == 0, status
    after = results()
    assert all(np.array_equal(a, b) for a, b in zip(before, after))
print("same")
"""


@pytest.mark.gpu
def test_new_handles_after_a_device_reset():
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("same"), r.stdout + r.stderr


def test_pool_follows_the_context(monkeypatch):
    class Lib:
        context, blocks = 3, {}

        def msosm_host_alloc(self, size, pinned, out):
            b = ctypes.create_string_buffer(size)
            self.blocks[ctypes.addressof(b)] = b
            out._obj.value = ctypes.addressof(b)
            return 0

        def msosm_context_id(self, out):
            out._obj.value = self.context
            return 0
    f = Lib()
    monkeypatch.setattr(_abi, "lib", lambda: f)
    for name, value in (("_free", {}), ("_total", 0), ("_context", 0), ("_others", {})):
        monkeypatch.setattr(_pinned, name, value)
    used = []

    def read(p):
        used.append(p)
    _pinned.fetch(1 << 16, np.float32, read)
    held = _pinned.empty(1 << 18, np.uint8)  # the same block, in use across the reset
    f.context = 4
    _pinned.fetch(1 << 16, np.float32, read)
    first, second = used
    assert held.ctypes.data == first != second
    del held
    gc.collect()
    _pinned.fetch(1 << 16, np.float32, read)
    assert used[2] == second  # not the block of the context that is gone
    f.context = 3  # another live device's: its own blocks again
    _pinned.fetch(1 << 16, np.float32, read)
    assert used[3] == first and _pinned._total == 1 << 18
