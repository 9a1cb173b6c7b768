"""Results written to host memory by a kernel: only where the whole result lies
in one block of msosm_host_alloc.  The rule on the CPU (tests/cpp/
host_blocks_check.cpp); on the GPU, profiles read into such a block, into a part
of one, into other page-locked memory and into ordinary memory are the same."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_ranges_within_one_block(tmp_path):
    exe = str(tmp_path / "host_blocks_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-I", os.path.join(ROOT, "msosm_gpu_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "host_blocks_check.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


@pytest.mark.gpu
def test_profiles_into_every_kind_of_host_memory():
    import torch
    from msosm_gpu_b200 import Dedisperser
    from msosm_gpu_b200._abi import check, lib
    bw, bins, dms = 16e6, 1000, np.linspace(0.0, 9.0, 9).astype(np.float32)
    d = Dedisperser(bw, dms, 1242e6, 1024, 64, series=False)
    d.fold_init(2000.25 / bw, bw, time_bin=bins, discard_Nd=1)
    rng = np.random.default_rng(2)
    for _ in range(2):
        d.filter_block((rng.standard_normal(d.block_samples) + 0j).astype(np.complex64))
    ref = d.get_profiles()
    assert np.abs(ref).max() > 0
    n = ref.size
    block = ctypes.c_void_p()
    check(lib().msosm_host_alloc(4 * (n + 3), 1, ctypes.byref(block)))
    whole = np.ctypeslib.as_array(ctypes.cast(block, ctypes.POINTER(ctypes.c_float)), (n + 3,))
    whole[:] = -1.0
    pinned = torch.empty(n + 2, pin_memory=True).numpy()
    for room in (whole[3:], pinned[:n], pinned[2:], np.empty(n, np.float32), np.empty(n + 1, np.float32)[1:], whole[:n]):
        assert np.all(whole[:3] == -1.0)  # outside every range so far
        room[:] = -1.0
        check(lib().msosm_dedisp_get_profiles(d._h, ctypes.c_void_p(room.ctypes.data)))
        assert np.array_equal(room, ref.reshape(-1))
    check(lib().msosm_host_free(block, 1))
