"""Fold_GPU on raw device pointers: a and b may be overwritten as soon as
calculate_intensity returns, and the C++ drop-in takes the event-ordered entry
for every class derived from MSOSM_GPU_BATCH."""
import os
import subprocess

import numpy as np
import pytest

from msosm_gpu_b200 import Dedisperser
from msosm_gpu_b200.fold import Fold_GPU

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_dropin_classes_take_the_handle_entry(tmp_path):
    exe = str(tmp_path / "fold_route_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "fold_route_check.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("pols", [1, 2])
def test_series_overwritten_right_after_the_call(pols):
    import torch
    size, ps, bins = 1 << 22, 4 * 4096, 64  # 256 periods a chunk
    f = Fold_GPU((ps + 0.25) / 1e6, 1e6, size, time_bin=bins)
    x = [torch.empty(size, dtype=torch.complex64, device="cuda") for _ in range(pols)]
    side = torch.cuda.Stream()
    for call in range(6):
        for p in x:
            p.fill_(3.0 if pols == 1 else complex(0.0, 3.0))
        torch.cuda.synchronize()
        f.calculate_intensity(*x)
        with torch.cuda.stream(side):  # another stream: nothing orders it after the fold's
            for p in x:
                p.fill_(-100.0)
        f.fold_data()
        assert np.all(f.total_intensity == np.float32(np.sqrt(9.0 * pols)))
        torch.cuda.synchronize()


@pytest.mark.gpu
def test_raw_pointers_equal_handles():
    """Two overlap-save polarisations through their handles and through their
    series' addresses: the same profile, bit for bit."""
    bw, f0, fft, count = 4e6, 1248e6, 2048, 16
    pols = [Dedisperser(bw, [2.0], f0, fft, count, osm=True) for _ in range(2)]
    n = pols[0].block_samples
    folds = [Fold_GPU((1500.25) / bw, bw, n, time_bin=100) for _ in range(2)]
    rng = np.random.default_rng(3)
    for _ in range(4):
        for d in pols:
            d.filter_block((rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64))
        folds[0].calculate_intensity(*pols)
        folds[1].calculate_intensity(*[d.output_device_ptr() for d in pols])
        for f in folds:
            f.fold_data()
    a, b = (f.fold_data_bins() for f in folds)
    assert np.abs(a).max() > 0 and np.array_equal(a, b)
