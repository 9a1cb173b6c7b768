"""Folding: the span table as a launch parameter and through its staging (at,
just below and just above the limit), the reduction of partial rows in both
forms, profiles too long for shared memory, periods left open over several
calls, and Fold_GPU's direct fold from one sample a bin to bins longer than a
call -- against the FP64 oracle (relative RMS 2e-5, the fold tests' bound)."""
import numpy as np
import pytest

import oracle as O
from msosm_gpu_b200 import Dedisperser
from msosm_gpu_b200.fold import Fold_GPU

pytestmark = pytest.mark.gpu

BW, F0, RTOL = 4e6, 1248e6, 2e-5


def rel_rms(a, b):
    return float(np.sqrt(np.mean(np.abs(a - b) ** 2) / max(np.mean(np.abs(b) ** 2), 1e-300)))


@pytest.mark.parametrize("trials,ps,bins", [
    (3, 64, 64),       # 130 spans in a call: through the staging
    (3, 65, 13),       # 127 or 128
    (16, 4100, 1024),  # 16384 values: the 16-byte reduction
    (16, 4100, 1023),  # 16368: the other form
    (33, 2055, 685),   # not a multiple of four
    (2, 5000, 5000),   # more bins than shared memory keeps
    (2, 30000, 100),   # a period open over four calls
])
def test_fused_fold(trials, ps, bins):
    fft, count, calls = 512, 32, 14
    dms = np.linspace(0.0, 0.4, trials).astype(np.float32)
    d = Dedisperser(BW, dms, F0, fft, count, series=False)
    assert d.fftpoint == fft
    period = (ps + 0.25) / BW
    d.fold_init(period, BW, time_bin=bins, discard_Nd=1)
    assert d.period_samples == ps
    o = O.Dedisp(BW, dms, F0, fft, count)
    folds = [O.Fold(period, BW, d.block_samples, time_bin=bins) for _ in dms]
    for f in folds:
        f.discard_samples(1)
    rng = np.random.default_rng(ps)
    for _ in range(calls):
        x = (rng.standard_normal(d.block_samples) + 1j * rng.standard_normal(d.block_samples)).astype(np.complex64)
        d.filter_block(x)
        for f, y in zip(folds, o.filter(x.astype(np.complex128))):
            f.fold_data(np.abs(y) ** 2)
    ref = np.stack([f.fold_data_bins() for f in folds])
    assert np.abs(ref).max() > 0
    assert rel_rms(d.get_profiles(), ref) < RTOL


@pytest.mark.parametrize("size,ps,bins", [
    (8192, 64, 64),        # 129 spans
    (8192, 65, 5),
    (8192, 97, 97),
    (50000, 777, 7),
    (50000, 8193, 8193),
    (4096, 20000, 3),      # a call shorter than a bin
    (1 << 20, 49600, 1024),
])
def test_series_fold(size, ps, bins):
    fs = 1e6
    period = (ps + 0.25) / fs
    g, o = Fold_GPU(period, fs, size, time_bin=bins), O.Fold(period, fs, size, time_bin=bins)
    assert (g.period_samples, g.time_bin) == (ps, bins) == (o.period_samples, o.time_bin)
    g.discard_samples(1)
    o.discard_samples(1)
    rng = np.random.default_rng(size + ps)
    for _ in range(max(4, 3 * ps // size + 2)):
        x = rng.random(size).astype(np.float32)
        g.set_intensity(x)
        g.fold_data()
        o.fold_data(x)
    ref = o.fold_data_bins()
    assert np.abs(ref).max() > 0
    assert rel_rms(g.fold_data_bins(), ref) < RTOL
