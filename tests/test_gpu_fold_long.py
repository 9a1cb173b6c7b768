"""Folding of materialised series into long bins: periods of many calls, one bin,
bins below, at and above the length at which whole blocks share a bin, rows that
begin in the tail no bin covers, several trials; and the time of a call, which
must not depend on how the period is cut into bins."""
import time

import numpy as np
import pytest

import oracle as O
from msosm_gpu_b200 import Dedisperser
from msosm_gpu_b200.fold import Fold_GPU

pytestmark = pytest.mark.gpu

# Positive samples: every addition adds at most 2^-24 of the sum.  A sample
# passes at most 32 + 3 + 8 + 5 of them in FP32 (its accumulator, the four of a
# lane, eight spans, the lanes of a warp), the FP64 sums are rounded to FP32 per
# row and at the end, and the scale by 1 / samples a bin rounds once more.
BOUND = 51 * 2.0 ** -24


@pytest.mark.parametrize("size,ps,bins", [
    (1 << 16, 100000, 97),      # 1030 samples a bin, a tail of 90
    (1 << 16, 1024 * 40, 40),   # exactly 1024
    (1 << 16, 1025 * 40, 40),
    (30000, 1500, 1),           # many short periods in a row of samples
    (30001, 2 * 2100, 2),
    (4097, 50000, 3),           # a call shorter than a bin
    (1 << 18, 300007, 7),       # a tail
    (1 << 20, 700001, 4),
    (1 << 20, 65537, 64),
    (12345, 5 * 4096 + 4095, 5),
    (1 << 21, 1500 * 20, 20),   # 1398 bins of 1500 in a call: a warp each
    (1 << 22, 4096 * 3 + 2, 3),  # 1024 of 4096
    (1 << 22, 4097 * 3, 3),     # 4097: whole blocks again
])
def test_long_bins(size, ps, bins):
    fs = 1e6
    period = (ps + 0.25) / fs
    g, o = Fold_GPU(period, fs, size, time_bin=bins), O.Fold(period, fs, size, time_bin=bins)
    assert (g.period_samples, g.time_bin) == (o.period_samples, bins)
    g.discard_samples(1)
    o.discard_samples(1)
    rng = np.random.default_rng(size + ps)
    for _ in range(max(4, 3 * g.period_samples // size + 2)):
        x = rng.random(size).astype(np.float32)
        g.set_intensity(x)
        g.fold_data()
        o.fold_data(x)
    ref = o.fold_data_bins()
    assert ref.min() > 0
    assert np.abs(g.fold_data_bins() / ref - 1.0).max() < BOUND


@pytest.mark.parametrize("trials,ps,bins", [(1, 60000, 3), (5, 60000, 50), (5, 9000, 2)])
def test_long_bins_of_a_long_transform(trials, ps, bins):
    """The series fold behind the four-step transforms, against the profile of
    the series it read (relative RMS 2e-5, the fold tests' bound)."""
    bw, fft, count = 4e6, 1 << 15, 2
    dms = np.linspace(0.0, 30.0, trials).astype(np.float32)
    d = Dedisperser(bw, dms, 1248e6, fft, count)
    period = (ps + 0.25) / bw
    d.fold_init(period, bw, time_bin=bins, discard_Nd=1)
    folds = [O.Fold(period, bw, d.block_samples, time_bin=bins) for _ in dms]
    for f in folds:
        f.discard_samples(1)
    rng = np.random.default_rng(ps)
    for _ in range(max(3, 3 * ps // d.block_samples + 2)):
        d.filter_block((rng.standard_normal(d.block_samples) + 1j * rng.standard_normal(d.block_samples)).astype(np.complex64))
        for f, y in zip(folds, d.get_output()):
            f.fold_data(np.abs(y.astype(np.complex128)) ** 2)
    ref = np.stack([f.fold_data_bins() for f in folds])
    assert ref.min() > 0
    err = np.sqrt(np.mean((d.get_profiles() - ref) ** 2) / np.mean(ref ** 2))
    assert err < 2e-5


def test_time_does_not_depend_on_the_bins():
    import torch

    def us(ps, bins):
        f = Fold_GPU((ps + 0.25) / 16e6, 16e6, 1 << 20, time_bin=bins)
        f.set_intensity(np.ones(1 << 20, np.float32))
        t = []
        for _ in range(12):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            f.fold_data()
            f.fold_data_bins()
            t.append(time.perf_counter() - t0)
        return 1e6 * float(np.median(t))

    base = us(49600, 1024)
    for ps, bins in ((11200000, 4), (11200000, 64), (524288, 4), (49600, 1)):
        assert us(ps, bins) < 4 * base, (ps, bins)  # 50 to 70 times with a period's lanes alone
