"""How a call is cut into block ranges and what that may cost in precision: f16
operands share one scale per range, so a burst must leave the blocks of later
ranges alone; a bin is summed in FP32 over a range, so calls of many periods need
several ranges however many trials there are."""
import numpy as np
import pytest

import oracle as O
from msosm_gpu_b200 import Dedisperser

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fft,trials", [(4096, 296), (8192, 148), (16384, 148), (8192, 1)])
def test_burst_leaves_later_ranges_alone(fft, trials):
    """With eight ranges of the 256 blocks, those from block 64 on lie in ranges
    that neither hold the burst nor gather from it: bit for bit the series
    without it."""
    bw, f0, m, count = 64e6, 1368e6, fft // 2, 256
    dms = np.linspace(0.0, 3.0, trials).astype(np.float32)
    rng = np.random.default_rng(fft)
    x = (rng.standard_normal(count * m) + 1j * rng.standard_normal(count * m)).astype(np.complex64)
    loud = x.copy()
    loud[3 * m:4 * m] += (1e6 * np.exp(2j * np.pi * 0.1234 * np.arange(m))).astype(np.complex64)
    d = Dedisperser(bw, dms, f0, fft, count, precision="fp16")
    assert d.fftpoint == fft and max(d.delaycount) < 24  # 3 + 24 < 32, where the second range begins
    out = []
    for v in (x, loud):
        d.reset()
        d.filter_block(v)
        out.append(d.get_output())
    quiet, burst = (y.reshape(trials, count, m) for y in out)
    assert np.array_equal(quiet[:, 64:], burst[:, 64:])
    assert not np.array_equal(quiet[:, 3], burst[:, 3])


@pytest.mark.parametrize("fft,trials", [(512, 600), (4096, 400), (16384, 100)])  # 12 ranges each, or more
def test_many_periods_and_trials(fft, trials):
    """1310 periods a call of many trials, which leave a trial one range or two.
    Against the profile of the trial's own series in FP64.  Relative RMS: the
    sums over a range 2^-23 / sqrt(12) sqrt(1310 / 3) / R <= 6.9e-8 with R >=
    sqrt(1310 / 12), the result's own rounding 3.4e-8: 1e-7 in all."""
    bw, f0, m = 16e6, 1242e6, fft // 2
    samples, ps, bins = 1 << 21, 1600, 100
    count = samples // m
    dms = np.linspace(0.0, 0.003 if fft < 4096 else 4.0, trials).astype(np.float32)
    rng = np.random.default_rng(fft)
    x = (rng.standard_normal(samples) + 1j * rng.standard_normal(samples)).astype(np.complex64)
    d = Dedisperser(bw, dms, f0, fft, count, series=False)
    assert d.fftpoint == fft
    period = (ps + 0.25) / bw
    d.fold_init(period, bw, time_bin=bins, discard_Nd=1)
    d.filter_block(x)
    p = d.get_profiles()
    for i in (0, trials // 2, trials - 1):
        one = Dedisperser(bw, dms[i:i + 1], f0, fft, count)
        one.filter_block(x)
        y = one.get_output()[0].astype(np.complex128)
        f = O.Fold(period, bw, samples, time_bin=bins)
        f.discard_samples(1)
        f.fold_data(y.real ** 2 + y.imag ** 2)
        ref = f.fold_data_bins()
        err = np.sqrt(np.mean((p[i] - ref) ** 2) / np.mean(ref ** 2))
        print(fft, i, err)
        assert err < 1e-7, (i, err)
