"""The packed FP32 dedispersion kernel (two blocks per step, or one block split
in two at 16384 points) and the fold it shares with the tensor-core kernel, at
every block FFT size, with block counts below, at and just past a whole step and
bins of one sample up to more than a lane group sums at once: series and folded
profiles against the FP64 oracle (relative RMS 2e-5, the FP32 path's bound)."""
import numpy as np
import pytest

import oracle as O
from msosm_gpu_b200 import Dedisperser

pytestmark = pytest.mark.gpu

BW, F0 = 4e6, 1248e6
RTOL = 2e-5


def rel_rms(a, b):
    return float(np.sqrt(np.mean(np.abs(a - b) ** 2) / max(np.mean(np.abs(b) ** 2), 1e-300)))


def blocks_per_step(log2n):
    return 1 if log2n == 14 else max(1, 2 * 4096 // (1 << log2n)) * (1 if log2n < 13 else 2)


# (samples per period, output bins): one sample a bin; odd short bins; a bin a
# lane sums alone and the next longer one; the longest lane groups
BINS = [(97, 97), (1003, 143), (2048, 64), (2145, 65), (9000, 4)]


@pytest.mark.parametrize("log2n", range(6, 15))
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_step_edges_and_bins(log2n, extra):
    fft = 1 << log2n
    m = fft // 2
    bps = blocks_per_step(log2n)
    count = max(1, 2 * bps + extra)
    ps, bins = BINS[(log2n + extra) % len(BINS)]
    period = (ps + 0.25) / BW
    dms = [0.0, 0.004 * (m / 32) ** 2, 0.006 * (m / 32) ** 2] if log2n < 12 else [0.0, 20.0, 57.0]
    rng = np.random.default_rng(100 * log2n + extra)
    both = Dedisperser(BW, dms, F0, fft, count)
    only = Dedisperser(BW, dms, F0, fft, count, series=False)
    assert both.fftpoint == fft
    discard = max(1, int(both.Nd.max()))  # with 0 the reference's Fold_GPU (and the oracle) folds nothing
    for d in (both, only):
        d.fold_init(period, BW, time_bin=bins, discard_Nd=discard)
        assert d.period_samples == ps
    o = O.Dedisp(BW, dms, F0, fft, count)
    folds = []
    for _ in dms:
        f = O.Fold(period, BW, count * m, time_bin=bins)
        f.discard_samples(discard)
        folds.append(f)
    calls = max(2, -(-(discard + 3 * ps) // (count * m)))
    for _ in range(calls):
        x = (rng.standard_normal(count * m) + 1j * rng.standard_normal(count * m)).astype(np.complex64)
        both.filter_block(x)
        only.filter_block(x)
        y = o.filter(x.astype(np.complex128))
        assert rel_rms(both.get_output(), y) < RTOL
        for f, s in zip(folds, y):
            f.fold_data(np.abs(s) ** 2)
    ref = np.stack([f.fold_data_bins() for f in folds])
    assert np.abs(ref).max() > 0
    for d in (both, only):
        assert rel_rms(d.get_profiles(), ref) < RTOL
    assert np.array_equal(both.get_profiles(), only.get_profiles())


def test_many_items_take_the_counter_round():
    """More work items than resident thread blocks, twice over the same handle
    (the item counter is back at zero), equal to one trial at a time."""
    dms = np.linspace(0.0, 3.0, 700).astype(np.float32)
    rng = np.random.default_rng(5)
    xs = [(rng.standard_normal(64 * 512) + 1j * rng.standard_normal(64 * 512)).astype(np.complex64) for _ in range(2)]
    d = Dedisperser(16e6, dms, 1242e6, 1024, 64)
    for x in xs:
        d.filter_block(x)
    y = d.get_output()
    for i in (0, 333, 699):
        one = Dedisperser(16e6, dms[i:i + 1], 1242e6, 1024, 64)
        for x in xs:
            one.filter_block(x)
        assert np.array_equal(y[i], one.get_output()[0])
