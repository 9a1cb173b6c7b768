"""Precision of the four-step transforms: a folded profile against FP64 at the
sizes whose column passes have three stages.  Nearly all of its error is the
rounding of the twiddle factors, which scales every sample of a bin alike, so it
does not average out: with all of a block FFT's factors as products of two table
values 6.3e-7 to 6.9e-7 relative RMS, with rows of 16384 points (and two column
stages) 5.5e-7 to 6.1e-7, with table values 4.6e-7 to 5.1e-7.  Bound: 6e-7."""
import numpy as np
import pytest

import oracle as O
from msosm_gpu_b200 import Dedisperser

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2n,dm,osm", [(20, 5.0, True), (20, 60.0, False), (21, 5.0, True), (21, 60.0, False)])
def test_profile_of_a_four_step_transform(log2n, dm, osm):
    bw, f0, fft, count = 16e6, 1242e6, 1 << log2n, 1 << (22 - log2n)
    period, bins = 0.0031, 1024
    d = Dedisperser(bw, [dm], f0, fft, count, osm=osm)
    assert d.fftpoint == fft
    discard = max(1, int(d.Nd.max()))
    d.fold_init(period, bw, time_bin=bins, discard_Nd=discard)
    f = O.Fold(period, bw, d.block_samples, time_bin=bins)
    f.discard_samples(discard)
    o = O.Dedisp(bw, [dm], f0, fft, count, osm=osm)
    rng = np.random.default_rng(log2n)
    n = d.block_samples
    x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    d.filter_block(x)
    y = o.filter(x.astype(np.complex128))[0]
    f.fold_data(np.abs(y) ** 2)
    ref = f.fold_data_bins()
    err = np.sqrt(np.mean((d.get_profiles()[0] - ref) ** 2) / np.mean(ref ** 2))
    print(log2n, osm, err)
    assert err < 6e-7
