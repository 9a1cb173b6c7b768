"""Transforms above one thread block: every split of the sizes 2^15 .. 2^22 into
columns and rows, one trial without block delays (both row passes in one kernel)
and several trials (spectra through the ring), uint16 and complex input, against
the FP64 oracle (relative RMS 2e-5, the FP32 path's bound)."""
import numpy as np
import pytest

import oracle as O
from msosm_gpu_b200 import Dedisperser

pytestmark = pytest.mark.gpu

BW, F0, RTOL = 16e6, 1242e6, 2e-5


def rel_rms(a, b):
    return float(np.sqrt(np.mean(np.abs(a - b) ** 2) / max(np.mean(np.abs(b) ** 2), 1e-300)))


@pytest.mark.parametrize("log2n,dms,count,calls,kind", [
    (15, [3.0], 3, 2, "c64"),
    (15, [3.0, 5.0], 2, 2, "u16"),
    (16, [10.0], 2, 2, "u16"),
    (17, [20.0], 2, 1, "c64"),
    (18, [40.0, 50.0], 1, 2, "u16"),
    (19, [50.0], 1, 2, "c64"),
    (20, [50.0], 2, 1, "u16"),
    (21, [50.0], 1, 2, "u16"),
    (22, [60.0], 1, 1, "c64"),
])
def test_overlap_save_sizes(log2n, dms, count, calls, kind):
    fft = 1 << log2n
    d = Dedisperser(BW, dms, F0, fft, count, osm=True)
    assert d.fftpoint == fft
    o = O.Dedisp(BW, dms, F0, fft, count, osm=True)
    rng = np.random.default_rng(log2n)
    for _ in range(calls):
        n = d.block_samples
        if kind == "c64":
            x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
            xo = x.astype(np.complex128)
        else:
            x = np.clip(np.rint(rng.standard_normal((n, 2)) * 900) + 32768, 0, 65535).astype(np.uint16)
            xo = O.decode_uint16(x)
        d.filter_block(x)
        assert rel_rms(d.get_output(), o.filter(xo)) < RTOL


def test_multi_segment_one_trial_with_and_without_delays():
    """MS-OSM at 2^16: DM 0 (no block delays, one row pass) and a DM whose
    smear spans several blocks (spectra through the ring)."""
    for dm in (0.0, 60.0):
        d = Dedisperser(BW, [dm], F0, 1 << 16, 2)
        o = O.Dedisp(BW, [dm], F0, 1 << 16, 2)
        rng = np.random.default_rng(3)
        for _ in range(4):
            n = d.block_samples
            x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
            d.filter_block(x)
            assert rel_rms(d.get_output(), o.filter(x.astype(np.complex128))) < RTOL
