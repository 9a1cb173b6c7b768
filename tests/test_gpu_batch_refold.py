"""Members of a batch that start a new stream with another fold, or none, or
get their first fold, after the batch was made: every result equals that of the
same calls through handles of their own, bit for bit."""
import numpy as np
import pytest

from msosm_gpu_b200 import DedispBatch, Dedisperser

pytestmark = pytest.mark.gpu

BW, F0 = 16e6, 1242e6
SHAPES = [([0.0, 3.0, 8.0], 4096, 40), ([1.0, 5.0], 4096, 33), ([0.5, 2.0, 4.0], 8192, 20)]


def configure(d, bins, ps):
    d.fold_init((ps + 0.25) / BW, BW, time_bin=bins, discard_Nd=int(d.Nd.max()))


def test_refolded_members_equal_their_own_calls():
    rng = np.random.default_rng(8)
    ours, own = ([Dedisperser(BW, dms, F0, fft, count, precision="fp16") for dms, fft, count in SHAPES]
                 for _ in range(2))
    for hs in (ours, own):
        configure(hs[0], 64, 5000)
        configure(hs[2], 64, 5000)
    batch = DedispBatch(ours)

    def call():
        xs = [(rng.standard_normal(d.block_samples) + 1j * rng.standard_normal(d.block_samples)).astype(np.complex64)
              for d in ours]
        batch.filter_block(xs)
        for d, x in zip(own, xs):
            d.filter_block(x)
        for a, b in zip(ours, own):
            assert np.array_equal(a.get_output(), b.get_output())
            if a.folding:
                p = a.get_profiles()
                assert np.abs(p).max() > 0 and np.array_equal(p, b.get_profiles())

    call()
    call()
    for hs in (ours, own):
        configure(hs[1], 3000, 6000)     # a first fold
        hs[0].reset()
        configure(hs[0], 4000, 4000)     # more bins than shared memory holds
        hs[2].reset()                    # no fold any more
    call()
    call()
    for hs in (ours, own):
        hs[0].reset()
        configure(hs[0], 16, 300)
        configure(hs[2], 1, 8000)
    call()
    assert batch.info()["groups"] == 2
