"""A handle without series and without a fold has nowhere to write its output:
its filter calls are refused before anything is launched, alone and in a batch,
and the handle goes on once the fold is configured."""
import numpy as np
import pytest

from msosm_gpu_b200 import DedispBatch, Dedisperser, _abi

pytestmark = pytest.mark.gpu

BW, F0 = 16e6, 1242e6


@pytest.mark.parametrize("fft,precision", [(64, "fp32"), (4096, "fp32"), (16384, "fp32"), (4096, "fp16"),
                                           (8192, "fp16"), (16384, "bf16")])
def test_filter_without_output_is_refused(fft, precision):
    import torch
    dms = [0.0, 0.001] if fft < 4096 else [0.0, 5.0]
    ours, ref = (Dedisperser(BW, dms, F0, fft, 9, series=False, precision=precision) for _ in range(2))
    n = ours.block_samples
    rng = np.random.default_rng(fft)
    x = torch.from_numpy((rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)).cuda()
    for call in (lambda: ours.filter_block(x), lambda: DedispBatch([ours]).filter_block([x])):
        with pytest.raises(_abi.MsosmError) as e:
            call()
        assert e.value.status == _abi.ERR_STATE
    for d in (ours, ref):
        d.fold_init(500.25 / BW, BW, time_bin=50, discard_Nd=1)
        for _ in range(max(3, -(-2000 // n))):  # some whole periods after the discarded one
            d.filter_block(x)
    p = ours.get_profiles()
    assert np.abs(p).max() > 0 and np.array_equal(p, ref.get_profiles())
