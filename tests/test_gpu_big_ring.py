"""Spectrum rings above 4 GB, which the FP32 kernel no longer addresses with
32-bit byte offsets: one long call against the same stream in three calls of a
handle whose ring stays below, bit for bit (17 GB on the device)."""
import numpy as np
import pytest

from msosm_gpu_b200 import Dedisperser

pytestmark = pytest.mark.gpu


class Series:
    def __init__(self, d):
        self.handle = d
        self.__cuda_array_interface__ = {"data": (d.output_device_ptr(), False), "shape": (d.block_samples,),
                                         "typestr": "<c8", "version": 3}


@pytest.mark.parametrize("fft,third", [(4096, 43691), (16384, 10923)])
def test_one_long_call_equals_three(fft, third):
    import torch
    bw, f0, m = 16e6, 1242e6, fft // 2
    g = torch.Generator(device="cuda").manual_seed(fft)
    x = torch.view_as_complex(torch.randn(3 * third * m, 2, generator=g, device="cuda"))
    torch.cuda.synchronize()
    long, short = (Dedisperser(bw, [60.0], f0, fft, c) for c in (3 * third, third))
    assert long.fftpoint == short.fftpoint == fft and 2 < int(long.delaycount[0])
    assert long.ring_slots * fft * 8 > 1 << 32 >= short.ring_slots * fft * 8
    long.filter_block(x)
    long.synchronize()
    y = torch.as_tensor(Series(long), device="cuda")
    n = third * m
    for i in range(3):
        short.filter_block(x[i * n:(i + 1) * n])
        short.synchronize()
        assert torch.equal(torch.view_as_real(y[i * n:(i + 1) * n]),
                           torch.view_as_real(torch.as_tensor(Series(short), device="cuda")))
    assert float(y[-n:].abs().max()) > 0
