"""Precision of the DM-proposal network's sums against FP64.

Weight gradient of one layer over samples and phases of products of one sign
(inputs and gradients positive).  An FP32 addition rounds its result by 0.42 x
2^-24 of it in the mean (half an ulp, uniform, over mantissas as they come), a
chain of n equal terms by sqrt(n / 3) times that, and independent chains average
out.  A value is the sum of 64 or more blocks' chains of at most 256 terms
(256 / 3 / 64), four warps of each in order (4 / 3 / 16), the FP64 sum of the
blocks, and its rounding (1): 0.42 sqrt(2.4) = 0.66 x 2^-24.  With the blocks
added in FP32, eight slices in order (8 / 3), it would be 0.96.  Bound: 0.75.

Heads: FP64 sums rounded once, 2^-24 of the sum of magnitudes at most beside the
pooled values' own error (their 32 + 5 additions of values of one sign)."""
import numpy as np
import pytest

import cnn_ref as R
from msosm_gpu_b200.dm_proposal import DMProposalNet

pytestmark = pytest.mark.gpu

BOUND = 0.75 * 2.0 ** -24


@pytest.mark.parametrize("cin,length,channels,B", [(64, 256, 32, 256), (16, 1024, 8, 64), (32, 128, 32, 1024)])
def test_sums_of_one_layer(cin, length, channels, B):
    kernel, layers = 7, 1
    net = DMProposalNet(cin, length, channels, kernel, layers, max_batch=B, dm_weight=0.0, seed=1)
    rng = np.random.default_rng(B)
    th = net.params()
    conv = channels * cin * kernel
    th[:conv] = np.abs(th[:conv])  # every activation and, with label 0, every gradient positive
    th[-2 * channels - 2:-channels - 2] = np.abs(th[-2 * channels - 2:-channels - 2]) * 0.01
    net.set_params(th)
    x = rng.random((B, cin, length)).astype(np.float32)
    zero = np.zeros(B, np.float32)
    a = (cin, channels, kernel, layers)
    _, g = net.gradient(x, zero, zero, want_grad=True)
    _, rg, _, _ = R.loss_and_grad(th, x, zero, zero, *a, 0.0)
    err = np.linalg.norm(g[:conv] - rg[:conv]) / np.linalg.norm(rg[:conv])
    print("dw", cin, length, channels, B, err * 2 ** 24)
    assert rg[:conv].min() > 0 and err < BOUND
    logit, off = net.forward(x)
    rl, ro, _, h, ps = R.forward(th, x, *a)
    for got, ref, w in ((logit, rl, ps[2]), (off, ro, ps[4])):
        e = np.abs(got - ref) / (h @ np.abs(w))
        print("head", np.sqrt(np.mean(e ** 2)) * 2 ** 24)
        assert np.sqrt(np.mean(e ** 2)) < 2.0 ** -24 * (1 + np.sqrt(37) / np.sqrt(3))
    net.close()
