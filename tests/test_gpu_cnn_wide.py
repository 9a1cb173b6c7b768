"""The DM-proposal network's widest kernels over its shortest profiles, where the
weights of a whole block of channels exceed a block's shared memory: forward
and gradient against the FP64 restatement (oracle/cnn_ref.py) at the bounds of
the other tests of this network (1e-4)."""
import numpy as np
import pytest

import cnn_ref as R
from msosm_gpu_b200.dm_proposal import DMProposalNet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,channels,kernel", [
    (8, 112, 15),   # the widest that fits whole
    (8, 120, 15),   # fifteen channel groups: eight and seven
    (16, 128, 15),
    (128, 256, 15),
    (8, 128, 13),
])
def test_short_profiles_with_wide_kernels(cin, channels, kernel):
    length, layers, B = 32, 2, 3
    net = DMProposalNet(cin, length, channels, kernel, layers, max_batch=B, dm_weight=0.25, seed=1)
    rng = np.random.default_rng(channels)
    th = net.params() + rng.standard_normal(net.n_params).astype(np.float32) * 0.02
    net.set_params(th)
    x = rng.standard_normal((B, cin, length)).astype(np.float32)
    y = (np.arange(B) % 2 == 0).astype(np.float32)
    t = rng.standard_normal(B).astype(np.float32)
    a = (cin, channels, kernel, layers)
    logit, off = net.forward(x)
    rl, ro, _, _, _ = R.forward(th, x, *a)
    np.testing.assert_allclose(logit, rl, rtol=1e-4, atol=1e-5)
    np.testing.assert_allclose(off, ro, rtol=1e-4, atol=1e-5)
    loss, g = net.gradient(x, y, t, want_grad=True)
    rloss, rg, _, _ = R.loss_and_grad(th, x, y, t, *a, 0.25)
    assert abs(loss - rloss) <= 1e-5 * max(1.0, abs(rloss))
    o = 0
    for kind, shp in R.shapes(*a):
        n = int(np.prod(shp))
        gb, rb = g[o:o + n].astype(np.float64), rg[o:o + n]
        err = np.linalg.norm(gb - rb) / max(np.linalg.norm(rb), 1e-12)
        assert err < 1e-4, (kind, shp, err)
        o += n
    net.close()
