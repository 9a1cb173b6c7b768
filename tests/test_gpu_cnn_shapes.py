"""The convolution kernels of the DM-proposal network at the edges of their
tiles: lengths and channel counts that leave blocks part empty, every kernel
width, one sample and an odd batch, against the FP64 restatement
(oracle/cnn_ref.py).  Forward rtol 1e-4, gradients 1e-4 relative per parameter
block (the bounds of the other tests of this network)."""
import numpy as np
import pytest

import cnn_ref as R
from msosm_gpu_b200.dm_proposal import DMProposalNet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,length,channels,kernel,layers,B", [
    (8, 32, 8, 1, 1, 1),       # smallest of everything
    (8, 32, 40, 3, 2, 3),      # five channel groups, half a warp of phases
    (24, 64, 24, 5, 2, 5),     # an input chunk and a half
    (16, 96, 8, 9, 2, 2),      # phases not a whole block
    (40, 160, 16, 11, 2, 2),   # a ragged second phase block
    (8, 288, 72, 13, 2, 2),    # three output tiles of the weight gradient, the last part empty
    (32, 320, 16, 15, 1, 33),  # widest kernel, odd batch
    (64, 256, 32, 7, 4, 17),   # the defaults
])
def test_forward_and_gradient_at_tile_edges(cin, length, channels, kernel, layers, B):
    import torch
    net = DMProposalNet(cin, length, channels, kernel, layers, max_batch=B + 2, dm_weight=0.25, seed=1)
    rng = np.random.default_rng(length + channels)
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
    # device inputs that are not 16-byte aligned give the same numbers
    buf = torch.zeros(x.size + 1, device="cuda")
    buf[1:] = torch.from_numpy(x).reshape(-1).cuda()
    torch.cuda.synchronize()
    l2, o2 = net.forward(buf[1:].view(B, cin, length))
    assert np.array_equal(l2, logit) and np.array_equal(o2, off)
    net.close()
