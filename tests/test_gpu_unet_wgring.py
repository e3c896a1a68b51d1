"""The ring form of the tap-stacked weight gradient
(csrc/sepx_unet_wgring.inc) at the edges of its plans, against the FP64
restatement: one and three sy per CTA, one and two blocks of 128 rows, MMAs
over three planes at once and per plane, rings that wrap in every phase.

Tolerance: every sum has the same BF16 products as the FP64 one and differs by
FP32 accumulation order: relative L2 <= 1e-5, as the other weight-gradient
tests.  Partial sums are added in a fixed order: two runs give the same bits."""
import numpy as np
import pytest

from oracle import unet_oracle as U
from tests.harness import rel_l2

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# cin, cout, nb, D, H, W: the two narrowest layers; N = 8 per dz (odd groups,
# 128 rows); long windows; one sy per CTA; two row blocks (48, 56, 64 outputs);
# one dz per MMA (112 inputs); the widest combination the kernel takes; many
# windows per CTA
CASES = [(8, 1, 1, 1, 1, 1), (8, 16, 2, 5, 33, 7), (24, 32, 1, 4, 17, 30), (16, 8, 1, 71, 16, 8),
         (48, 16, 1, 23, 50, 41), (32, 32, 2, 17, 20, 22), (80, 32, 1, 9, 18, 15), (32, 48, 1, 6, 16, 16),
         (48, 48, 2, 5, 16, 16), (64, 64, 4, 8, 8, 8), (48, 56, 1, 3, 9, 31), (112, 48, 1, 7, 16, 17),
         (104, 40, 1, 4, 12, 9), (16, 16, 2, 48, 96, 96), (32, 24, 1, 64, 96, 80)]


@pytest.mark.parametrize("cin,cout,nb,D,H,W", CASES)
def test_ring_weight_gradient(cin, cout, nb, D, H, W):
    from sep_code_gb300 import unet as net
    from sep_code_gb300._lib import lib
    lib.sepx_setup_cuda(1)
    st = lib.sepx_get_stream()
    rng = np.random.default_rng(cin * 1000 + cout + D)
    V, cp = nb * D * H * W, (cout + 7) // 8 * 8
    x = U.bf16(rng.standard_normal((nb, D, H, W, cin)))
    dy = np.zeros((nb, D, H, W, cp))
    dy[..., :cout] = U.bf16(rng.standard_normal((nb, D, H, W, cout)))
    xw = np.full((V, cin + 16), np.nan, np.float32)   # slices of wider buffers whose other channels are NaN
    xw[:, 8:8 + cin] = x.reshape(V, cin)
    dw_ = np.full((V, cp + 8), np.nan, np.float32)
    dw_[:, 8:] = dy.reshape(V, cp)
    xt, dt = (torch.tensor(v).to(torch.bfloat16).cuda() for v in (xw, dw_))
    want = U.conv_wgrad(x, dy[..., :cout], 27, cin).ravel() + 0.25
    want_b = dy[..., :cout].sum((0, 1, 2, 3)) - 0.5
    outs = []
    for with_bias in (True, True, False):
        dw = torch.full((27 * cin * cout,), 0.25).cuda()
        db = torch.full((cout,), -0.5).cuda()
        torch.cuda.synchronize()
        net._chk(lib.sepx_unet_conv_wgrad_bias(net._p(xt), cin + 16, 8, nb, D, H, W, cin, 27, net._p(dt), cp + 8, 8,
                                               cout, net._p(dw), net._p(db) if with_bias else None, st))
        lib.sepx_synchronize()
        assert lib.sepx_unet_status() == 0
        outs.append((dw.cpu().numpy(), db.cpu().numpy()))
    assert rel_l2(outs[0][0], want) <= 1e-5
    assert rel_l2(outs[0][1], want_b) <= 1e-5
    assert all(np.array_equal(a, b) for a, b in zip(outs[0], outs[1]))
    assert np.array_equal(outs[0][0], outs[2][0]) and (outs[2][1] == -0.5).all()
