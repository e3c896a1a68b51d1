"""Weight gradients of long runs of tiles (csrc/sepx_unet_wgring.inc) against
64-bit sums: the accumulators are read out several times a run, because the
tensor cores truncate as they add.

Tolerance: truncation loses half a unit in the last place of the running sum
per MMA, at most 2^-24 of it; as the sum grows in proportion to the MMAs done,
that is 2^-25 of the final one per MMA on average.  A tile is eight MMAs, so
an accumulator that takes `tiles` tiles may be off by 8 * tiles * 2^-25; the
FP32 additions of the read-outs and partial sums round to nearest, 5e-7 for
all of them.  (ReLU activations, so that the sums grow as in training.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# cin, cout, nb, D, H, W, tiles an accumulator takes at most on 152 SMs: all
# taps in one CTA (16 channels; two blocks), one sy a CTA, two row blocks, one
# dz per MMA
CASES = [(8, 16, 4, 64, 64, 64, 16), (16, 16, 2, 96, 100, 90, 28), (32, 48, 4, 64, 64, 64, 47),
         (64, 64, 2, 64, 64, 64, 32), (112, 48, 2, 64, 64, 64, 62), (80, 32, 2, 64, 64, 64, 32)]


@pytest.mark.parametrize("cin,cout,nb,D,H,W,tiles", CASES)
def test_accumulator_chains_are_bounded(cin, cout, nb, D, H, W, tiles):
    from sep_code_gb300 import unet as net
    from sep_code_gb300._lib import lib
    lib.sepx_setup_cuda(1)
    st = lib.sepx_get_stream()
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    V = nb * D * H * W
    x = torch.relu(torch.randn((V, cin), device="cuda", generator=g)).to(torch.bfloat16)
    dy = torch.randn((V, cout), device="cuda", generator=g).to(torch.bfloat16)
    outs = []
    for _ in range(2):
        dw = torch.zeros((27, cin, cout), device="cuda")
        db = torch.zeros(cout, device="cuda")
        torch.cuda.synchronize()
        net._chk(lib.sepx_unet_conv_wgrad_bias(net._p(x), cin, 0, nb, D, H, W, cin, 27, net._p(dy), cout, 0, cout,
                                               net._p(dw), net._p(db), st))
        lib.sepx_synchronize()
        assert lib.sepx_unet_status() == 0
        outs.append((dw, db))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    X = torch.nn.functional.pad(x.double().view(nb, D, H, W, cin), (0, 0, 1, 1, 1, 1, 1, 1))
    Y = dy.double()
    want = torch.stack([X[:, t // 9:t // 9 + D, t // 3 % 3:t // 3 % 3 + H, t % 3:t % 3 + W].reshape(-1, cin).t() @ Y
                        for t in range(27)])
    err = float((outs[0][0].double() - want).norm() / want.norm())
    assert err <= 8 * tiles * 2.0 ** -25 + 5e-7, err
    b = Y.sum(0)
    assert float((outs[0][1].double() - b).norm() / b.norm()) <= 5e-7
