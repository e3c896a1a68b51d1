"""The convolution that pools its output in the epilogue gives the bits of the
convolution followed by the pooling kernel: tile and window edges, one to five
column blocks, and the shapes that fall back to the two kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# (cin, cout, nb, D, H, W): one plane pair, uneven windows, ragged even rows
# and columns, cout that is no multiple of 16; the last three fall back (rows
# fewer than a tile's, weights that do not fit, 96 output channels)
CASES = [(16, 16, 1, 2, 16, 8), (8, 16, 2, 38, 18, 10), (32, 24, 1, 10, 46, 30), (48, 48, 1, 6, 32, 24),
         (32, 80, 2, 8, 16, 14), (24, 8, 1, 50, 130, 94), (16, 16, 1, 4, 8, 8), (112, 48, 1, 4, 16, 16),
         (16, 96, 1, 4, 16, 16)]


@pytest.mark.parametrize("relu", [0, 1])
@pytest.mark.parametrize("cin,cout,nb,D,H,W", CASES)
def test_conv_pool_bits(cin, cout, nb, D, H, W, relu):
    from sep_code_gb300 import unet as net
    from sep_code_gb300._lib import lib
    lib.sepx_setup_cuda(1)
    st = lib.sepx_get_stream()
    g = torch.Generator().manual_seed(D * 1000 + H + cin)
    V = nb * D * H * W
    x = torch.randn((V, cin), generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn((27, cin, cout), generator=g) / np.sqrt(27 * cin)).cuda()
    b = torch.randn(cout, generator=g).cuda()
    pk = torch.zeros(lib.sepx_unet_packed_elems(cout, cin, 27, 0), dtype=torch.bfloat16).cuda()
    y = [torch.full((V, cout + 16), -3.0, dtype=torch.bfloat16).cuda() for _ in range(2)]
    p = [torch.full((V // 8, cout + 8), 9.0, dtype=torch.bfloat16).cuda() for _ in range(2)]
    torch.cuda.synchronize()
    P = net._p
    net._chk(lib.sepx_unet_pack_weights(P(w), cout, cin, 27, 0, P(pk), st))
    net._chk(lib.sepx_unet_conv_fwd_pool(P(x), cin, 0, nb, D, H, W, cin, 27, P(pk), P(b), cout, relu, P(y[0]), cout + 16,
                                         8, P(p[0]), cout + 8, 8, st))
    net._chk(lib.sepx_unet_conv_fwd(P(x), cin, 0, nb, D, H, W, cin, 27, P(pk), P(b), cout, relu, P(y[1]), cout + 16, 8,
                                    None, None, st))
    net._chk(lib.sepx_unet_avgpool(P(y[1]), cout + 16, 8, nb, D, H, W, cout, P(p[1]), cout + 8, 8, st))
    lib.sepx_synchronize()
    assert lib.sepx_unet_status() == 0
    assert torch.equal(y[0].cpu().view(torch.int16), y[1].cpu().view(torch.int16))
    assert torch.equal(p[0].cpu().view(torch.int16), p[1].cpu().view(torch.int16))
