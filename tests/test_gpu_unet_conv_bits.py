"""Convolution kernels that add an output's terms in the same order give the same
bits: the z-walk kernel (csrc/sepx_unet_zwfwd.inc) those of the halo-staged one,
the one with streamed weights (csrc/sepx_unet_kstream.inc) those of the gather
kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# (cin, cout, nb, D, H, W): layers that both kernels sum in one range (304 and
# more tiles of 128 voxels, so that the gather kernel does not split K either
# with the halo kernels on)
ONE_RANGE = [(112, 48, 1, 41, 33, 40), (48, 112, 2, 23, 31, 40), (160, 16, 1, 19, 48, 56), (16, 128, 2, 60, 8, 48)]


@pytest.mark.parametrize("cin,cout,nb,D,H,W", ONE_RANGE)
def test_streamed_weights_give_the_bits_of_the_gather_kernel(cin, cout, nb, D, H, W):
    from sep_code_gb300 import unet as net
    from sep_code_gb300._lib import lib
    lib.sepx_setup_cuda(1)
    st = lib.sepx_get_stream()
    g = torch.Generator().manual_seed(cin * cout)
    V = nb * D * H * W
    x = torch.randn((V, cin), generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn((27, cin, cout), generator=g) / np.sqrt(27 * cin)).cuda()
    pk = torch.zeros(lib.sepx_unet_packed_elems(cout, cin, 27, 0), dtype=torch.bfloat16).cuda()
    outs = []
    torch.cuda.synchronize()
    net._chk(lib.sepx_unet_pack_weights(net._p(w), cout, cin, 27, 0, net._p(pk), st))
    for halo in (1, 0):
        yf = torch.zeros((V, cout)).cuda()
        torch.cuda.synchronize()
        prev = lib.sepx_unet_set_halo(halo)
        try:
            net._chk(lib.sepx_unet_conv_fwd(net._p(x), cin, 0, nb, D, H, W, cin, 27, net._p(pk), None, cout, 0, None,
                                            0, 0, net._p(yf), None, st))
        finally:
            lib.sepx_unet_set_halo(prev)
        lib.sepx_synchronize()
        outs.append(yf.cpu())
    assert lib.sepx_unet_status() == 0
    assert torch.equal(outs[0].view(torch.int32), outs[1].view(torch.int32))

@pytest.mark.parametrize("pair", [(16, 96, 80, 2, 21, 33, 26), (24, 128, 16, 1, 9, 48, 40), (32, 112, 48, 1, 13, 40, 19),
                                  (8, 96, 16, 1, 30, 70, 70)])
def test_zwalk_gives_the_bits_of_the_halo_kernel(pair):
    """A layer's first channels as a narrower layer of their own: the z-walk
    kernel adds every output's terms in the order of the halo-staged one, so
    both give the same bits."""
    from sep_code_gb300 import unet as net
    from sep_code_gb300._lib import lib
    cin, wide, narrow, nb, D, H, W = pair
    lib.sepx_setup_cuda(1)
    st = lib.sepx_get_stream()
    g = torch.Generator().manual_seed(cin * wide)
    V = nb * D * H * W
    x = torch.randn((V, cin), generator=g).to(torch.bfloat16).cuda()
    w = torch.randn((27, cin, wide), generator=g) / np.sqrt(27 * cin)
    outs = []
    for cout in (wide, narrow):
        wt = w[..., :cout].contiguous().cuda()
        pk = torch.zeros(lib.sepx_unet_packed_elems(cout, cin, 27, 0), dtype=torch.bfloat16).cuda()
        yf = torch.zeros((V, cout)).cuda()
        torch.cuda.synchronize()
        net._chk(lib.sepx_unet_pack_weights(net._p(wt), cout, cin, 27, 0, net._p(pk), st))
        net._chk(lib.sepx_unet_conv_fwd(net._p(x), cin, 0, nb, D, H, W, cin, 27, net._p(pk), None, cout, 0, None, 0, 0,
                                        net._p(yf), None, st))
        lib.sepx_synchronize()
        outs.append(yf[:, :narrow].cpu())
    assert lib.sepx_unet_status() == 0
    assert torch.equal(outs[0].view(torch.int32), outs[1].view(torch.int32))
