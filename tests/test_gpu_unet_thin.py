"""The z-walk convolution of a packed 8-channel volume (rows of voxels loaded as
runs of memory) gives the bits of the same volume as a slice of a wider buffer
(a row per voxel), at the edges of tiles, rows and windows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("cout,nb,D,H,W", [(16, 1, 1, 16, 8), (16, 2, 3, 17, 9), (24, 1, 35, 18, 41), (48, 3, 8, 33, 16),
                                           (16, 1, 70, 100, 130)])
def test_packed_rows_bits(cout, nb, D, H, W):
    from sep_code_gb300 import unet as net
    from sep_code_gb300._lib import lib
    lib.sepx_setup_cuda(1)
    st = lib.sepx_get_stream()
    g = torch.Generator().manual_seed(D * 1000 + H + W)
    V = nb * D * H * W
    x = torch.randn((V, 8), generator=g).to(torch.bfloat16)
    wide = torch.full((V, 24), 7.0, dtype=torch.bfloat16)
    wide[:, 8:16] = x
    x, wide = x.cuda(), wide.cuda()
    w = (torch.randn((27, 8, cout), generator=g) / np.sqrt(27 * 8)).cuda()
    b = torch.randn(cout, generator=g).cuda()
    pk = torch.zeros(lib.sepx_unet_packed_elems(cout, 8, 27, 0), dtype=torch.bfloat16).cuda()
    out = [torch.zeros((V, cout), device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    P = net._p
    net._chk(lib.sepx_unet_pack_weights(P(w), cout, 8, 27, 0, P(pk), st))
    for o, (src, cs, co) in zip(out, ((x, 8, 0), (wide, 24, 8))):
        net._chk(lib.sepx_unet_conv_fwd(P(src), cs, co, nb, D, H, W, 8, 27, P(pk), P(b), cout, 0, None, 0, 0, P(o), None,
                                        st))
    lib.sepx_synchronize()
    assert lib.sepx_unet_status() == 0
    assert torch.equal(out[0].cpu().view(torch.int32), out[1].cpu().view(torch.int32))
    assert float(out[0].abs().max()) > 0
