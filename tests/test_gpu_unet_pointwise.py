"""The U-Net's pointwise kernels where their forms change: nearest upsampling of
packed 8-channel volumes (two children per 32-byte store, if the volume is
aligned for it), the 8 -> 16 channel 1x1x1 convolution around the number of
threads of its grid (two voxels a thread, or one), and the network's input with
and without the FP32 copy.

Upsampling and the input are copies: the bits of PyTorch's on the CPU.  The
convolution adds 8 products and a bias in FP32, nine roundings of at most 2^-24
of the terms' sum: 9 * 2^-24 = 5.4e-7 of it; and a voxel's result does not
depend on the volume around it: the same bits in pieces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

GRID = 4 * 152 * 256   # threads of the 1x1x1 convolution's largest grid


def _net():
    from sep_code_gb300 import unet as net
    from sep_code_gb300._lib import lib
    lib.sepx_setup_cuda(1)
    return net, lib, lib.sepx_get_stream()


@pytest.mark.parametrize("off", [0, 8, 16])
@pytest.mark.parametrize("nb,D,H,W", [(1, 1, 1, 1), (2, 3, 5, 7), (1, 8, 33, 64)])
def test_upsample_packed_bits(nb, D, H, W, off):
    net, lib, st = _net()
    x = torch.randn((nb, D, H, W, 8), generator=torch.Generator().manual_seed(W + off)).to(torch.bfloat16)
    n = x.numel() * 8
    y = torch.full((n + 32,), 5.0, dtype=torch.bfloat16, device="cuda")
    xd, yd = x.cuda(), y[off:]
    torch.cuda.synchronize()
    net._chk(lib.sepx_unet_upsample(net._p(xd), 8, 0, nb, D, H, W, 8, net._p(yd), 8, 0, st))
    lib.sepx_synchronize()
    want = x.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3).reshape(-1)
    got = y.cpu()
    assert torch.equal(got[off:off + n].view(torch.int16), want.view(torch.int16))
    assert (got[:off] == 5.0).all() and (got[off + n:] == 5.0).all()


@pytest.mark.parametrize("V", [1, 255, GRID - 1, GRID, GRID + 1, 2 * GRID, 2 * GRID + 5])
def test_conv_8_16_around_the_grid(V):
    net, lib, st = _net()
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randn((V, 8), device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn((1, 8, 16), device="cuda", generator=g)
    b = torch.randn(16, device="cuda", generator=g)
    m = torch.randn((V, 16), device="cuda", generator=g).to(torch.bfloat16)
    pk = torch.zeros(lib.sepx_unet_packed_elems(16, 8, 1, 0), dtype=torch.bfloat16, device="cuda")
    y, yp = (torch.full((V, 24), -3.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    yf = torch.zeros((V, 16), device="cuda")
    torch.cuda.synchronize()
    net._chk(lib.sepx_unet_pack_weights(net._p(w), 16, 8, 1, 0, net._p(pk), st))

    def conv(v0, v1, out, relu, mask, f32):
        net._chk(lib.sepx_unet_conv_fwd_masked(net._p(x[v0:]), 8, 0, 1, 1, 1, v1 - v0, 8, 1, net._p(pk), net._p(b), 16,
                                               relu, net._p(out[v0:]), 24, 8, f32, None,
                                               net._p(mask[v0:]) if mask is not None else None, 16 if mask is not None else 0,
                                               0, st))
    conv(0, V, y, 0, None, net._p(yf))
    lib.sepx_synchronize()
    xs, ws = x.double(), w[0].to(torch.bfloat16).double()
    want, mag = xs @ ws + b.double(), xs.abs() @ ws.abs() + b.double().abs()
    assert bool(((yf.double() - want).abs() <= 9 * 2.0 ** -24 * mag).all())
    assert torch.equal(y[:, 8:], yf.to(torch.bfloat16)) and bool((y[:, :8] == -3.0).all())
    conv(0, V, y, 1, m, None)
    step = 100000
    for v0 in range(0, V, step):
        conv(v0, min(v0 + step, V), yp, 1, m, None)
    lib.sepx_synchronize()
    assert torch.equal(y.view(torch.int16), yp.view(torch.int16))


@pytest.mark.parametrize("V", [1, 777, 300001])
def test_input_with_and_without_the_float_copy(V):
    net, lib, st = _net()
    x = torch.randn(V, generator=torch.Generator().manual_seed(V))
    xd = x.cuda()
    y = [torch.full((V, 16), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    xf = torch.zeros(V, device="cuda")
    torch.cuda.synchronize()
    net._chk(lib.sepx_unet_to_bf16(net._p(xd), V, 0.3, net._p(y[0]), 16, 8, st))
    net._chk(lib.sepx_unet_input(net._p(xd), V, 0.3, net._p(y[1]), 16, 8, net._p(xf), st))
    lib.sepx_synchronize()
    s = x * np.float32(0.3)
    assert torch.equal(xf.cpu(), s)
    for t in y:
        t = t.cpu()
        assert torch.equal(t[:, 8], s.to(torch.bfloat16)) and (t[:, :8] == 7.0).all() and (t[:, 9:] == 0).all()
