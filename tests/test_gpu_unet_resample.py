"""The pooling and upsampling kernels' coordinates (reciprocal divisions) on odd
and uneven volumes, channel counts with 1 to 14 groups and slices of wider
buffers, bit for bit against PyTorch on the CPU: the sums take the children in
the same order in FP32 and round once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# coarse shapes (nb, D, H, W) and channels
@pytest.mark.parametrize("nb,D,H,W,c", [(1, 1, 1, 1, 8), (2, 3, 5, 7, 24), (1, 7, 1, 13, 16), (3, 2, 31, 33, 48),
                                        (1, 9, 17, 3, 112)])
def test_pool_and_upsample_bits(nb, D, H, W, c):
    from sep_code_gb300 import unet as net
    from sep_code_gb300._lib import lib
    lib.sepx_setup_cuda(1)
    st = lib.sepx_get_stream()
    g = torch.Generator().manual_seed(nb * 1000 + c + W)
    fine = torch.randn((nb, 2 * D, 2 * H, 2 * W, c), generator=g).to(torch.bfloat16)
    coarse = torch.randn((nb, D, H, W, c), generator=g).to(torch.bfloat16)
    fmask = torch.randn((nb, 2 * D, 2 * H, 2 * W, c), generator=g).to(torch.bfloat16)
    cmask = torch.randn((nb, D, H, W, c), generator=g).to(torch.bfloat16)
    kids = [fine[:, a::2, b::2, d::2].float() for a in (0, 1) for b in (0, 1) for d in (0, 1)]
    s = torch.zeros_like(kids[0])
    for k in kids:
        s = s + k

    def up(t):
        return t.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)

    def wide(t):      # a slice of a buffer 16 channels wider, from channel 8
        w = torch.full((*t.shape[:-1], c + 16), 5.0, dtype=torch.bfloat16)
        w[..., 8:8 + c] = t
        return w.cuda()

    cs = c + 16
    f, q, fm, cm = wide(fine), wide(coarse), wide(fmask), wide(cmask)
    pool, upb = wide(torch.zeros_like(coarse)), wide(torch.zeros_like(coarse))
    upd, pb = wide(torch.zeros_like(fine)), wide(fine)
    torch.cuda.synchronize()
    p = net._p
    net._chk(lib.sepx_unet_avgpool(p(f), cs, 8, nb, 2 * D, 2 * H, 2 * W, c, p(pool), cs, 8, st))
    net._chk(lib.sepx_unet_upsample(p(q), cs, 8, nb, D, H, W, c, p(upd), cs, 8, st))
    net._chk(lib.sepx_unet_upsample_bwd_masked(p(f), cs, 8, nb, D, H, W, c, p(upb), cs, 8, p(cm), cs, 8, st))
    net._chk(lib.sepx_unet_avgpool_bwd_masked(p(q), cs, 8, nb, 2 * D, 2 * H, 2 * W, c, p(pb), cs, 8, 1, p(fm), cs, 8, st))
    lib.sepx_synchronize()
    zero = torch.zeros(())
    want = {"pool": (pool, (s * 0.125).to(torch.bfloat16)), "up": (upd, up(coarse)),
            "up_bwd": (upb, torch.where(cmask.float() > 0, s.to(torch.bfloat16).float(), zero).to(torch.bfloat16)),
            "pool_bwd": (pb, torch.where(fmask.float() > 0, (up(coarse).float() * 0.125 + fine.float()).to(torch.bfloat16)
                                         .float(), zero).to(torch.bfloat16))}
    for name, (got, w) in want.items():
        got = got.cpu()
        assert np.array_equal(got[..., 8:8 + c].float().numpy(), w.float().numpy()), name
        assert (got[..., :8] == 5.0).all() and (got[..., 8 + c:] == 5.0).all(), name
