"""The halo-staged convolution (conv_halo_kernel, csrc/sepx_unet.cu) on the
layers that are its own: 81 to 128 output channels, whose three column blocks do
not fit one MMA of the z-walk kernel, and 40 -> 65..80, whose weights leave that
kernel's ring no room.  Against the FP64 restatement and the gather kernel.

Tolerances: an FP32 output differs from the FP64 sum of the same BF16 products
by FP32 accumulation alone: at most 27 * 40 terms, each addition rounding the
running sum to 2^-24, so relative L2 <= sqrt(1080) * 2^-24 = 2.0e-6 for the
random signs used here; 1e-5 as the other convolution tests, twice that between
the two kernels.  A BF16 output rounds once more (2^-9): 4e-3."""
import numpy as np
import pytest

from oracle import unet_oracle as U
from tests.harness import rel_l2

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# (cin, cout, nb, D, H, W): one tile and ragged ones, one and several channel
# pairs, odd group counts, the widest columns, more tiles than resident CTAs
CASES = [(8, 96, 1, 1, 16, 8), (8, 128, 2, 3, 17, 9), (16, 96, 1, 5, 31, 23), (16, 81, 1, 2, 18, 10),
         (24, 128, 1, 4, 33, 16), (32, 112, 2, 3, 20, 27), (40, 80, 1, 5, 19, 30), (40, 72, 1, 17, 48, 50),
         (16, 128, 1, 40, 64, 40)]


@pytest.mark.parametrize("cin,cout,nb,D,H,W", CASES)
def test_halo_convolution_of_wide_layers(cin, cout, nb, D, H, W):
    from sep_code_gb300 import unet as net
    from sep_code_gb300._lib import lib
    rng = np.random.default_rng(D * 1000 + H + cin)
    V = nb * D * H * W
    x = U.bf16(rng.standard_normal((nb, D, H, W, cin)))
    w = (rng.standard_normal((27, cin, cout)) / np.sqrt(27 * cin)).astype(np.float32)
    b = rng.standard_normal(cout).astype(np.float32)
    lib.sepx_setup_cuda(1)
    st = lib.sepx_get_stream()
    xw = np.full((V, cin + 8), np.nan, np.float32)   # a slice of a wider buffer whose other channels are NaN
    xw[:, 8:] = x.reshape(V, cin)
    xt = torch.tensor(xw).to(torch.bfloat16).cuda()
    wt, bt = torch.tensor(w).cuda(), torch.tensor(b).cuda()
    pk = torch.zeros(lib.sepx_unet_packed_elems(cout, cin, 27, 0), dtype=torch.bfloat16).cuda()
    resid = torch.tensor(rng.standard_normal((V, cout)).astype(np.float32)).cuda()
    yf, yg = (torch.zeros((V, cout), dtype=torch.float32).cuda() for _ in range(2))
    torch.cuda.synchronize()
    net._chk(lib.sepx_unet_pack_weights(net._p(wt), cout, cin, 27, 0, net._p(pk), st))

    def conv(out):
        net._chk(lib.sepx_unet_conv_fwd(net._p(xt), cin + 8, 8, nb, D, H, W, cin, 27, net._p(pk), net._p(bt), cout,
                                        0, None, 0, 0, net._p(out), net._p(resid), st))
    conv(yf)
    prev = lib.sepx_unet_set_halo(0)
    try:
        conv(yg)
    finally:
        lib.sepx_unet_set_halo(prev)
    lib.sepx_synchronize()
    assert lib.sepx_unet_status() == 0
    want = U.conv_fwd(x, U.bf16(w), b, False).reshape(V, cout)
    got, gather = (t.cpu().numpy().astype(np.float64) - resid.cpu().numpy() for t in (yf, yg))
    assert rel_l2(got, want) <= 1e-5
    assert rel_l2(got, gather) <= 2e-5
    if cout % 8:
        return
    # ReLU into a slice of a wider buffer, then masked without bias (a data gradient's form)
    mask = torch.tensor(rng.standard_normal((V, cout)).astype(np.float32)).to(torch.bfloat16).cuda()
    y = torch.full((V, cout + 8), -3.0, dtype=torch.bfloat16).cuda()
    y2 = torch.zeros((V, cout), dtype=torch.bfloat16).cuda()
    torch.cuda.synchronize()
    net._chk(lib.sepx_unet_conv_fwd(net._p(xt), cin + 8, 8, nb, D, H, W, cin, 27, net._p(pk), net._p(bt), cout, 1,
                                    net._p(y), cout + 8, 8, None, None, st))
    net._chk(lib.sepx_unet_conv_fwd_masked(net._p(xt), cin + 8, 8, nb, D, H, W, cin, 27, net._p(pk), None, cout, 0,
                                           net._p(y2), cout, 0, None, None, net._p(mask), cout, 0, st))
    lib.sepx_synchronize()
    assert lib.sepx_unet_status() == 0
    yh = y.float().cpu().numpy()
    assert (yh[:, :8] == -3.0).all()
    assert rel_l2(yh[:, 8:], np.maximum(want, 0)) <= 4e-3
    assert rel_l2(y2.float().cpu().numpy(), (want - b) * (mask.float().cpu().numpy() > 0)) <= 4e-3
