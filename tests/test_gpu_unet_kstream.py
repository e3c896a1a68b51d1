"""The convolution with streamed weights (csrc/sepx_unet_kstream.inc) at the
edges of its tiles, K ranges and plane rings, against the FP64 restatement and
against the gather kernel it takes these layers from.

Tolerances: an FP32 output differs from the FP64 sum of the same BF16 products
by FP32 accumulation alone: at most 27 * 208 terms, each addition rounding the
running sum to 2^-24, so relative L2 <= sqrt(5616) * 2^-24 = 4.5e-6 for the
random signs used here; 1e-5 as the other convolution tests, twice that
between the two kernels.  A BF16 output rounds once more (2^-9): 4e-3."""
import numpy as np
import pytest

from oracle import unet_oracle as U
from tests.harness import rel_l2

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# (cin, cout, nb, D, H, W): K ranges inside one dz and across them, full and
# ragged rows; one range (>= 304 tiles of 128 voxels) with uneven runs of
# planes, ragged rows and columns, planes smaller than a tile (H = 8, W = 4);
# the widest columns (np = 128) and plane slots (160, 208 channels); two layers
# short of the line (the gather kernel takes them)
CASES = [(112, 48, 2, 12, 32, 24), (112, 48, 2, 13, 31, 24), (48, 112, 2, 12, 32, 16), (128, 128, 1, 24, 32, 24),
         (208, 16, 1, 24, 32, 24), (112, 48, 1, 41, 33, 40), (48, 112, 2, 23, 31, 40), (160, 16, 1, 19, 48, 56),
         (16, 128, 2, 60, 8, 48), (32, 1, 1, 700, 16, 4), (112, 48, 1, 1, 16, 8), (16, 16, 2, 22, 9, 31)]


@pytest.mark.parametrize("cin,cout,nb,D,H,W", CASES)
def test_kstream_convolution(cin, cout, nb, D, H, W):
    from sep_code_gb300 import unet as net
    from sep_code_gb300._lib import lib
    rng = np.random.default_rng(D * 1000 + H + cin)
    V = nb * D * H * W
    x = U.bf16(rng.standard_normal((nb, D, H, W, cin)))
    w = (rng.standard_normal((27, cin, cout)) / np.sqrt(27 * cin)).astype(np.float32)
    b = rng.standard_normal(cout).astype(np.float32)
    lib.sepx_setup_cuda(1)
    st = lib.sepx_get_stream()
    xw = np.full((V, cin + 8), 7.0, np.float32)      # the input is a slice of a wider buffer
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
