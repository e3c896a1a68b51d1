"""The z-walk convolution (csrc/sepx_unet_zwfwd.inc) at the edges of its tiles,
windows and channel groups, against the FP64 restatement.

Tolerances: an FP32 output differs from the FP64 sum of the same BF16 products
by FP32 accumulation alone: at most 27 * 80 terms, each addition rounding the
running sum to 2^-24, so relative L2 <= sqrt(2160) * 2^-24 = 2.8e-6 for the
random signs used here; 1e-5 as the other convolution tests.  A BF16 output
rounds that once more (2^-9): 4e-3."""
import numpy as np
import pytest

from oracle import unet_oracle as U
from tests.harness import rel_l2

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# (cin, cout, nb, D, H, W): one plane, planes fewer than a window, windows of
# uneven length and several per CTA, ragged rows and columns, odd group
# counts (8, 24, 40), the smallest and largest column blocks (np 16 .. 80),
# weights that leave one CTA per SM (80 -> 32, 32 -> 80)
CASES = [(8, 16, 1, 1, 16, 8), (16, 16, 2, 3, 17, 9), (16, 1, 1, 5, 16, 24), (24, 24, 1, 7, 31, 23),
         (40, 48, 1, 18, 16, 15), (48, 16, 1, 50, 96, 96), (32, 32, 3, 33, 40, 47), (80, 32, 1, 19, 33, 16),
         (32, 80, 2, 11, 18, 40), (48, 64, 1, 9, 48, 50), (8, 16, 1, 37, 130, 90)]


@pytest.mark.parametrize("cin,cout,nb,D,H,W", CASES)
def test_zwalk_convolution(cin, cout, nb, D, H, W):
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
    yf = torch.zeros((V, cout), dtype=torch.float32).cuda()
    torch.cuda.synchronize()
    net._chk(lib.sepx_unet_pack_weights(net._p(wt), cout, cin, 27, 0, net._p(pk), st))
    net._chk(lib.sepx_unet_conv_fwd(net._p(xt), cin + 8, 8, nb, D, H, W, cin, 27, net._p(pk), net._p(bt), cout, 0,
                                    None, 0, 0, net._p(yf), net._p(resid), st))
    lib.sepx_synchronize()
    assert lib.sepx_unet_status() == 0
    want = U.conv_fwd(x, U.bf16(w), b, False).reshape(V, cout)
    got = yf.cpu().numpy().astype(np.float64) - resid.cpu().numpy()
    assert rel_l2(got, want) <= 1e-5
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
