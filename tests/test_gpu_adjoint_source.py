"""The RTM adjoint adds the source values of a step inside the next one, on
grids of every size; its two-row tile (no such form) adds them by a launch per
step.  Both give the same image, bit for bit: on a small grid and on one of 47
million cells, with sources that share a cell or lie at the ends of the updated
box."""
import numpy as np
import pytest

from sep_code_gb300 import gpu_funcs as gf
from sep_code_gb300._lib import check, lib

pytestmark = pytest.mark.gpu

ADJOINT = 2   # PropMode


@pytest.mark.parametrize("n,nt", [((80, 64, 90), 14), ((368, 360, 380), 7)])
def test_fused_source_values_give_the_same_image(n, nt):
    n1, n2, n3 = n
    rng = np.random.default_rng(nt)
    gf.setup_cuda(1)
    gf.create_gpu_space(10.0, 10.0, 10.0, 50.0, 0.0005, 0.0005, n1, n2, n3)
    tab = np.zeros((1, 8), np.float32)
    tab[0, 3] = 1.0
    gf.transfer_sinc_table_s(tab)
    gf.transfer_sinc_table_d(tab)
    xe, ye, ze = 4 + (n1 - 8) // 16 * 16, 4 + (n2 - 8) // 16 * 16, n3 - 8
    pts = [(40, 30, 20)] * 3 + [(41, 30, 20), (4, 4, 4), (xe - 1, ye - 1, ze - 1), (4, ye - 1, 20), (xe - 1, 4, ze - 1),
           (40, 30, 20)]
    src = np.array([x + n1 * (y + n2 * z) for x, y, z in pts], np.int32)
    vals = rng.standard_normal((len(pts), nt + 9)).astype(np.float32)
    gf.transfer_source_func(src, vals)
    z = np.arange(n3, dtype=np.float32)[:, None, None]
    gf.transfer_vel_func1(np.ascontiguousarray(np.broadcast_to(((1500 + 4 * z) * 1e-3) ** 2, (n3, n2, n1)), np.float32))
    ix, iy = np.meshgrid(np.arange(24, 56, dtype=np.int32), np.arange(20, 36, dtype=np.int32))
    rec = (ix + n1 * (iy + n2 * 25)).reshape(-1).astype(np.int32)
    data = rng.standard_normal((rec.size, nt + 9)).astype(np.float32)
    gf.transfer_receiver_func(32, 16, rec, data)
    image = {}
    try:
        for rows in (1, 2):
            check(lib.sepx_set_tile_rows(ADJOINT, rows))
            check(lib.sepx_source_prop_resident(1, len(pts), nt))
            gf.set_traces(data)
            check(lib.sepx_rtm_adjoint_resident(1, len(pts), nt, 1))
            image[rows] = gf.get_image((n3, n2, n1))
    finally:
        check(lib.sepx_set_tile_rows(ADJOINT, 1))
    assert gf.device_error() == 0
    assert np.abs(image[1]).max() > 0
    assert np.array_equal(image[1].view(np.uint32), image[2].view(np.uint32))
